"""Kept keys first, on the GPU: the scan's order and the moved rows equal torch's sort, gather and scatter exactly."""
import pytest
import torch

import flash_attention_v100 as fa
from flash_attention_v100 import modules
from flash_attention_v100.kernels import _cabi

pytestmark = pytest.mark.gpu


def _mask(B, N, form, device):
    if form == "none":
        return torch.zeros(B, N, dtype=torch.bool, device=device)
    if form == "all":
        return torch.ones(B, N, dtype=torch.bool, device=device)
    gen = torch.Generator().manual_seed(N)
    if form == "tail":
        return (torch.arange(N)[None, :] >= torch.randint(1, N + 1, (B, 1), generator=gen)).to(device)
    return (torch.rand(B, N, generator=gen) < 0.4).to(device)


@pytest.mark.parametrize("dtype,H,D", [(torch.bfloat16, 1, 8), (torch.float16, 3, 24), (torch.float32, 2, 64)])
@pytest.mark.parametrize("N", [1, 31, 33, 1023, 1024, 1025, 2500])
@pytest.mark.parametrize("form", ["none", "all", "tail", "holes"])
def test_equals_the_torch_operations(device, dtype, H, D, N, form):
    B = 3
    mask = _mask(B, N, form, device)
    k, v, gk, gv = (torch.randn(B, N, H, D, device=device).to(dtype) for _ in range(4))
    k.requires_grad_(True), v.requires_grad_(True)
    assert modules._rows_can_be_moved(k, v, mask)
    want = modules.compact_keys(k, v, mask)
    want_grads = torch.autograd.grad(want[:2], (k, v), (gk, gv))
    for m in (mask, mask.t().contiguous().t()):             # also a mask whose keys are not neighbours in memory
        got = modules._CompactKeys.apply(k, v, m)
        grads = torch.autograd.grad(got[:2], (k, v), (gk, gv.transpose(1, 2).contiguous().transpose(1, 2)))
        assert got[2].dtype == torch.int32 and not got[2].requires_grad
        assert all(torch.equal(a, b) for a, b in zip(got, want)) and all(torch.equal(a, b) for a, b in zip(grads, want_grads))


def test_rule_and_refusals(device):
    k = torch.zeros(2, 5, 3, 4, device=device)              # rows of 48 bytes
    mask = torch.zeros(2, 5, dtype=torch.bool, device=device)
    assert modules._rows_can_be_moved(k, k, mask)
    assert not modules._rows_can_be_moved(k[..., :3].contiguous(), k[..., :3].contiguous(), mask)       # 36 bytes
    assert not modules._rows_can_be_moved(k.transpose(1, 2).contiguous().transpose(1, 2), k, mask)      # not dense
    assert not modules._rows_can_be_moved(k, k, mask.cpu())
    order = torch.zeros(2, 5, dtype=torch.int32, device=device)
    call = lambda src, row: _cabi.load().fa_b200_permute_rows(src, k.data_ptr(), k.data_ptr(), k.data_ptr(), order.data_ptr(), 2, 5, row, 0,
                                                              0, None)
    assert call(k.data_ptr(), 40) == _cabi.FA_EALIGN and call(k.data_ptr() + 4, 48) == _cabi.FA_EALIGN and call(None, 48) == _cabi.FA_EINVAL


def test_layer_with_one_frozen_projection(device):
    """A key projection without gradients: the value's still flow (and the layer equals the bias form of its mask)."""
    torch.manual_seed(0)
    layer = fa.EnhancedMultiHeadAttention(64, 1, enable_multi_gpu=False).to(device, torch.float16)
    x = torch.randn(2, 70, 64, device=device, dtype=torch.float16)
    mask = _mask(2, 70, "holes", device)
    layer.k_proj.requires_grad_(False)
    out, _ = layer(x, key_padding_mask=mask)
    float_mask = torch.zeros(mask.shape, device=device).masked_fill_(mask, float("-inf"))
    ref, _ = layer(x, key_padding_mask=float_mask)
    g = torch.randn_like(out)
    a = torch.autograd.grad(out, layer.v_proj.weight, g)[0]
    b = torch.autograd.grad(ref, layer.v_proj.weight, g)[0]
    assert (out - ref).norm() <= 2e-3 * ref.norm() and (a - b).norm() <= 2e-3 * b.norm()
