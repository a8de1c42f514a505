"""The walk over blocks in the forms test_gpu_walk_blocks leaves out: dropout (bits drawn in the kernel and from the call's
buffer), a bias by TMA and by direct loads with d(loss)/d(scores), both together, and the form without a workspace, whose
two converting warps also meet the staging of results.

As there: in a call with more blocks than SMs every column is, bit for bit, that column in a call of its own (in which a
CTA has one block, and which draws the same dropout by its origin), and two calls agree.  Blocks of one to seven steps and
blocks without any.
"""
import ctypes

import pytest
import torch

from flash_attention_v100.kernels import _cabi
from flash_attention_v100.ops import attention as ops

pytestmark = pytest.mark.gpu
SEED, OFFSET, P = 99, 3, 0.2


def _step(form, q, k, v, g, bias, causal, lengths, origin):
    scale, p = q.shape[3] ** -0.5, P if "drop" in form else 0.0
    o, lse, bits = ops.launch_forward(q, k, v, scale, causal, p, SEED, OFFSET, bias=bias, key_lengths=lengths, dropout_origin=origin,
                                      keep_bits="new", forward_only=False)
    if form.startswith("static"):
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
        params = ops._base_params(q, k, v, o, lse, scale, causal, p, SEED, OFFSET, 0, origin, d_o=g, dq=dq, dk=dk, dv=dv)
        keep = None
        if lengths is not None:
            params.kv_lengths, keep = ops._lengths_operand(lengths, q)
        _cabi.raise_for_status(_cabi.load().fa_b200_bwd_static(ctypes.byref(params)), "fa_b200_bwd_static")
        return {"o": o, "dq": dq, "dk": dk, "dv": dv}
    ds = None if bias is None else torch.zeros(q.shape[0], q.shape[2], q.shape[1], k.shape[1], device=q.device)
    grads = ops.launch_backward(g, q, k, v, o, lse, scale, causal, p, SEED, OFFSET, bias=bias, d_scores=ds, key_lengths=lengths,
                                dropout_origin=origin, keep_bits=(bits, True) if "buffered" in form else None)
    out = dict(zip(("o", "dq", "dk", "dv"), (o, *grads)))
    return out if ds is None else dict(out, ds=ds)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("form", ["drop drawn", "drop buffered", "bias", "bias drop drawn", "bias drop buffered", "static", "static drop"])
@pytest.mark.parametrize("N,causal,counts", [(128, False, None), (300, True, None), (513, False, None), (640, True, None),
                                             (896, False, (1, 896, 128, 129, 700))])
def test_columns_equal_calls_of_one_column(device, dtype, D, form, N, causal, counts):
    B, H, Hkv = 20, 16, 8                                # dK/dV 160 blocks or more, dQ 320
    gen = torch.Generator(device=device).manual_seed(N + D)
    mk = lambda h: torch.randn(B, N, h, D, generator=gen, device=device).to(dtype)
    q, k, v, g = mk(H), mk(Hkv), mk(Hkv), mk(H)
    bias = torch.randn(1, H, N, N, generator=gen, device=device) if "bias" in form else None        # (N 513: direct loads)
    lengths = None if counts is None else torch.tensor(counts * (B // len(counts)), dtype=torch.int32, device=device)
    whole = _step(form, q, k, v, g, bias, causal, lengths, None)
    again = _step(form, q, k, v, g, bias, causal, lengths, None)
    for n in whole:
        assert torch.equal(whole[n], again[n]), f"{n}: two calls differ"
    for b, hk in ((0, 0), (2, 3), (3, 5), (B - 1, Hkv - 1)):
        at = lambda t: t[b:b + 1, :, hk * (t.shape[2] // Hkv):(hk + 1) * (t.shape[2] // Hkv)]
        heads = slice(2 * hk, 2 * hk + 2)
        alone = _step(form, at(q), at(k), at(v), at(g), None if bias is None else bias[:, heads], causal,
                      None if lengths is None else lengths[b:b + 1], (b, 2 * hk, H))
        for n in whole:
            x = whole["ds"][b:b + 1, heads] if n == "ds" else at(whole[n])
            assert torch.equal(x, alone[n]), f"{n} of column ({b}, {hk})"
