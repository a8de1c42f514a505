"""The fp32 forward's pipeline: numbers of 64-key blocks around its two stages and two score buffers, key counts and
both causal alignments, against float64 at the library's fp32 tolerance."""
import pytest
import torch

from flash_attention_v100.ops import attention as ops
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nq,Nk,causal,shift,lengths", [(1, 1, False, 0, None), (127, 64, False, 0, None), (129, 65, False, 0, None),
                                                        (128, 128, True, 0, None), (300, 193, False, 0, None), (385, 385, True, 0, None),
                                                        (70, 333, True, 263, None), (130, 320, False, 0, [1, 64, 257])])
def test_block_counts(device, Nq, Nk, causal, shift, lengths):
    B, H, Hkv = 3 if lengths else 2, 4, 2
    gen = torch.Generator().manual_seed(Nq + Nk)
    q, k, v = (torch.randn(B, n, h, 64, generator=gen) for n, h in ((Nq, H), (Nk, Hkv), (Nk, Hkv)))
    bias = None
    if lengths:
        hidden = torch.arange(Nk)[None, :] >= torch.tensor(lengths)[:, None]
        bias = torch.zeros(B, 1, 1, Nk).masked_fill_(hidden[:, None, None, :], float("-inf")).double()
    ro, rlse = ao.attention_forward(q, k, v, causal=causal, bias=bias, causal_shift=shift, compute_dtype=torch.float64)
    ld = torch.tensor(lengths, device=device, dtype=torch.int32) if lengths else None
    q, k, v = (t.to(device) for t in (q, k, v))
    runs = [ops.launch_forward(q, k, v, 0.125, causal, key_lengths=ld, causal_shift=shift) for _ in range(3)]
    ops.check_status(device)
    for o, lse in runs:
        assert (o.cpu().double() - ro).norm() <= 1e-5 * ro.norm() and (lse.cpu().double() - rlse).abs().max() <= 1e-5 * max(1.0, rlse.abs().max().item())
        assert torch.equal(o, runs[0][0]) and torch.equal(lse, runs[0][1])
