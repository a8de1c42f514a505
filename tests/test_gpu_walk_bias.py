"""The walk over blocks of the instance that also writes d(loss)/d(scores), where many of a call's blocks have one key tile:
with one tile a block's row vectors are read and its row sums left within the same step, in the same room.

Every column of a call with more blocks than SMs is the result of that column in a call of its own, in which every CTA has
one block, bit for bit, time after time; and one of them agrees with the oracle (tolerances of test_gpu_pair_kernels).
"""
import pytest
import torch

from flash_attention_v100.ops.attention import launch_backward, launch_forward
from oracle import attention_oracle as ao
from test_gpu_pair_kernels import TOL, _rel

pytestmark = pytest.mark.gpu
NAMES = ("o", "dq", "dk", "dv", "ds")


def _step(q, k, v, g, bias, causal, lengths):
    scale = q.shape[3] ** -0.5
    res = torch.empty_like(q)
    o, lse = launch_forward(q, k, v, scale, causal, bias=bias, key_lengths=lengths, o_residual=res)
    ds = torch.zeros(q.shape[0], q.shape[2], q.shape[1], k.shape[1], device=q.device)
    return (o, *launch_backward(g, q, k, v, o, lse, scale, causal, bias=bias, d_scores=ds, key_lengths=lengths, o_residual=res), ds)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Nq,Nk,causal,counts,form", [
    (256, 128, False, None, "heads"),                    # one key tile, whole; the bias by TMA
    (256, 77, False, None, "heads"),                     # ... rows TMA cannot address
    (200, 100, False, None, "keys"),                     # ... one row for all queries
    (256, 256, True, None, "heads"),                     # the first query tile sees one key tile, the second two
    (130, 130, True, None, "keys"),
    (256, 300, False, (1, 128, 129, 300), "heads"),      # one, one, two and three key tiles by key counts
    (256, 301, False, (300, 7, 128, 1), "keys"),
])
def test_blocks_of_one_key_tile(device, dtype, D, Nq, Nk, causal, counts, form):
    B, H = 20, 16
    gen = torch.Generator(device=device).manual_seed(Nk + D)
    mk = lambda n: torch.randn(B, n, H, D, generator=gen, device=device).to(dtype)
    q, k, v, g = mk(Nq), mk(Nk), mk(Nk), mk(Nq)
    bias = torch.randn((1, H, Nq, Nk) if form == "heads" else (B, 1, 1, Nk), generator=gen, device=device)
    lengths = None if counts is None else torch.tensor(counts * (B // len(counts)), dtype=torch.int32, device=device)
    whole = _step(q, k, v, g, bias, causal, lengths)
    for _ in range(4):
        for n, x, y in zip(NAMES, whole, _step(q, k, v, g, bias, causal, lengths)):
            assert torch.equal(x, y), f"{n}: two calls differ"
    for b in range(B):
        for h in range(H):
            at = lambda t: t[b:b + 1, :, h:h + 1]
            own = bias[:, h:h + 1] if form == "heads" else bias[b:b + 1]
            alone = _step(at(q), at(k), at(v), at(g), own, causal, None if lengths is None else lengths[b:b + 1])
            for n, x, y in zip(NAMES, whole, alone):
                assert torch.equal(x[b:b + 1, h:h + 1] if n == "ds" else at(x), y), f"{n} of column ({b}, {h})"
    b, h = 2, 5                                          # (a count of 129 or 128 keys)
    ref_bias = (bias[:, h:h + 1] if form == "heads" else bias[b:b + 1]).expand(1, 1, Nq, Nk).cpu().clone()
    if lengths is not None:
        ref_bias[..., int(lengths[b]):] = float("-inf")
    ref_bias.requires_grad_(True)
    ref = ao.attention_forward_backward(*(t[b:b + 1, :, h:h + 1].float().cpu() for t in (q, k, v, g)), causal=causal, scale=D ** -0.5, bias=ref_bias)
    ref = dict(zip(NAMES, (ref[0], *ref[2:], ref_bias.grad)))
    for n, x in zip(NAMES, whole):
        x = x[b:b + 1, h:h + 1] if n == "ds" else x[b:b + 1, :, h:h + 1]
        assert _rel(x, ref[n]) <= TOL[dtype], (n, _rel(x, ref[n]))
