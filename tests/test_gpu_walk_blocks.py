"""Backward kernels whose CTAs go on from one block of the grid to the next.

A CTA that has ended a block must not leave anything of it to the next one: the rows of a block that follows one without
steps (a key tile behind every query or beyond a key count), blocks of a single step, more blocks than SMs, and every
ring position a block can begin at (n steps per block with n from 1 to 7 meet rings of 2, 3 and 4 stages).  Each block's
result is that of the same columns in a call of their own, in which every CTA has one block, bit for bit; and all of it
agrees with the oracle (tolerance of the dtype, which the other tests of these kernels use).
"""
import pytest
import torch

from flash_attention_v100.ops.attention import launch_backward, launch_forward, saves_output_residual
from flash_attention_v100.testing import rel_l2, tolerance
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


def _inputs(dtype, B, Nq, Nk, H, Hkv, D, device, seed):
    gen = torch.Generator().manual_seed(seed)
    mk = lambda n, h: torch.randn(B, n, h, D, generator=gen).to(dtype).to(device)
    return mk(Nq, H), mk(Nk, Hkv), mk(Nk, Hkv), mk(Nq, H)


def _step(q, k, v, g, causal, lengths=None, fast=False):
    scale = q.shape[-1] ** -0.5
    lo = torch.empty_like(q) if saves_output_residual(q.dtype) else None
    o, lse = launch_forward(q, k, v, scale, causal, key_lengths=lengths, o_residual=lo)
    return (o,) + launch_backward(g, q, k, v, o, lse, scale, causal, key_lengths=lengths, o_residual=lo, fast=fast)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("N,causal", [(128, False), (300, True), (513, False), (640, True), (897, False)])
def test_columns_of_a_call_with_many_blocks_equal_calls_of_one_column(device, dtype, D, N, causal):
    B, H, Hkv = 10, 16, 8                         # more blocks than SMs from one tile a column on
    q, k, v, g = _inputs(dtype, B, N, N, H, Hkv, D, device, 7 * N + D)
    whole = _step(q, k, v, g, causal)
    for b, hk in ((0, 0), (3, 5), (B - 1, Hkv - 1)):
        sl = lambda t: t[b:b + 1, :, hk * (t.shape[2] // Hkv):(hk + 1) * (t.shape[2] // Hkv)]
        part = _step(sl(q), sl(k), sl(v), sl(g), causal)
        for n, x, y in zip(("o", "dq", "dk", "dv"), whole, part):
            assert torch.equal(sl(x), y), f"{n} of column ({b}, {hk})"
    again = _step(q, k, v, g, causal)
    for n, x, y in zip(("o", "dq", "dk", "dv"), whole, again):
        assert torch.equal(x, y), f"{n}: two calls differ"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [40, 64, 128])
@pytest.mark.parametrize("fast", [False, True])
def test_blocks_without_steps_between_others(device, dtype, D, fast):
    """Key counts that leave up to nine tiles in a row without a step, before and behind long ones."""
    B, Nq, Nk, H = 12, 260, 1200, 16
    q, k, v, g = _inputs(dtype, B, Nq, Nk, H, H, D, device, D)
    lengths = torch.tensor([1, 1200, 128, 129, 7, 1100, 1, 1, 640, 1200, 3, 250], dtype=torch.int32, device=device)
    got = _step(q, k, v, g, False, lengths, fast)
    for b in (0, 3, 7, 9):
        n = int(lengths[b])
        ref = ao.attention_forward_backward(*(t[b:b + 1, :, :2].float().cpu() for t in (q, k[:, :n], v[:, :n], g)), causal=False, scale=D ** -0.5)
        for name, x, r in zip(("o", "dq", "dk", "dv"), got, (ref[0],) + tuple(ref[2:])):
            x = x[b:b + 1, :, :2].float().cpu()
            if name in ("dk", "dv"):
                assert not x[:, n:].any(), f"{name} of padding keys"
                x = x[:, :n]
            if name in ("dq", "dk") and n == 1:
                continue                          # one key: P is 1 and dS only rounding
            assert rel_l2(x, r) <= tolerance(dtype), (name, b)
