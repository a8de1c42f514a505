"""A bias brought to shared memory by TMA: sizes at the edges of its 128 x 128 tiles and of the 32-column boxes, both
head-size classes, broadcast forms, strided views, and rows TMA cannot address (which keep the direct loads).
Tolerances as in test_gpu_pair_kernels: the rounding of the result is all that is left of the pairs' arithmetic.
"""
import pytest
import torch

from flash_attention_v100.ops.attention import launch_backward, launch_forward
from test_gpu_pair_kernels import TOL, _case, _rand, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("form", ["full", "heads", "query"])
@pytest.mark.parametrize("D,Nq,Nk,causal", [(64, 260, 132, False), (64, 516, 516, True), (128, 300, 260, False), (128, 260, 260, True),
                                            (96, 129, 384, False), (40, 64, 4, False)])
def test_sizes_and_forms(device, dtype, form, D, Nq, Nk, causal):
    _case(device, dtype, 2, Nq, Nk, 2, 2, D, causal, form=form, seed=Nq + D)


@pytest.mark.parametrize("D", [64, 128])
def test_groups_key_counts_and_bottom_right(device, D):
    _case(device, torch.bfloat16, 2, 140, 300, 4, 2, D, False, form="heads", lengths=[1, 129], seed=5)
    _case(device, torch.float16, 1, 100, 336, 4, 1, D, True, form="full", shift=236, seed=6)


@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 64), (torch.float16, 64), (torch.bfloat16, 128)])
def test_every_tile_is_read_before_the_next_one_lands(device, dtype, D):
    """Enough blocks for several per SM and several steps each, where a tile overwritten too early shows: the staged
    bias against the same bias in rows TMA cannot address, which the kernels load directly.  The arithmetic is the
    same, so results are equal bit for bit."""
    B, N, H = 4, 1024, 8
    gen = torch.Generator(device=device).manual_seed(1)
    q, k, v, g = (torch.randn(B, N, H, D, generator=gen, device=device).to(dtype) for _ in range(4))
    bias = torch.randn(1, H, N, N, generator=gen, device=device) * 0.5
    wide = torch.zeros(1, H, N, N + 1, device=device)
    wide[..., :N] = bias

    def run(b):
        o, lse = launch_forward(q, k, v, D ** -0.5, False, bias=b)
        ds = torch.zeros(B, H, N, N, device=device)
        return (o, lse, ds, *launch_backward(g, q, k, v, o, lse, D ** -0.5, False, bias=b, d_scores=ds))
    want = run(wide[..., :N])
    for _ in range(4):
        assert all(torch.equal(a, b) for a, b in zip(run(bias), want))


def test_bias_views(device):
    """A bias cut out of a wider tensor: with rows on 16-byte boundaries, and shifted by one value."""
    B, N, H, D = 2, 200, 2, 64
    q, k, v, g = (_rand((B, N, H, D), torch.float16, i).to(device) for i in range(4))
    dense = _rand((1, H, N, N), torch.float32, 9).to(device)
    want = None
    for offset in (None, 4, 1):
        bias = dense
        if offset is not None:
            wide = torch.full((1, H, N, N + 8), 100.0, device=device)
            wide[..., offset:offset + N] = dense
            bias = wide[..., offset:offset + N]
        o, lse = launch_forward(q, k, v, 0.125, False, bias=bias)
        ds = torch.zeros(B, H, N, N, device=device)
        got = (o, lse, ds, *launch_backward(g, q, k, v, o, lse, 0.125, False, bias=bias, d_scores=ds))
        want = want or got
        assert all(_rel(a, b) <= TOL[torch.float16] for a, b in zip(got, want))


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Nk", [197, 129, 3])
@pytest.mark.parametrize("shape,H", [((1, 1), 2), ((2, 1), 2), ((2, 1), 1), ((1, 1), 1), ((2, 2), 2)])
def test_masks_cut_out_of_wider_rows(device, D, Nk, shape, H):
    """mask[..., :Nq, :Nk] of a buffer whose rows are a multiple of 16 bytes apart while Nk is none, with dimensions of
    size one in front.  The same values in rows TMA cannot address take the direct loads: equal bit for bit."""
    Nq, dtype = 130, torch.bfloat16
    q, g = (_rand((2, Nq, H, D), dtype, s).to(device) for s in (1, 2))
    k, v = (_rand((2, Nk, H, D), dtype, s).to(device) for s in (3, 4))
    values = _rand((*shape, Nq, Nk), torch.float32, 5).to(device)

    def run(pitch):
        wide = torch.full((*shape, Nq + 7, pitch), 100.0, device=device)
        wide[:, :, :Nq, :Nk] = values
        bias = wide[:, :, :Nq, :Nk]
        o, lse = launch_forward(q, k, v, D ** -0.5, False, bias=bias)
        ds = torch.zeros(2, H, Nq, Nk, device=device)
        return (o, lse, ds, *launch_backward(g, q, k, v, o, lse, D ** -0.5, False, bias=bias, d_scores=ds))
    assert all(torch.equal(a, b) for a, b in zip(run(200), run(201)))
