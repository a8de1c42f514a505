"""The launch that writes a call's dropout bits takes one query row a lane in small calls and four in large ones.

Columns of a large call (query blocks of 128, odd and even numbers of them) are columns of the same dropout stream in a
call of their own (query blocks of 32), which starts at that column's origin: the outputs that the bits decide agree bit
for bit, in the forward (bits by query) and in the backward (bits by key).  The walk over the causal mask's blocks, shapes
with a shift, and key counts that are no multiple of a tile are all in it.
"""
import pytest
import torch

from flash_attention_v100.ops.attention import launch_backward, launch_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Nq,Nk,H,causal,shift", [
    (16, 640, 640, 16, True, 0),            # 5 blocks of 128: the middle one is half a pair
    (16, 512, 512, 16, True, 0),
    (64, 130, 129, 16, False, 0),
    (32, 200, 700, 12, True, 500),          # no pairs: bottom-right mask
])
def test_columns_of_a_large_call_draw_the_bits_of_a_small_one(device, B, Nq, Nk, H, causal, shift):
    D, p, seed, offset = 64, 0.3, 77, 5
    gen = torch.Generator().manual_seed(Nq + Nk)
    mk = lambda n: torch.randn(B, n, H, D, generator=gen).to(torch.float16).to(device)
    q, k, v, g = mk(Nq), mk(Nk), mk(Nk), mk(Nq)

    def step(q, k, v, g, **kw):
        o, lse, bits = launch_forward(q, k, v, D ** -0.5, causal, p, seed, offset, keep_bits="new", forward_only=False,
                                      causal_shift=shift, **kw)
        assert bits is not None
        return (o,) + tuple(launch_backward(g, q, k, v, o, lse, D ** -0.5, causal, p, seed, offset, fast=False,
                                            keep_bits=(bits, True), causal_shift=shift, **kw))

    whole = step(q, k, v, g)
    for b, h in ((0, 0), (B // 2, 3), (B - 1, H - 1)):
        at = lambda t: t[b:b + 1, :, h:h + 1]
        alone = step(at(q), at(k), at(v), at(g), dropout_origin=(b, h, H))
        for name, x, y in zip(("o", "dq", "dk", "dv"), whole, alone):
            assert torch.equal(at(x), y), (name, b, h)
