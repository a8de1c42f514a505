"""The forward's packed tiles and split schedule (fa_b200_fwd_with_workspace): few queries against many keys.

Sizes sit at the edges of the 128-row tiles, of the 128-key blocks and of the ranges the units are cut into; head
groups are powers of two and not.  Tolerance: the library's, as for the schedule of whole pairs, whose arithmetic this
is up to the order of fp32 sums and the value a row's maximum has when P is rounded to fp16; the two are also
compared with each other.  Rounding every P to fp16 leaves 2^-12 / sqrt(3) = 1.4e-4 of the result's norm (terms of
random sign), rounding the result to fp16 2.1e-4: 2.5e-4 for one schedule and sqrt(2) of it, 3.6e-4, between two;
5e-4 is asked for.  In bf16 values that differ by d = 2e-4 round apart in a share d / 2^-8 of cases, by 2^-8 each: a
norm of sqrt(d 2^-8) = 8.8e-4; 1.5e-3 is asked for.  The same bounds hold with a NaN-free column beside a NaN one.
"""
import ctypes

import pytest
import torch

import flash_attention_v100 as fa
from flash_attention_v100.kernels import _cabi
from flash_attention_v100.ops import attention as ops
from flash_attention_v100.testing import rel_l2, tolerance
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


def _rand(shape, dtype, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype)


def _check(device, dtype, B, Nq, Nk, H, Hkv, D, causal=False, shift=0, lengths=None, residual=False, split=True):
    q, k, v = _rand((B, Nq, H, D), dtype, 1), _rand((B, Nk, Hkv, D), dtype, 2), _rand((B, Nk, Hkv, D), dtype, 3)
    bias = None
    if lengths is not None:
        hidden = torch.arange(Nk)[None, :] >= torch.tensor(lengths)[:, None]
        bias = torch.zeros(B, 1, 1, Nk).masked_fill_(hidden[:, None, None, :], float("-inf"))
    ro, rlse = ao.attention_forward(q.float(), k.float(), v.float(), causal=causal, scale=D ** -0.5, bias=bias, causal_shift=shift)
    ld = torch.tensor(lengths, device=device, dtype=torch.int32) if lengths is not None else None
    q, k, v = (t.to(device) for t in (q, k, v))
    o0, lse0 = ops.launch_forward(q, k, v, D ** -0.5, causal, key_lengths=ld, causal_shift=shift)
    # rows and strides as a slice of a wider tensor has them
    wide = torch.full((B, Nq, H + 1, D), 7.0, dtype=dtype, device=device)
    lo = torch.empty_like(q) if residual else None
    out = (wide[:, :, :H], torch.empty(B, H, Nq, device=device))
    p = ops._base_params(q, k, v, *out, D ** -0.5, causal, 0.0, 0, 0, shift)
    p.kv_lengths = ld.data_ptr() if ld is not None else None
    assert (_cabi.load().fa_b200_fwd_workspace_bytes(ctypes.byref(p)) > 0) == split
    for rep in range(2):
        o, lse = ops.launch_forward(q, k, v, D ** -0.5, causal, key_lengths=ld, causal_shift=shift, out=out,
                                    o_residual=lo, split_keys=True)
        first = (o.clone(), lse.clone()) if rep == 0 else first
    assert torch.equal(o, first[0]) and torch.equal(lse, first[1]), "not bit-reproducible"
    assert (wide[:, :, H] == 7.0).all()
    assert rel_l2(o, ro) <= tolerance(dtype, "auto", D) and rel_l2(lse, rlse) <= 1e-4
    assert rel_l2(o, o0) <= (1.5e-3 if dtype == torch.bfloat16 else 5e-4) and (lse - lse0).abs().max() <= 2e-3
    if residual:
        assert rel_l2(o.double() + lo.double(), ro) <= 3e-4
    ops.check_status(device)


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 128)], ids=["fp16-d64", "bf16-d128"])
@pytest.mark.parametrize("H,Hkv", [(2, 2), (8, 2), (6, 2), (12, 1)], ids=["g1", "g4", "g3", "g12"])
@pytest.mark.parametrize("Nq,Nk,shift", [(1, 1300, None), (5, 1409, 1404), (33, 1537, 1504), (130, 2000, 1870)])
def test_decoding_and_chunks(device, dtype, D, H, Hkv, Nq, Nk, shift):
    _check(device, dtype, 2, Nq, Nk, H, Hkv, D, shift is not None, shift or 0)


@pytest.mark.parametrize("lengths", [[1, 4000, 129], [2048, 2047, 2049], [1, 1, 1]])
def test_ragged_caches(device, lengths):
    _check(device, torch.bfloat16, 3, 1, 4000, 8, 2, 64, lengths=lengths)
    _check(device, torch.float16, 3, 3, 4000, 4, 4, 128, lengths=lengths, residual=True)


def test_many_batch_entries(device):
    """The start of a range is found by a scan over 32 batch entries at a time."""
    lengths = [1 + 74 * i % 3000 for i in range(70)]
    _check(device, torch.float16, 70, 1, 3000, 4, 4, 64, lengths=lengths)
    _check(device, torch.bfloat16, 40, 1, 1280, 4, 1, 128)


@pytest.mark.parametrize("longest", [128, 300, 2900])
def test_many_pairs_of_a_few_blocks(device, longest):
    """Ranges that hold many pairs, end inside the units that stand for a pair's start, or hold nothing else."""
    gen = torch.Generator().manual_seed(longest)
    lengths = torch.randint(1, longest + 1, (64,), generator=gen).tolist()
    _check(device, torch.float16, 64, 1, 3000, 4, 4, 64, lengths=lengths)
    _check(device, torch.bfloat16, 64, 3, 3000, 8, 2, 128, lengths=lengths[::-1])
    _check(device, torch.float16, 25, 150, 3000, 4, 4, 128, lengths=lengths[:25])
    _check(device, torch.float16, 5, 1, 6000, 32, 32, 64, lengths=[longest, 1, 1, 6000, 1])


@pytest.mark.parametrize("N", [1664, 2501])
def test_prompts(device, N):
    """Self-attention of one request with few heads: pairs of very different length under the causal mask."""
    _check(device, torch.bfloat16, 1, N, N, 2, 2, 128, True, residual=True)
    _check(device, torch.float16, 1, N, N, 3, 1, 64)


def test_rule_leaves_the_rest_alone(device):
    """Enough work for every SM, or too little to share: no scratch is asked for and none is used."""
    _check(device, torch.float16, 2, 128, 128, 4, 4, 64, True, split=False)
    q = torch.zeros(4, 4096, 32, 64, device=device, dtype=torch.float16)
    p = ops._base_params(q, q, q, q, torch.empty(4, 32, 4096, device=device), 0.125, True, 0.0, 0, 0)
    assert _cabi.load().fa_b200_fwd_workspace_bytes(ctypes.byref(p)) == 0
    # too little scratch, or misaligned: the schedule of whole pairs
    q, k = _rand((1, 1, 2, 64), torch.float16, 1).to(device), _rand((1, 2000, 2, 64), torch.float16, 2).to(device)
    o0, lse0 = ops.launch_forward(q, k, k, 0.125, False)
    p = ops._base_params(q, k, k, torch.empty_like(q), torch.empty_like(lse0), 0.125, False, 0.0, 0, 0)
    n = int(_cabi.load().fa_b200_fwd_workspace_bytes(ctypes.byref(p)))
    buf = torch.empty(n + 256, dtype=torch.uint8, device=device)
    for offset, size in ((0, n - 1), (16, n)):
        o, lse = torch.empty_like(o0), torch.empty_like(lse0)
        p = ops._base_params(q, k, k, o, lse, 0.125, False, 0.0, 0, 0)
        assert _cabi.load().fa_b200_fwd_with_workspace(ctypes.byref(p), buf.data_ptr() + offset, size) == 0
        assert torch.equal(o, o0) and torch.equal(lse, lse0)


def test_key_counts_alone_do_not_cut_calls_of_several_tiles(device):
    """Whole pairs that fill the SMs evenly stay whole where a unit costs the same either way, whatever the counts."""
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    q, k = (torch.zeros(sms // 2, n, 2, 128, device=device, dtype=torch.bfloat16) for n in (256, 3000))
    counts = torch.full((sms // 2,), 3000, device=device, dtype=torch.int32)
    for given in (False, True):
        p = ops._base_params(q, k, k, q, torch.empty(1, device=device), 0.125, False, 0.0, 0, 0)
        if given:
            p.kv_lengths = counts.data_ptr()
        assert _cabi.load().fa_b200_fwd_workspace_bytes(ctypes.byref(p)) == 0


def test_rows_with_nan_and_infinite_scores(device):
    """A NaN in one range's keys reaches the row's result, as with whole pairs; other columns stay clean."""
    q, k = _rand((1, 4, 2, 64), torch.float16, 1).to(device), _rand((1, 1500, 2, 64), torch.float16, 2).to(device)
    v = k.clone()
    k[0, 700, 0, 3] = float("nan")
    o, lse = fa.flash_attention_v100(q, k, v, return_softmax_lse=True, enable_multi_gpu=False)
    o0, _ = ops.launch_forward(q, k, v, 0.125, False)
    assert torch.isnan(o[:, :, 0]).all() and torch.isnan(o0[:, :, 0]).all()
    assert torch.isfinite(o[:, :, 1]).all() and rel_l2(o[:, :, 1], o0[:, :, 1]) <= 5e-4


def test_captured_in_a_graph(device):
    q, k = _rand((2, 1, 8, 128), torch.bfloat16, 1).to(device), _rand((2, 3000, 2, 128), torch.bfloat16, 2).to(device)
    run = lambda: fa.flash_attention_v100(q, k, k, enable_multi_gpu=False)
    want = run().clone()
    side = torch.cuda.Stream(device=device)
    with torch.cuda.stream(side):
        run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
