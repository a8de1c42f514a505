"""The tensor-core kernels with P and dS as hi + lo pairs: additive bias, head sizes other than 64 and 128.

Sizes sit at the edges of the 128-row tiles, of the 64-column boxes and of the MMAs' 16-column steps.  Tolerance:
with pairs nothing but the rounding of the result is left (bf16 at most 2^-9 relative to the value, 1.66e-3 as a
norm; fp16 an eighth of that, 2.1e-4), so fp16 is held to twice its rounding and bf16 to the library's 2e-3.
"""
import numpy as np
import pytest
import torch

import flash_attention_v100 as fa
from flash_attention_v100.kernels import _cabi
from flash_attention_v100.ops.attention import launch_backward, launch_forward, saves_output_residual
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu
TOL = {torch.float16: 4.2e-4, torch.bfloat16: 2e-3}


def _rel(got, ref):
    got, ref = got.detach().double().cpu(), ref.detach().double().cpu()
    return (got - ref).norm().item() / max(ref.norm().item(), 1e-3 * ref.numel() ** 0.5)


def _rand(shape, dtype, seed, std=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std).to(dtype)


def _bias_of(form, B, H, Nq, Nk, seed):
    if form is None:
        return None
    shape = {"full": (B, H, Nq, Nk), "heads": (1, H, Nq, Nk), "query": (1, 1, Nq, Nk), "padding": (B, 1, 1, Nk)}[form]
    bias = _rand(shape, torch.float32, seed)
    if form == "padding":
        bias[..., Nk // 2 + 1:] = float("-inf")
    return bias


def _case(device, dtype, B, Nq, Nk, H, Hkv, D, causal, form=None, p=0.0, buffered=False, shift=0, lengths=None, seed=0):
    q, k, v = _rand((B, Nq, H, D), dtype, seed), _rand((B, Nk, Hkv, D), dtype, seed + 1), _rand((B, Nk, Hkv, D), dtype, seed + 2)
    d_o, scale = _rand((B, Nq, H, D), dtype, seed + 3), D ** -0.5
    bias = _bias_of(form, B, H, Nq, Nk, seed + 4)
    keep, p_eff, stream = None, 0.0, (0, 0)
    if p > 0:
        stream = (0xC0FFEE + seed, 11 + seed)
        keep = np.empty((B, H, Nq, Nk), np.uint8)
        lib = _cabi.load()
        assert lib.fa_b200_dropout_mask_host(*stream, p, B, H, Nq, Nk, keep.ctypes.data) == 0
        keep, p_eff = torch.from_numpy(keep), float(lib.fa_b200_dropout_effective_p(p))
    ref_bias = bias
    if lengths is not None:          # the oracle takes key counts as a -inf mask
        hidden = torch.arange(Nk)[None, :] >= torch.tensor(lengths)[:, None]
        ref_bias = torch.zeros(B, 1, 1, Nk).masked_fill_(hidden[:, None, None, :], float("-inf")) + (0 if bias is None else bias)
    if ref_bias is not None:
        ref_bias = ref_bias.clone().requires_grad_(True)
    ro, rlse, rdq, rdk, rdv = ao.attention_forward_backward(q.float(), k.float(), v.float(), d_o.float(), causal=causal, scale=scale,
                                                            dropout_p=p_eff, keep_mask=keep, bias=ref_bias, causal_shift=shift)
    qd, kd, vd, gd = (t.to(device) for t in (q, k, v, d_o))
    bd = bias.to(device) if bias is not None else None
    ld = torch.tensor(lengths, device=device, dtype=torch.int32) if lengths is not None else None
    res = torch.empty_like(qd) if saves_output_residual(dtype) else None
    got = launch_forward(qd, kd, vd, scale, causal, p, *stream, bias=bd, key_lengths=ld, causal_shift=shift, o_residual=res,
                         keep_bits="new" if buffered else None, forward_only=False)
    o, lse, bits = got if buffered else (*got, None)
    ds = torch.zeros(B, H, Nq, Nk, device=device) if bias is not None else None
    run = lambda: launch_backward(gd, qd, kd, vd, o, lse, scale, causal, p, *stream, bias=bd, d_scores=ds, key_lengths=ld,
                                  causal_shift=shift, o_residual=res, keep_bits=(bits, True) if bits is not None else None)
    dq, dk, dv = run()
    errs = {n: _rel(a, b) for n, a, b in (("o", o, ro), ("lse", lse, rlse), ("dq", dq, rdq), ("dk", dk, rdk), ("dv", dv, rdv))}
    if bias is not None and lengths is None:
        dims = [i for i in range(4) if bias.shape[i] == 1 and ds.shape[i] != 1]
        errs["dbias"] = _rel(ds.sum(dim=dims, keepdim=True) if dims else ds, ref_bias.grad)
    assert all(e <= TOL[dtype] for e in errs.values()), errs
    assert all(torch.equal(a, b) for a, b in zip((dq, dk, dv), run())), "gradients are not bit-reproducible"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("D", [8, 24, 40, 56, 72, 96, 120])
def test_head_sizes(device, dtype, D):
    _case(device, dtype, 1, 129, 129, 2, 2, D, True, seed=D)
    _case(device, dtype, 2, 70, 257, 4, 2, D, False, seed=D + 1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("form", ["full", "heads", "query", "padding"])
@pytest.mark.parametrize("D,Nq,Nk,causal", [(64, 300, 300, False), (128, 128, 129, False), (96, 259, 259, True), (64, 1, 384, False)])
def test_bias(device, dtype, form, D, Nq, Nk, causal):
    _case(device, dtype, 2, Nq, Nk, 2, 1, D, causal, form=form, seed=Nq + D)


@pytest.mark.parametrize("dtype,D", [(torch.float16, 32), (torch.bfloat16, 96), (torch.bfloat16, 128)], ids=["fp16-d32", "bf16-d96", "bf16-d128-bias"])
@pytest.mark.parametrize("buffered", [False, True], ids=["drawn", "buffer"])
def test_dropout(device, dtype, D, buffered):
    form = "heads" if D == 128 else None
    _case(device, dtype, 1, 200, 200, 2, 2, D, True, form=form, p=0.2, buffered=buffered, seed=3)
    _case(device, dtype, 1, 130, 260, 2, 2, D, False, form=form, p=0.5, buffered=buffered, seed=4)


@pytest.mark.parametrize("dtype,D,form", [(torch.float16, 80, None), (torch.bfloat16, 64, "heads")], ids=["fp16-d80", "bf16-d64-bias"])
def test_key_counts_and_bottom_right(device, dtype, D, form):
    _case(device, dtype, 3, 140, 300, 2, 2, D, False, form=form, lengths=[1, 128, 299], seed=5)
    _case(device, dtype, 1, 100, 333, 4, 2, D, True, form=form, shift=233, seed=6)


def test_rows_whose_first_keys_are_hidden(device):
    """Row 5 sees no key at all (NaN and -inf, as on the CUDA-core tiles); rows 7.. see none in their first two key
    blocks, while their neighbours in the warp do."""
    q, k, v = (_rand((1, n, 1, 64), torch.float16, n).to(device) for n in (64, 400, 401))
    v = v[:, :400].contiguous()
    bias = torch.zeros(1, 1, 64, 400, device=device)
    bias[0, 0, 5] = float("-inf")
    bias[0, 0, 7::3, :300] = float("-inf")
    o, lse = launch_forward(q, k, v, 0.125, False, bias=bias)
    with fa.kernel_variant("simt"):
        o2, lse2 = launch_forward(q, k, v, 0.125, False, bias=bias)
    assert torch.isnan(o[0, 5]).all() and torch.isnan(o2[0, 5]).all() and lse[0, 0, 5] == lse2[0, 0, 5] == float("-inf")
    keep = torch.arange(64, device=device) != 5
    assert _rel(o[:, keep], o2[:, keep]) <= 4.2e-4 and _rel(lse[:, :, keep], lse2[:, :, keep]) <= 1e-5


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("D,N,causal", [(64, 440, False), (128, 440, False), (64, 385, True), (96, 900, False)])
def test_fp32_results_are_as_exact_as_on_the_cuda_cores(device, dtype, D, N, causal):
    """lse and d(loss)/d(scores) against float64: the CUDA-core tiles' distance is the bound.  lse is rounded once behind
    either sum, by up to half a unit of its last place, which is most of both distances: a quarter more is allowed."""
    gen = torch.Generator(device=device).manual_seed(N)
    q, k, v, g = (torch.randn(2, N, 4, D, generator=gen, device=device).to(dtype) for _ in range(4))
    bias = torch.randn(1, 4, N, N, generator=gen, device=device) * 0.5
    qd, kd, vd, gd = (t.double().transpose(1, 2) for t in (q, k, v, g))
    s = qd @ kd.transpose(-1, -2) * D ** -0.5 + bias.double()
    if causal:
        s = s.masked_fill(torch.ones(N, N, device=device, dtype=torch.bool).triu(1), float("-inf"))
    lse_ref = torch.logsumexp(s, -1)
    p = torch.exp(s - lse_ref[..., None])
    ds_ref = p * (gd @ vd.transpose(-1, -2) - (gd * (p @ vd)).sum(-1, keepdim=True))

    def errors():
        res = torch.empty_like(q)
        o, lse = launch_forward(q, k, v, D ** -0.5, causal, bias=bias, o_residual=res)
        ds = torch.zeros(2, 4, N, N, device=device)
        launch_backward(g, q, k, v, o, lse, D ** -0.5, causal, bias=bias, d_scores=ds, o_residual=res)
        return [((a.double() - r).norm() / r.norm()).item() for a, r in ((lse, lse_ref), (ds, ds_ref))]
    with fa.kernel_variant("simt"):
        lse_simt, ds_simt = errors()
    lse_pair, ds_pair = errors()
    assert lse_pair <= 1.25 * lse_simt and ds_pair <= ds_simt, (lse_pair, lse_simt, ds_pair, ds_simt)
