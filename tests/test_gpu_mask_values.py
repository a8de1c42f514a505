"""Additive masks of large finite values on the tensor-core kernels: the lowest (and largest) values of a type and -1e9,
where multiplying the bias by log2(e) overflows or is rounded by more than a unit.

A row all of whose keys carry such a value is uniform over them (its scores vanish in the rounding of score + bias), as
on the CUDA-core tiles and in torch.  Both kernel families round that sum alike, so they have to agree to the rounding
of the 16-bit results (tolerances of test_gpu_pair_kernels); d(loss)/d(scores) and lse are fp32.
"""
import pytest
import torch

import flash_attention_v100 as fa
from flash_attention_v100.ops.attention import launch_backward, launch_forward
from test_gpu_pair_kernels import TOL, _rand, _rel

pytestmark = pytest.mark.gpu
VALUES = {"fp32-min": torch.finfo(torch.float32).min, "bf16-min": torch.finfo(torch.bfloat16).min, "fp32-max": torch.finfo(torch.float32).max,
          "-1e9": -1e9, "-1e4": -1e4}


def _masked(form, value, H, Nq, Nk):
    if form == "padding":                       # (B, 1, 1, Nk): the second batch entry has no key at all
        bias = torch.zeros(2, 1, 1, Nk)
        bias[0, ..., Nk - 20:] = value
        bias[1] = value
        return bias
    bias = _rand((1, H, Nq, Nk), torch.float32, 9)
    if form == "rows":
        bias[:, :, 7::50] = value               # whole rows among ordinary ones
    else:
        bias[..., :30] = value                  # left padding: with a causal mask the first rows see nothing else
    return bias


def _run(q, k, v, g, bias, causal):
    scale = q.shape[3] ** -0.5
    res = torch.empty_like(q)                   # delta without the rounding of o, on either kernel family
    o, lse = launch_forward(q, k, v, scale, causal, bias=bias, o_residual=res)
    ds = torch.zeros(q.shape[0], q.shape[2], q.shape[1], k.shape[1], device=q.device)
    grads = launch_backward(g, q, k, v, o, lse, scale, causal, bias=bias, d_scores=ds, o_residual=res)
    return dict(zip(("o", "lse", "ds", "dq", "dk", "dv"), (o, lse, ds, *grads)))


@pytest.mark.parametrize("value", VALUES)
@pytest.mark.parametrize("form,causal", [("rows", False), ("rows", True), ("left", True), ("padding", False)])
@pytest.mark.parametrize("dtype,D,N", [(torch.bfloat16, 64, 200), (torch.float16, 64, 201), (torch.bfloat16, 128, 260), (torch.float16, 96, 132)],
                         ids=["bf16-d64", "fp16-d64-direct", "bf16-d128", "fp16-d96"])
def test_as_on_the_cuda_cores(device, dtype, D, N, form, causal, value):
    q, k, v, g = (_rand((2, N, 2, D), dtype, s).to(device) for s in range(4))
    bias = _masked(form, VALUES[value], 2, N, N).to(device)
    with fa.kernel_variant("simt"):
        want = _run(q, k, v, g, bias, causal)
    got = _run(q, k, v, g, bias, causal)
    for n in want:
        assert torch.isfinite(want[n]).all() and torch.isfinite(got[n]).all(), n
        assert _rel(got[n], want[n]) <= TOL[dtype], (n, _rel(got[n], want[n]))


@pytest.mark.parametrize("dtype,D,N", [(torch.bfloat16, 64, 200), (torch.float16, 64, 201), (torch.bfloat16, 128, 260), (torch.float16, 96, 132)],
                         ids=["bf16-d64", "fp16-d64-direct", "bf16-d128", "fp16-d96"])
@pytest.mark.parametrize("row", [float("-inf"), float("nan")], ids=["-inf", "nan"])
def test_a_row_without_a_result_has_no_gradient_where_it_sees_nothing(device, dtype, D, N, row):
    """Under a causal mask d(loss)/d(scores) of a row that is no number stays zero beyond the diagonal (which the sum over
    a broadcast bias' batch would spread to other entries), and dK of keys no such row sees stays a number."""
    q, k, v, g = (_rand((2, N, 2, D), dtype, s).to(device) for s in range(4))
    bias = _rand((1, 2, N, N), torch.float32, 9).to(device)
    bias[:, :, 70] = row
    with fa.kernel_variant("simt"):
        want = _run(q, k, v, g, bias, True)
    got = _run(q, k, v, g, bias, True)
    assert (got["ds"][:, :, 70, 71:] == 0).all() and torch.equal(torch.isnan(got["ds"]), torch.isnan(want["ds"]))
    assert torch.isfinite(got["dk"][:, 71:]).all()


@pytest.mark.parametrize("dtype,D,N", [(torch.bfloat16, 64, 200), (torch.float16, 64, 201), (torch.bfloat16, 128, 260), (torch.float16, 96, 132)],
                         ids=["bf16-d64", "fp16-d64-direct", "bf16-d128", "fp16-d96"])
@pytest.mark.parametrize("where", ["g", "v"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), "max"])
def test_one_value_that_is_no_number_leaves_the_other_rows_alone(device, dtype, D, N, where, value):
    """An infinity, a NaN or the type's largest value in one row of dO or V (an overflowing loss scale): gradients that
    are numbers on the CUDA cores are the same numbers here, but for a dP that overflows the tensor core's sum."""
    t = {n: _rand((2, N, 2, D), dtype, s) for s, n in enumerate("qkvg")}
    if value == "max":
        # (the largest bf16 value times another one is an infinity in fp32 arithmetic as well)
        value = 65504.0 if dtype == torch.float16 else 2.0 ** 120
    t[where][0, 100, 0, 3] = value
    bias = _rand((1, 2, N, N), torch.float32, 9).to(device)
    q, k, v, g = (x.to(device) for x in t.values())
    with fa.kernel_variant("simt"):
        want = _run(q, k, v, g, bias, False)
    got = _run(q, k, v, g, bias, False)
    for n in ("ds", "dq", "dk", "dv"):
        assert torch.isfinite(got[n][torch.isfinite(want[n])]).all(), n
    if where == "g":
        for b in range(2):
            for h in range(2):
                for n in ("ds", "dq"):
                    a, w = ((x[b, h] if n == "ds" else x[b, :, h]).double() for x in (got[n], want[n]))
                    rows = torch.arange(N, device=device) != 100
                    err = ((a - w).norm(dim=1) / w.norm(dim=1))[rows].max().item()
                    assert err <= 2 * TOL[dtype], (n, b, h, err)
