"""The tensor-core backward of fp32 calls (operands as three bf16 planes) against float64 and the CUDA-core kernels.

Sizes sit at the edges of its 128-row tiles and 64-row steps.  Tolerance: the library's for fp32; and where a call has
enough terms for an error to be a statistic (the larger sizes), no further from float64 than 1.1 times the CUDA-core
kernels on the same forward result (a tenth for the scatter of a norm over a few thousand roundings).
"""
import ctypes

import pytest
import torch

from flash_attention_v100.kernels import _cabi
from flash_attention_v100.ops import attention as ops
from oracle import attention_oracle as ao

pytestmark = pytest.mark.gpu


def _rel(got, ref):
    got, ref = got.double().cpu(), ref.double().cpu()
    if ref.norm().item() < 1e-9:        # a single key: P = 1, dS = dP - delta cancels terms of order one
        return got.norm().item() / ref.numel() ** 0.5
    return (got - ref).norm().item() / max(ref.norm().item(), 1e-3 * ref.numel() ** 0.5)


def _run(device, B, Nq, Nk, H, Hkv, D, causal, shift=0, lengths=None, std=1.0, compare=False, seed=0):
    gen = torch.Generator().manual_seed(seed)
    q, k, v, g = (torch.randn(B, n, h, D, generator=gen) * s for n, h, s in ((Nq, H, std), (Nk, Hkv, std), (Nk, Hkv, 1.0), (Nq, H, 1.0)))
    bias = None
    if lengths is not None:
        hidden = torch.arange(Nk)[None, :] >= torch.tensor(lengths)[:, None]
        bias = torch.zeros(B, 1, 1, Nk).masked_fill_(hidden[:, None, None, :], float("-inf")).double()
    ref = ao.attention_forward_backward(q, k, v, g, causal=causal, bias=bias, causal_shift=shift, compute_dtype=torch.float64)[2:]
    ld = torch.tensor(lengths, device=device, dtype=torch.int32) if lengths is not None else None
    q, k, v, g = (t.to(device) for t in (q, k, v, g))
    scale = D ** -0.5
    kw = dict(key_lengths=ld, causal_shift=shift)
    o, lse = ops.launch_forward(q, k, v, scale, causal, **kw)
    got = ops.launch_backward(g, q, k, v, o, lse, scale, causal, **kw)
    again = ops.launch_backward(g, q, k, v, o, lse, scale, causal, **kw)
    assert all(torch.equal(a, b) for a, b in zip(got, again)), "not bit-reproducible"
    with ops.kernel_variant("simt"):
        plain = ops.launch_backward(g, q, k, v, o, lse, scale, causal, **kw)
    ops.check_status(device)
    assert not all(torch.equal(a, b) for a, b in zip(got, plain)), "the CUDA-core kernels ran"
    for name, a, b, r in zip(("dq", "dk", "dv"), got, plain, ref):
        e, e0 = _rel(a, r), _rel(b, r)
        assert e <= (1.1 * e0 if compare else 1e-5), (name, e, e0)


@pytest.mark.parametrize("Nq,Nk,causal", [(1, 1, False), (63, 65, False), (64, 64, True), (129, 129, True), (130, 257, False), (200, 128, True)])
def test_edges(device, Nq, Nk, causal):
    _run(device, 2, Nq, Nk, 2, 2, 64, causal, seed=Nq)


def test_groups_key_counts_and_bottom_right(device):
    _run(device, 2, 150, 150, 6, 2, 64, True)
    _run(device, 3, 70, 300, 4, 1, 64, False, lengths=[1, 128, 299])
    _run(device, 1, 100, 333, 2, 1, 64, True, shift=233)
    _run(device, 1, 300, 300, 2, 2, 64, True, lengths=[190])


@pytest.mark.parametrize("N,causal,std", [(1024, True, 1.0), (1500, False, 1.0), (777, True, 3.0), (2048, False, 0.3)])
def test_no_less_exact_than_the_cuda_cores(device, N, causal, std):
    _run(device, 1, N, N, 4, 4, 64, causal, std=std, compare=True, seed=N)


def test_rule_and_strided_gradients(device):
    """What stays on the CUDA cores; too little scratch; outputs written through strides that are no multiple of 4."""
    lib = _cabi.load()
    q = torch.randn(1, 70, 3, 64, device=device)
    o, lse = ops.launch_forward(q, q, q, 0.125, True)
    want = ops.launch_backward(q, q, q, q, o, lse, 0.125, True)

    def params(out, **fields):
        p = ops._base_params(q, q, q, o, lse, 0.125, True, 0.0, 0, 0)
        p.d_o = ops._tensor4(q)
        p.dq, p.dk, p.dv = (ops._tensor4(t) for t in out)
        for n, x in fields.items():
            setattr(p, n, x)
        return p

    size = lambda **f: int(lib.fa_b200_bwd_scratch_bytes(ctypes.byref(params(want, **f))))
    n = size()
    assert n > 0 and size(D=65) == 0 and size(D=40) == 0 and size(dropout_p=0.5) == 0 and size(dtype=_cabi.Params().dtype) == 0
    assert size(variant=_cabi.VARIANT_SIMT) == 0 and size(d_scores=q.data_ptr()) == 0
    buf = torch.empty(n, dtype=torch.uint8, device=device)
    wide = [torch.full((1, 70, 3, 67), 7.0, device=device) for _ in range(3)]
    out = [t[..., 1:65] for t in wide]
    assert lib.fa_b200_bwd_with_scratch(ctypes.byref(params(out)), buf.data_ptr(), n) == 0
    assert all(torch.equal(a, b) for a, b in zip(out, want))
    assert all((t[..., 0] == 7.0).all() and (t[..., 65:] == 7.0).all() for t in wide)
    assert lib.fa_b200_bwd_with_scratch(ctypes.byref(params(out)), buf.data_ptr(), n - 1) == _cabi.FA_EWORKSPACE   # and no workspace


def test_other_forwards_and_what_their_kernel_refuses_stay_on_the_cuda_cores(device):
    """The planes' error is the CUDA cores' behind the TF32 forward only: an explicit backward, whose o and lse may come
    from anywhere, a forward run on the CUDA cores, and tensors or scales that forward does not take keep theirs."""
    gen = torch.Generator().manual_seed(3)
    q, k, v, g = (torch.randn(1, 130, 2, 64, generator=gen).to(device) for _ in range(4))
    o, lse = ops.launch_forward(q, k, v, 0.125, True)
    planes = ops.launch_backward(g, q, k, v, o, lse, 0.125, True)
    with ops.kernel_variant("simt"):
        plain = ops.launch_backward(g, q, k, v, o, lse, 0.125, True)
        o1, lse1 = ops.launch_forward(q, k, v, 0.125, True)
        plain1 = ops.launch_backward(g, q, k, v, o1, lse1, 0.125, True)
    same = lambda a, b: all(torch.equal(x, y) for x, y in zip(a, b))
    assert not same(planes, plain)
    explicit = lambda **kw: ops.flash_attention_backward_enhanced(g, q, k, v, o, lse, scale=0.125, causal=True, **kw)
    assert same(explicit(), plain) and same(explicit(own_forward=True), planes)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    with ops.kernel_variant("simt"):
        out = ops.EnhancedFlashAttentionV100Function.apply(*leaves, 0.125, True)
    assert same(torch.autograd.grad(out, leaves, g), plain1)
    lib = _cabi.load()

    def size(t, scale):
        p = ops._base_params(t, k, v, o, lse, scale, True, 0.0, 0, 0, d_o=g, dq=q, dk=k, dv=v)
        return int(lib.fa_b200_bwd_scratch_bytes(ctypes.byref(p)))
    odd = torch.zeros(1, 130, 2, 67, device=device)[..., :64]
    assert size(q, 0.125) > 0 and size(odd, 0.125) == 0 and size(q, -0.125) == 0


def test_without_room_for_the_planes_the_cuda_cores_serve_the_call(device, monkeypatch):
    q = torch.randn(1, 70, 3, 64, device=device)
    o, lse = ops.launch_forward(q, q, q, 0.125, True)
    run = lambda: ops.launch_backward(q, q, q, q, o, lse, 0.125, True)
    planes = run()
    with ops.kernel_variant("simt"):
        plain = run()
    same = lambda a, b: all(torch.equal(x, y) for x, y in zip(a, b))
    assert not same(planes, plain)
    with monkeypatch.context() as m:
        m.setattr(ops, "F32_PLANES_MAX_BYTES", 1000)
        assert same(run(), plain)

    def full(self, size, **kw):                       # the allocator has nothing for a large byte buffer
        if kw.get("dtype") == torch.uint8 and size > 100000:
            raise torch.cuda.OutOfMemoryError("no block")
        return torch.empty(size, dtype=kw.get("dtype", self.dtype), device=self.device)
    with monkeypatch.context() as m:
        m.setattr(torch.Tensor, "new_empty", full)
        assert same(run(), plain)


def test_memory_estimate_covers_the_planes(device):
    from flash_attention_v100.ops import memory
    B, N, H = 2, 1000, 4
    q, g = (torch.randn(B, N, H, 64, device=device) for _ in range(2))
    o, lse = ops.launch_forward(q, q, q, 0.125, True)
    est = memory.estimate_peak_memory_usage(B, N, N, H, 64, torch.float32)["total_memory_mb"] * 2 ** 20
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated(device)
    torch.cuda.reset_peak_memory_stats(device)
    ops.launch_backward(g, q, q, q, o, lse, 0.125, True)
    torch.cuda.synchronize()
    held = (3 * q.numel() + 2 * o.numel()) * 4 + lse.numel() * 4          # q, k, v, o, dO and lse of the estimate
    assert held + torch.cuda.max_memory_allocated(device) - before <= est + (1 << 16)
