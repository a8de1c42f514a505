"""The native autograd operator against the general form of the same call: same bits, same refusals, and nobody who
watches operators (a transform, a mode, saved-tensor hooks) is passed by."""
import pytest
import torch

import flash_attention_v100 as fa
from flash_attention_v100.ops import attention as ops

pytestmark = pytest.mark.gpu


def _rand(*shape, dtype, device, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(device)


def _general(q, k, v, causal, shift=0, lengths=None, mode="balanced"):
    q, k, v, scale = ops.validate_inputs(q, k, v)
    return ops.FlashAttentionV100Function.apply(q, k, v, scale, causal, 0.0, None, None, None, True, True, False, True, None, True, mode,
                                                False, 1, 0, lengths, shift, None, None)


@pytest.fixture(autouse=True)
def _registered(device):
    ops._status_word(device)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("Nq,Nk,H,Hkv,D,causal,align,counts,mode", [
    (1, 1, 1, 1, 8, False, "top_left", False, "balanced"), (128, 128, 4, 4, 64, True, "top_left", False, "balanced"),
    (77, 200, 8, 2, 96, True, "bottom_right", False, "balanced"), (1, 700, 8, 2, 128, False, "top_left", True, "balanced"),
    (300, 300, 4, 1, 64, False, "top_left", True, "speed"), (64, 64, 2, 2, 37, True, "top_left", False, "balanced")])
@pytest.mark.parametrize("wants", ["qkv", "k", "none"])
def test_same_bits_as_the_general_form(device, dtype, Nq, Nk, H, Hkv, D, causal, align, counts, mode, wants):
    B = 3
    base = [_rand(B, n, h, D, dtype=dtype, device=device, seed=i) for i, (n, h) in enumerate(((Nq, H), (Nk, Hkv), (Nk, Hkv)))]
    lengths = torch.tensor([1, Nk, (Nk + 1) // 2], dtype=torch.int32, device=device) if counts else None
    g = _rand(B, Nq, H, D, dtype=dtype, device=device, seed=9)
    got = []
    for native in (True, False):
        q, k, v = (t.clone().requires_grad_(n in wants) for t, n in zip(base, "qkv"))
        if native:
            served = ops.native_call(q, k, v, None, causal, align == "bottom_right", lengths, mode == "speed") is not None
            assert served == (D % 8 == 0 or dtype == torch.float32 and D % 4 == 0)      # rows in 16-byte pieces
            o, lse = fa.flash_attention_v100(q, k, v, causal=causal, return_softmax_lse=True, key_lengths=lengths, causal_alignment=align,
                                             optimization_strategy=mode, enable_multi_gpu=False)
        else:
            o, lse = _general(q, k, v, causal, Nk - Nq if align == "bottom_right" else 0, lengths, mode)
        assert not lse.requires_grad and o.requires_grad == (wants != "none")
        if wants != "none":
            o.backward(g)
        got.append((o.detach(), lse, q.grad, k.grad, v.grad))
    fast_dq = mode == "speed" and dtype != torch.float32 and D == 64
    for n, x, y in zip(("o", "lse", "dq", "dk", "dv"), *got):
        assert (x is None) == (y is None), n
        if x is not None and not (fast_dq and n == "dq"):          # (dQ in no fixed order there)
            assert torch.equal(x, y), n


def test_gradients_of_any_layout_twice_and_under_hooks(device):
    q, k, v = (_rand(2, 100, 4, 64, dtype=torch.bfloat16, device=device, seed=i).requires_grad_(True) for i in range(3))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.to(device)):
        o = fa.flash_attention_v100(q, k, v, causal=True, enable_multi_gpu=False)
    assert len(packed) == 6                                          # q, k, v, o, lse and o's residual
    ref = _general(q, k, v, True)[0]
    for g in (torch.ones((), dtype=q.dtype, device=device).expand_as(o), _rand(2, 4, 100, 64, dtype=q.dtype, device=device, seed=5).transpose(1, 2),
              _rand(2, 100, 4, 128, dtype=q.dtype, device=device, seed=6)[..., ::2]):
        for x, y in zip(torch.autograd.grad(o, (q, k, v), g, retain_graph=True), torch.autograd.grad(ref, (q, k, v), g, retain_graph=True)):
            assert torch.equal(x, y)
    torch.autograd.grad(o.sum(), q)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o.sum(), q)


def test_a_changed_operand_is_noticed(device):
    q, k, v = (_rand(1, 64, 2, 64, dtype=torch.float16, device=device, seed=i).requires_grad_(True) for i in range(3))
    o = fa.flash_attention_v100(q, k, v, enable_multi_gpu=False)
    with torch.no_grad():
        k.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        o.sum().backward()


def test_who_watches_operators_gets_the_general_form(device):
    q = _rand(2, 64, 2, 64, dtype=torch.float16, device=device, seed=1)
    call = lambda t: ops.native_call(t, t, t, None, False, False, None, False)
    assert call(q) is not None
    seen = []
    torch.func.vmap(lambda t: (seen.append(call(t)), t)[1])(q[None])
    torch.func.grad(lambda t: (seen.append(call(t)), t.float().sum())[1])(q)
    with torch.autograd.forward_ad.dual_level():
        seen.append(call(torch.autograd.forward_ad.make_dual(q, q)))

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    with Mode():
        seen.append(call(q))

    class Sub(torch.Tensor):
        pass
    seen.append(call(q.as_subclass(Sub)))
    seen.append(call(q.cpu()))
    seen.append(call(q[..., :0]))
    with ops.kernel_variant("simt"):
        seen.append(call(q))
    assert seen == [None] * 8
    with pytest.raises(RuntimeError):                               # as before: no rule for forward mode
        with torch.autograd.forward_ad.dual_level():
            d = torch.autograd.forward_ad.make_dual(q, q)
            fa.flash_attention_v100(d, d, d, enable_multi_gpu=False)


def test_refusals_keep_their_types(device):
    q = _rand(2, 64, 4, 64, dtype=torch.float16, device=device, seed=1)
    f = lambda *a, **kw: fa.flash_attention_v100(*a, enable_multi_gpu=False, **kw)
    with pytest.raises(ValueError, match="divisible"):
        f(q, q[:, :, :3], q[:, :, :3])
    with pytest.raises(ValueError, match="same dtype"):
        f(q, q.float(), q)
    with pytest.raises(ValueError, match="bottom-right"):
        f(q, q[:, :32], q[:, :32], causal=True, causal_alignment="bottom_right")
    with pytest.raises(ValueError, match="causal_alignment"):
        f(q, q, q, causal_alignment="middle")
    with pytest.raises(ValueError, match="scale is NaN"):
        f(q, q, q, scale=float("nan"))
    with pytest.raises(ValueError, match="key_lengths"):
        f(q, q, q, key_lengths=torch.ones(3, dtype=torch.int32, device=device))


def test_other_threads_run_while_a_call_waits_for_the_launch_queue(device):
    """A kernel of about a second ahead of more calls than the launch queue holds: the calling thread has to wait for
    room, and this one goes on ticking meanwhile.  (With the interpreter held it stood still for most of the second.)"""
    import threading
    import time
    q = _rand(1, 128, 2, 64, dtype=torch.float16, device=device, seed=1)
    assert ops.native_call(q, q, q, None, False, False, None, False) is not None
    torch.cuda.synchronize(device)
    took = []

    def calls():
        start = time.perf_counter()
        with torch.no_grad():
            for _ in range(4000):
                ops.native_call(q, q, q, None, False, False, None, False)
        took.append(time.perf_counter() - start)
    torch.cuda._sleep(1_500_000_000)                                # cycles, 0.8 s or more
    worker = threading.Thread(target=calls)
    gap, last = 0.0, time.perf_counter()
    worker.start()
    while worker.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    worker.join()
    torch.cuda.synchronize(device)
    assert took[0] > 0.5                                            # the queue was full
    assert gap < 0.5 * took[0]
