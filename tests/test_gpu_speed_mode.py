"""optimization_strategy="speed": a preference that calls without a faster kernel of that kind run without."""
import pytest
import torch

import flash_attention_v100 as fa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D,biased", [(torch.bfloat16, 96, False), (torch.float16, 40, False), (torch.float32, 64, False), (torch.float32, 48, False),
                                            (torch.float16, 128, False), (torch.bfloat16, 64, True), (torch.float16, 20, False)])
def test_a_training_step_of_every_kind(device, dtype, D, biased):
    gen = torch.Generator().manual_seed(D)
    q, k, v, g = (torch.randn(2, 130, 2, D, generator=gen).to(device=device, dtype=dtype) for _ in range(4))
    bias = torch.randn(1, 2, 130, 130, generator=gen).to(device) if biased else None

    def step(strategy):
        leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
        out = fa.flash_attention_v100(*leaves, causal=True, bias=bias, optimization_strategy=strategy, enable_multi_gpu=False)
        return (out,) + torch.autograd.grad(out, leaves, g)
    assert all(torch.equal(a, b) for a, b in zip(step("speed"), step("balanced")))
