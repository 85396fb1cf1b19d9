"""Where packed-pair kernels do not run although the length has them: a
forced two-pass strategy takes two passes."""
import pytest

import algofft
from helpers import tol_c2c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [algofft.KernelSixStep, algofft.KernelEightStep])
@pytest.mark.parametrize("n", [1 << k for k in (15, 20, 21, 22, 23, 24)])
def test_step_strategies_are_two_pass(n, strategy):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.view_as_complex(torch.randn(n, 2, generator=g, device="cuda"))
    y = torch.empty_like(x)
    with algofft.NewPlanWithOptions(n, algofft.PlanOptions(Strategy=strategy)) as p:
        assert "-tp-" in p.Algorithm()
        p.Forward(y, x)
    ref = torch.fft.fft(x.to(torch.complex128))
    assert float(torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)) <= tol_c2c(n, False)
