"""Where packed-pair kernels do not run: a forced two-pass strategy takes two
passes, and columns of 128 rows stay on the scalar tile."""
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


@pytest.mark.parametrize("cols", [32, 66, 250])
def test_columns_of_128_rows_stay_scalar(cols):
    # the scalar tile runs arrays off 16 bytes (the odd pitch), so its results
    # are the same bits on aligned arrays
    import torch
    L = 128
    g = torch.Generator(device="cuda")
    g.manual_seed(cols)
    x = torch.view_as_complex(torch.randn(L * cols, 2, generator=g, device="cuda")).view(L, cols)
    wide = torch.zeros(L, cols + 1, dtype=torch.complex64, device="cuda")
    wide[:, :cols] = x
    wide = wide.view(-1)
    y = torch.empty(L * cols, dtype=torch.complex64, device="cuda")
    z = torch.empty_like(wide)
    ref = torch.fft.fft(x.to(torch.complex128), dim=0).reshape(-1)
    with algofft.NewPlan(L) as p:
        p.StridedBatch(y, x.reshape(-1), cols, cols, 1)
        p.StridedBatch(z, wide, cols, cols + 1, 1)
    assert torch.equal(torch.view_as_real(z.view(L, cols + 1)[:, :cols].reshape(-1)), torch.view_as_real(y))
    assert float(torch.linalg.vector_norm(y - ref) / torch.linalg.vector_norm(ref)) <= tol_c2c(L, False)
