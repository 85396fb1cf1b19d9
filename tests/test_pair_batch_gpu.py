"""Packed-pair passes on few and on many tiles: batches too small for the SMs
take narrower tiles of the same stages, so a transform is the same bits alone
and in a batch, both directions, at every two-pass length."""
import pytest

import algofft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("n", [1 << k for k in range(15, 21)])
def test_alone_and_in_a_batch(n, inverse):
    # a pass has n / 4096 to n / 8192 tiles of its wide form per transform, and
    # takes that from 128 tiles on
    import torch
    count = 2 * 128 * 8192 // n + 2
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.view_as_complex(torch.randn(n * count, 2, generator=g, device="cuda"))
    y = torch.empty_like(x)
    one = torch.empty_like(x[:n])
    with algofft.NewPlan(n) as p:
        assert p.Algorithm().endswith("-pair")
        (p.InverseBatch if inverse else p.ForwardBatch)(y, x, count)
        for i in (0, 1, count - 1):
            (p.Inverse if inverse else p.Forward)(one, x[i * n:(i + 1) * n])
            assert torch.equal(torch.view_as_real(one), torch.view_as_real(y[i * n:(i + 1) * n]))
