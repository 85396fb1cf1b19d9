"""Kernels that exist with evict-first and with default input reads, chosen by
the bytes a call moves: a transform's result is the same bits in a batch on
either side of the line, and right on both."""
import numpy as np
import pytest

import algofft
from helpers import tol_c2c

pytestmark = pytest.mark.gpu


def _data(count, seed, prec=0):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.view_as_complex(torch.randn(count, 2, generator=g, device="cuda",
                                             dtype=torch.float64 if prec else torch.float32))


@pytest.mark.parametrize("n,prec", [(65521, 0), (40009, 1)])
@pytest.mark.parametrize("inverse", [False, True])
def test_power_of_two_bluestein(n, prec, inverse):
    # M = 131072: more than 256 MiB of input, output and intermediates, or less
    import torch
    M, es = 131072, 16 if prec else 8
    many = (256 << 20) // (2 * (n + M) * es) + 2
    x = _data(n * many, n, prec)
    y = torch.empty_like(x)
    with algofft.Plan(n, prec, variant=f"gpu-sm100-bluestein-n{n}-p2") as p:
        run = p.InverseBatch if inverse else p.ForwardBatch
        run(y, x, many)
        few = torch.empty_like(x[:3 * n])
        run(few, x[-3 * n:], 3)
    assert torch.equal(torch.view_as_real(few), torch.view_as_real(y[-3 * n:]))
    v = x[-3 * n:].view(3, n).to(torch.complex128)
    ref = (torch.fft.ifft(v, dim=1) if inverse else torch.fft.fft(v, dim=1)).view(-1)
    assert float(torch.linalg.vector_norm(few - ref) / torch.linalg.vector_norm(ref)) <= 2 * tol_c2c(M, bool(prec))


@pytest.mark.parametrize("lengths", [[16411], [65521, 65536]])
def test_uneven_items(lengths):
    # plans that move less than 64 MiB, 64 to 512 MiB and more
    import torch
    unit = np.array(lengths * 10)
    size = int(unit.sum())
    x = _data(size * 84, 7)
    got = []
    for reps in ((4, 12, 84) if len(lengths) == 1 else (1, 4, 20)):
        y = torch.empty_like(x[:size * reps])
        with algofft.PlanUneven(np.tile(unit, reps)) as p:
            p.Forward(y, x[:size * reps])
        got.append(y[:size])
    ref = np.concatenate([np.fft.fft(r) for r in np.split(x[:size].cpu().numpy().astype(np.complex128),
                                                          np.cumsum(unit)[:-1])])
    for y in got:
        assert torch.equal(torch.view_as_real(y), torch.view_as_real(got[0]))
        assert np.linalg.norm(y.cpu().numpy() - ref) <= 2 * tol_c2c(131072, False) * np.linalg.norm(ref)
