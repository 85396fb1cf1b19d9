"""Bluestein on mixed FFT lengths whose split differs between the precisions,
or whose factor no prime of the sweep reaches in that role, against numpy's
FP64 FFT: complex64 M1 = 288 (288 x 432 for n = 61441), complex128 384 x 400,
320 x 432 and 384 x 384."""
import numpy as np
import pytest

import algofft
from helpers import rel_l2, seeded_complex, tol_c2c

pytestmark = pytest.mark.gpu

PRIMES = {0: [61441], 1: [75269, 68023, 73013]}  # precision -> lengths


@pytest.mark.parametrize("prec,n", [(p, n) for p in PRIMES for n in PRIMES[p]])
def test_split(prec, n):
    import torch
    count = 3
    x = seeded_complex(n * count, seed=n % 997, dtype=np.complex128 if prec else np.complex64)
    src = torch.from_numpy(x).cuda()
    dst = torch.empty_like(src)
    with algofft.Plan(n, prec, variant=f"gpu-sm100-bluestein-n{n}-mx") as p:
        p.ForwardBatch(dst, src, count)
        y = dst.cpu().numpy()
    ref = np.fft.fft(x.astype(np.complex128).reshape(count, n), axis=1).ravel()
    assert rel_l2(y, ref) <= 2 * tol_c2c(1 << (2 * n - 2).bit_length(), bool(prec))
