"""The allocation-free batched entry point on default complex64 plans
(gfft_plan_new without a variant), at every length that its fixed scratch
holds: 2^15..2^21, with the shipped wisdom and with none, against numpy's FP64
FFT.  Collected after every other file, as test_zz_no_alloc.py is."""
import ctypes

import numpy as np
import pytest

import algofft
from helpers import rel_l2, seeded_complex, tol_c2c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wisdom", [True, False])
@pytest.mark.parametrize("n", [1 << k for k in range(15, 22)])
def test_default_plans(n, wisdom):
    import torch
    saved = algofft.ExportWisdomToString()
    if not wisdom:
        algofft.ClearWisdom()
    count = 3
    x = seeded_complex(n * count, seed=n % 97)
    src = torch.from_numpy(x).cuda()
    got = torch.full_like(src, float("nan"))
    v = x.astype(np.complex128).reshape(count, n)
    try:
        with algofft.NewPlan(n) as p:
            for direction, ref in ((-1, np.fft.fft(v, axis=1)), (1, np.fft.ifft(v, axis=1))):
                s = algofft.lib().gfft_exec_batch_noalloc(
                    p._h, direction, ctypes.c_void_p(got.data_ptr()), got.numel(), ctypes.c_void_p(src.data_ptr()),
                    src.numel(), count, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
                assert s == 0, algofft.lib().gfft_last_error()
                torch.cuda.synchronize()
                p.Check()
                assert rel_l2(got.cpu().numpy(), ref.ravel()) <= tol_c2c(n, False)
    finally:
        algofft.ClearWisdom()
        algofft.ImportWisdomFromString(saved)
