"""ConvolveReal in float32: how far one sample reaches.  Overlap-save blocks
share transforms, so an Inf or the rounding error of a loud stretch enters
outputs beside its own; it stays within the window of one block (the power of
two of at least 8 (taps - 1), at least 4096), wherever it lies in its block,
for one signal and for many."""
import numpy as np
import pytest

import algofft

pytestmark = pytest.mark.gpu

# three chained transforms of at most 2^14 points, each within log2(N) roundings
TOL = 3 * 14 * 2.0 ** -23


def _window(nb):
    w = 4096
    while w < 8 * (nb - 1):
        w *= 2
    return w


@pytest.mark.parametrize("nb,na,count", [(33, 60000, 1), (33, 60000, 300), (513, 60000, 3), (700, 80000, 1),
                                         (1025, 90000, 2), (2049, 200000, 1), (2100, 200000, 40)])
def test_loud_and_non_finite_samples_stay_within_one_window(nb, na, count):
    import torch
    rng = np.random.default_rng(nb)
    b = rng.uniform(-1, 1, nb).astype(np.float32)
    a = rng.uniform(-1, 1, na).astype(np.float32)
    F = 1 << (na + nb).bit_length()
    ref = np.fft.irfft(np.fft.rfft(a.astype(np.float64), F) * np.fft.rfft(b.astype(np.float64), F), F)[:na + nb - 1]
    rms = np.sqrt(np.mean(ref ** 2))
    win = _window(nb)
    o = np.arange(na + nb - 1)
    kb = torch.from_numpy(b).cuda()
    base = torch.from_numpy(a).cuda().repeat(count, 1)
    dst = torch.empty(count * (na + nb - 1), device="cuda")
    for p in range(na // 2, na // 2 + 2 * win, win // 8):
        for bad in (np.inf, 1e7):
            x = base.clone()
            x[count // 2, p] = bad
            algofft.ConvolveRealBatch(dst, x.view(-1), na, count, kb)
            got = dst.view(count, -1)[count // 2].cpu().numpy().astype(np.float64)
            far = (o <= p - win) | (o >= p + win)
            err = np.max(np.abs(got[far] - ref[far]))
            assert err <= 10 * TOL * rms, (p, bad, err)
            assert bad == 1e7 or not np.isfinite(got[p:p + nb]).any()
