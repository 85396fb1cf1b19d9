"""Uneven batches whose Bluestein passes run on packed pairs: every column
length that has them, in launches of at least 296 CTAs (smaller ones take the
scalar tiles), with transforms at odd and even offsets (off 16 bytes, and on
them), forward and inverse, out of and in place, against numpy's FP64 FFT."""
import numpy as np
import pytest

import algofft
from helpers import tol_c2c

pytestmark = pytest.mark.gpu

# length -> (M1, M2) of its FFT length M; the middle pass runs columns of M2,
# the last one columns of M1
SPLITS = {9221: (80, 240), 10369: (112, 192), 8963: (128, 144), 16411: (144, 240), 18427: (192, 192),
          25087: (224, 224), 28669: (224, 256), 28687: (240, 240), 35851: (256, 288), 76801: (400, 400)}
COPIES = 34
PAIRED = {"mid": (192, 224, 240, 256), "out": (80, 112, 128, 144, 192, 224, 240, 256, 400)}


def test_launches_are_large_enough():
    ctas = {}
    for m1, m2 in SPLITS.values():
        ctas["mid", m2] = ctas.get(("mid", m2), 0) + COPIES * m1 // 16
        ctas["out", m1] = ctas.get(("out", m1), 0) + COPIES * m2 // 16
    for kind, lengths in PAIRED.items():
        for L in lengths:
            assert ctas[kind, L] >= 2 * 148, (kind, L, ctas[kind, L])


@pytest.mark.parametrize("inverse", [False, True])
def test_paired_items(inverse):
    import torch
    rng = np.random.default_rng(3)
    lengths = np.array(list(SPLITS) * COPIES)
    rng.shuffle(lengths)
    starts = np.concatenate([[0], np.cumsum(lengths)])
    odd = {int(n): {int(s) & 1 for s, m in zip(starts, lengths) if m == n} for n in SPLITS}
    assert all(v == {0, 1} for v in odd.values())  # each length on and off 16 bytes
    g = torch.Generator(device="cuda")
    g.manual_seed(4)
    x = torch.view_as_complex(torch.randn(int(starts[-1]), 2, generator=g, device="cuda"))
    y = torch.empty_like(x)
    z = x.clone()
    with algofft.PlanUneven(lengths) as p:
        run = p.Inverse if inverse else p.Forward
        run(y, x)
        run(z, z)
    assert torch.equal(torch.view_as_real(z), torch.view_as_real(y))
    xs, ys = x.cpu().numpy().astype(np.complex128), y.cpu().numpy()
    for i, n in enumerate(lengths):
        a, b = starts[i], starts[i + 1]
        ref = np.fft.ifft(xs[a:b]) if inverse else np.fft.fft(xs[a:b])
        assert np.linalg.norm(ys[a:b] - ref) <= 2 * tol_c2c(4 * int(n), False) * np.linalg.norm(ref), (i, n)
