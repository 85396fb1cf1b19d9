"""ConvolveReal in float32 on overlap-save blocks that share a transform in
pairs: kernel lengths at the edges of every block length, odd and even block
counts, a last block of one sample, unaligned and strided batches."""
import math

import numpy as np
import pytest

import algofft

pytestmark = pytest.mark.gpu

# three chained transforms of at most 2^14 points, each within log2(N) roundings
TOL = 3 * 14 * 2.0 ** -23


def _fp64(a, b):
    n = a.shape[-1] + b.size - 1
    F = 1 << math.ceil(math.log2(n))
    return np.fft.irfft(np.fft.rfft(a.astype(np.float64), F) * np.fft.rfft(b.astype(np.float64), F), F)[..., :n]


def _run(na, nb, count, offset=0, gap=0, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    ad, dd = na + gap, na + nb - 1 + 2 * gap
    a = rng.uniform(-1, 1, (count, ad)).astype(np.float32)
    b = rng.uniform(-1, 1, nb).astype(np.float32)
    ta = torch.zeros(offset + count * ad, device="cuda")
    ta[offset:] = torch.from_numpy(a.ravel()).cuda()
    td = torch.full((offset + count * dd,), 7.0, device="cuda")
    algofft.ConvolveRealBatch(td[offset:], ta[offset:], na, count, torch.from_numpy(b).cuda(), a_dist=ad, dst_dist=dd)
    torch.cuda.synchronize()
    got = td[offset:].cpu().numpy().reshape(count, dd)
    assert np.all(td[:offset].cpu().numpy() == 7) and np.all(got[:, na + nb - 1:] == 7)  # gaps untouched
    return got[:, :na + nb - 1], _fp64(a[:, :na], b)


@pytest.mark.parametrize("na,nb,count", [
    (8193, 1, 3), (8192 + 4096, 2, 1), (4096 * 3, 33, 700), (100003, 513, 2),
    (3 * (4096 - 512) - 512 + 1, 513, 1),         # a last block of one output
    (65537, 2049, 5), (65537, 2050, 5), (66000, 4097, 1), (66000, 4098, 9), (65536 * 2, 8193, 3),
    (1 << 20, 4097, 2), (1 << 19, 1025, 40)])
def test_block_pairs(na, nb, count):
    got, ref = _run(na, nb, count, seed=na + nb)
    for g, r in zip(got, ref):
        assert np.linalg.norm(g - r) <= TOL * np.linalg.norm(r)
        assert np.max(np.abs(g - r)) <= 10 * TOL * np.sqrt(np.mean(r ** 2))


@pytest.mark.parametrize("offset,gap", [(1, 0), (3, 5), (2, 1)])
def test_unaligned_and_strided(offset, gap):
    got, ref = _run(50001, 300, 4, offset=offset, gap=gap, seed=offset)
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


def test_non_finite_samples_stay_in_their_signal_and_blocks():
    import torch
    na, nb, count = 200000, 65, 3
    rng = np.random.default_rng(4)
    a = rng.uniform(-1, 1, (count, na)).astype(np.float32)
    b = rng.uniform(-1, 1, nb).astype(np.float32)
    clean = _fp64(a, b)
    a[1, 100000] = np.inf
    td = torch.empty(count * (na + nb - 1), device="cuda")
    algofft.ConvolveRealBatch(td, torch.from_numpy(a.ravel()).cuda(), na, count, torch.from_numpy(b).cuda())
    got = td.cpu().numpy().reshape(count, -1)
    for i in (0, 2):
        assert np.linalg.norm(got[i] - clean[i]) <= TOL * np.linalg.norm(clean[i])
    bad = ~np.isfinite(got[1])
    assert bad[100000:100000 + nb].all()
    assert not bad[:100000 - 32768].any() and not bad[100000 + nb + 32768:].any()
