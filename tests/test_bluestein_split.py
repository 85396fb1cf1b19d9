"""The mixed Bluestein FFT length and its split (gfft_bssplit.h, pure host
C++, built with g++): the smallest product of two factor lengths for every n,
its most balanced split with the first factor within 256 (complex64) or 288
(complex128) rows where one exists; and the primes of the GPU tests run every
factor length in every role that the rule gives it."""
import importlib
import importlib.util
import math
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "algo-fft_b200", "csrc")


def _lengths():
    spec = importlib.util.spec_from_file_location("gen_mixcols", os.path.join(CSRC, "gen_mixcols.py"))
    g = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(g)
    return g.bs_lengths()


@pytest.fixture(scope="module")
def splits(tmp_path_factory):
    """[prec] -> list of (first n, last n, M, M1)"""
    exe = str(tmp_path_factory.mktemp("split") / "bluestein_split_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "bluestein_split_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe] + [str(L) for L in _lengths()], capture_output=True, text=True, check=True, timeout=120)
    rows = [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]
    res = []
    for prec in (0, 1):
        r = [(n, M, m1) for p, n, M, m1 in rows if p == prec]
        res.append([(n, (r[i + 1][0] if i + 1 < len(r) else 131073) - 1, M, m1) for i, (n, M, m1) in enumerate(r)])
    return res


def test_smallest_product(splits):
    bs = _lengths()
    products = sorted({a * b for a in bs for b in bs})
    for prec in (0, 1):
        for lo, hi, M, m1 in splits[prec]:
            assert m1 in bs and M // m1 in bs and M % m1 == 0
            for n in (lo, hi):
                assert M == next(m for m in products if m >= 2 * n - 1)


@pytest.mark.parametrize("prec,wide", [(0, 256), (1, 288)])
def test_split_is_balanced_within_the_bound_on_m1(splits, prec, wide):
    bs = _lengths()
    for _, _, M, m1 in splits[prec]:
        fits = [a for a in bs if M % a == 0 and M // a in bs and a <= math.isqrt(M)]
        assert m1 == max([a for a in fits if a <= wide] or fits), (M, m1)


def test_gpu_primes_cover_every_factor_role(splits):
    sweep = importlib.import_module("test_mixcols_sweep_gpu").BS_PRIMES
    extra = importlib.import_module("test_bluestein_split_gpu").PRIMES
    for prec in (0, 1):
        reach, got = set(), set()
        for lo, hi, M, m1 in splits[prec]:
            primes = [n for n in range(lo, hi + 1) if all(n % d for d in range(2, math.isqrt(n) + 1))]
            for n in primes:
                if M < 1 << (2 * n - 2).bit_length():
                    roles = {(m1, 1), (M // m1, 2)}
                    reach |= roles
                    if n in sweep or n in extra[prec]:
                        got |= roles
        assert got == reach, (prec, reach - got)
