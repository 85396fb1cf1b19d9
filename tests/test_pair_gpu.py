"""Packed-pair multi-pass kernels (complex64 2^15..2^24) against the FP64 FFT:
every length, both directions, batches, in place, and buffers
off 16 bytes, which take the scalar kernels of the same split."""
import pytest

import algofft
from helpers import tol_c2c

pytestmark = pytest.mark.gpu

LENGTHS = [1 << k for k in range(15, 25)]


def _token(n):
    return next(t for t in algofft.Variants(n) if t.endswith("-pair"))


def _data(n, count, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.view_as_complex(torch.randn(n * count, 2, generator=g, device="cuda"))


def _err(got, want):
    import torch
    return float(torch.linalg.vector_norm(got - want) / torch.linalg.vector_norm(want))


@pytest.mark.parametrize("n", LENGTHS)
def test_pair_lengths(n):
    import torch
    count = max(1, min(3, (1 << 25) // n))
    x = _data(n, count, n % 997)
    ref = torch.fft.fft(x.view(count, n).to(torch.complex128), dim=1).view(-1)
    y = torch.empty_like(x)
    with algofft.Plan(n, variant=_token(n)) as p:
        assert p.Algorithm() == _token(n)
        p.ForwardBatch(y, x, count)
        assert _err(y, ref) <= tol_c2c(n, False)
        b = torch.empty_like(x)
        p.InverseBatch(b, y, count)
        assert _err(b, x) <= 2 * tol_c2c(n, False)
        z = x.clone()
        p.ForwardBatch(z, z, count)  # in place
        assert torch.equal(torch.view_as_real(z), torch.view_as_real(y))
        one = torch.empty_like(x[:n])
        p.Forward(one, x[:n])
        assert torch.equal(torch.view_as_real(one), torch.view_as_real(y[:n]))


@pytest.mark.parametrize("n", [1 << 15, 1 << 16, 1 << 17, 1 << 18, 1 << 19, 1 << 20, 1 << 21])
def test_pair_small_and_full_grids_agree(n):
    # one transform and a batch on either side of the grid-size rule
    import torch
    for count in (1, 2, 5, 37):
        if n * count > 1 << 25:
            continue
        x = _data(n, count, count)
        ref = torch.fft.ifft(x.view(count, n).to(torch.complex128), dim=1).view(-1)
        y = torch.empty_like(x)
        with algofft.Plan(n, variant=_token(n)) as p:
            for _ in range(3):  # launches that follow one another without a wait
                p.InverseBatch(y, x, count)
        assert _err(y, ref) <= tol_c2c(n, False)


@pytest.mark.parametrize("n", [1 << 15, 1 << 18, 1 << 19, 1 << 21])
def test_pair_unaligned_buffers(n):
    import torch
    x = _data(n + 1, 2, 3)
    ref = torch.fft.fft(x[1:1 + 2 * n].view(2, n).to(torch.complex128), dim=1).view(-1)
    d = torch.full((2 * n + 1,), 9 + 0j, dtype=torch.complex64, device="cuda")
    with algofft.Plan(n, variant=_token(n)) as p:
        p.ForwardBatch(d[1:], x[1:1 + 2 * n], 2)
        assert _err(d[1:], ref) <= tol_c2c(n, False)
        assert complex(d[0].item()) == 9
        aligned = torch.empty(2 * n, dtype=torch.complex64, device="cuda")
        p.ForwardBatch(aligned, x[1:1 + 2 * n], 2)  # only the source is off 16 bytes
        assert _err(aligned, ref) <= tol_c2c(n, False)


def test_pair_is_the_default_and_old_tokens_still_run():
    import torch
    n = 1 << 16
    x = _data(n, 2, 5)
    ref = torch.fft.fft(x.view(2, n).to(torch.complex128), dim=1).view(-1)
    for tok in [None] + [t for t in algofft.Variants(n) if "-tp-" in t]:
        y = torch.empty_like(x)
        with (algofft.Plan(n, variant=tok) if tok else algofft.NewPlan(n)) as p:
            assert tok or p.Algorithm().endswith("-pair")
            p.ForwardBatch(y, x, 2)
        assert _err(y, ref) <= tol_c2c(n, False)


@pytest.mark.parametrize("L", [32, 64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("cols,offset", [(2, 0), (66, 0), (62, 0), (33, 0), (64, 1)])
def test_pair_columns(L, cols, offset):
    # column batches: partial tiles, odd pitches and buffers off 16 bytes (the
    # scalar tile), both directions, out of and in place
    import torch
    x = _data(L * cols + offset, 1, L + cols)[offset:]
    ref = torch.fft.fft(x.view(L, cols).to(torch.complex128), dim=0).reshape(-1)
    y = torch.empty(L * cols + offset, dtype=torch.complex64, device="cuda")[offset:]
    with algofft.NewPlan(L) as p:
        p.StridedBatch(y, x, cols, cols, 1)
        assert _err(y, ref) <= tol_c2c(L, False)
        p.StridedBatch(y, y, cols, cols, 1, inverse=True)
        assert _err(y, x) <= 2 * tol_c2c(L, False)


@pytest.mark.parametrize("n,prec", [(1 << 15, 0), (1 << 18, 0), (1 << 20, 0), (1 << 16, 1), (50421, 0), (100000, 1),
                                    (1 << 21, 1)])
@pytest.mark.parametrize("shift", [0, 2, None])
def test_two_pass_outputs_that_overlap_their_inputs(n, prec, shift):
    # the intermediate lives in dst unless dst shares memory with src (the same
    # buffer, or one that starts a little later); None: separate buffers
    import torch
    count, dt = 3, (torch.complex128 if prec else torch.complex64)
    x = _data(n, count, 11).to(dt)
    ref = torch.fft.fft(x.view(count, n).to(torch.complex128), dim=1).view(-1)
    buf = torch.empty(n * count + 8, dtype=dt, device="cuda")
    src = buf[:n * count] if shift is not None else x
    if shift is not None:
        src.copy_(x)
    dst = buf[shift or 0:(shift or 0) + n * count]
    with algofft.NewPlanT(n, prec) as p:
        p.ForwardBatch(dst, src, count)
    assert _err(dst, ref) <= tol_c2c(n, bool(prec))


@pytest.mark.parametrize("n", [50789, 52433, 58963, 40993])
@pytest.mark.parametrize("prec", [0, 1])
def test_bluestein_splits_of_equal_lengths(n, prec):
    # M = 102400, 107520, 122880, 82944: 256 x 400, 240 x 448, 256 x 480, 192 x 432
    # (complex128 288 x 288), not the most balanced factors
    import torch
    dt = torch.complex128 if prec else torch.complex64
    x = _data(n, 2, n).to(dt)
    ref = torch.fft.ifft(x.view(2, n).to(torch.complex128), dim=1).view(-1)
    y = torch.empty_like(x)
    with algofft.Plan(n, prec, variant=f"gpu-sm100-bluestein-n{n}-mx") as p:
        p.InverseBatch(y, x, 2)
    assert _err(y, ref) <= tol_c2c(4 * n, bool(prec))


@pytest.mark.parametrize("n", [9437, 13007, 16411, 27793, 33013])
@pytest.mark.parametrize("count", [1, 7])
def test_bluestein_pair_passes(n, count):
    # M = 80 x 240, 112 x 240, 144 x 240, 224 x 256, 240 x 288: middle and last
    # passes in pairs or scalar by length; odd n puts every other transform off
    # 16 bytes, and the last pair of an odd n is half there
    import torch
    x = _data(n, count, n)
    ref = torch.fft.fft(x.view(count, n).to(torch.complex128), dim=1).view(-1)
    guard = torch.full((n * count + 2,), 5 + 0j, dtype=torch.complex64, device="cuda")
    y = guard[:n * count]
    with algofft.NewPlan(n) as p:
        p.ForwardBatch(y, x, count)
        assert _err(y, ref) <= tol_c2c(4 * n, False)
        assert (guard[n * count:] == 5).all()
        p.InverseBatch(y, y, count)
        assert _err(y, x) <= 2 * tol_c2c(4 * n, False)


@pytest.mark.parametrize("what", ["uneven", "in_place", "three_pass"])
def test_first_call_of_a_process_can_be_captured(what):
    # a fresh process whose first workspace is needed inside a stream capture
    import os
    import subprocess
    import sys
    body = {
        "uneven": "p = algofft.PlanUneven([65536, 16411, 40013, 1000]); x = c(p.Total()); y = torch.empty_like(x)\n"
                  "p.Forward(y, x)",
        "in_place": "p = algofft.NewPlan(1 << 16); y = c(1 << 16); run(lambda: p.Forward(y, y))",
        "three_pass": "p = algofft.NewPlan(1 << 21); x = c(1 << 21); y = torch.empty_like(x)\n"
                      "run(lambda: p.Forward(y, x))",
    }[what]
    code = ("import sys; sys.path.insert(0, 'algo-fft_b200')\nimport torch, algofft\n"
            "c = lambda n: torch.ones(n, dtype=torch.complex64, device='cuda')\n"
            "def run(f):\n    g = torch.cuda.CUDAGraph()\n    s = torch.cuda.Stream()\n"
            "    with torch.cuda.graph(g, stream=s):\n        f()\n    g.replay()\n"
            + body + "\ntorch.cuda.synchronize()\nassert abs(y[0].item()) > 1\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
