"""The transform calls this library is used for, as measurable cases.

A case is one call (or one forward/inverse pair) through the public entry
points on data that is already on the GPU, with the plan a program keeps
between calls.  Sizes are those of the repository's own configurations and
benchmark, or generic; draw() spreads over the same ranges.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "algo-fft_b200"))
import algofft  # noqa: E402

MAX_ELEMS = 1 << 26  # complex64 elements of the largest drawn batch (512 MiB)


def listed():
    return [
        # one Plan.Forward call on one short vector: the smallest call, all latency
        {"name": "forward_1024", "kind": "c2c", "n": 1024, "count": 1, "prec": 0, "inverse": False},
        # one Plan.Forward call on one long vector
        {"name": "forward_2e20", "kind": "c2c", "n": 1 << 20, "count": 1, "prec": 0, "inverse": False},
        # InverseBatch of frames of 4096 samples (spectral processing of long recordings)
        {"name": "inverse_4096_batch", "kind": "c2c", "n": 4096, "count": 16384, "prec": 0, "inverse": True},
        # ForwardBatch of long records
        {"name": "forward_2e18_batch", "kind": "c2c", "n": 1 << 18, "count": 256, "prec": 0, "inverse": False},
        # InverseBatch of very long records (beyond the two-pass lengths)
        {"name": "inverse_2e22_batch", "kind": "c2c", "n": 1 << 22, "count": 16, "prec": 0, "inverse": True},
        # double precision ForwardBatch
        {"name": "forward_2e16_c128", "kind": "c2c", "n": 1 << 16, "count": 512, "prec": 1, "inverse": False},
        # a 7-smooth length that is not a power of two
        {"name": "forward_10000_batch", "kind": "c2c", "n": 10000, "count": 4096, "prec": 0, "inverse": False},
        # a prime length (Bluestein)
        {"name": "forward_16411_batch", "kind": "c2c", "n": 16411, "count": 1022, "prec": 0, "inverse": False},
        # real frames to spectra and back (PlanReal Forward, then Inverse)
        {"name": "real_4096_round_trip", "kind": "real", "n": 4096, "count": 65536, "prec": 0},
        # a stack of images: Plan2D complex64 4096 x 4096, batch 8
        {"name": "plan2d_4096_batch8", "kind": "nd", "d0": 1, "d1": 4096, "d2": 4096, "count": 8, "real": False,
         "prec": 0, "inverse": False},
        # 64 long real signals filtered with one 4097-tap kernel
        {"name": "convolve_real_64x2e20", "kind": "conv", "n": 1 << 20, "taps": 4097, "count": 64, "prec": 0},
        # thousands of transforms of uneven lengths in one call
        {"name": "uneven_4000", "kind": "uneven", "count": 4000, "lengths_seed": 0, "inverse": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth7(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _is_prime(n):
    return n > 1 and all(n % p for p in range(2, int(n ** 0.5) + 1))


def draw(rng):
    kind = rng.choice(["pow2", "pow2", "pow2", "smooth", "prime", "real", "2d", "3d", "conv", "uneven"])
    prec = 1 if rng.random() < 0.25 else 0
    cap = MAX_ELEMS >> prec
    inverse = rng.random() < 0.5
    if kind in ("pow2", "smooth", "prime"):
        if kind == "pow2":
            n = 1 << rng.randint(4, 24)
        else:
            n = _log_int(rng, 60, 100000 if kind == "smooth" else 131071)
            while not (_smooth7(n) and n & (n - 1) if kind == "smooth" else _is_prime(n)):
                n += 1
        most = max(1, (cap if kind != "prime" else cap // 4) // n)
        return {"kind": "c2c", "n": n, "count": _log_int(rng, 1, most), "prec": prec, "inverse": inverse}
    if kind == "real":
        n = 2 * _log_int(rng, 32, 1 << 16)
        if rng.random() < 0.7:
            n = 1 << (n.bit_length() - 1)
        else:
            while not _smooth7(n):
                n += 2
        return {"kind": "real", "n": n, "count": _log_int(rng, 1, 2 * cap // n), "prec": prec}
    if kind in ("2d", "3d"):
        top = 4096 if kind == "2d" else 256

        def axis():
            d = _log_int(rng, 32, top)
            if rng.random() < 0.6:
                return 1 << (d.bit_length() - 1)
            while not _smooth7(d) or d % 2:
                d += 1
            return d

        d0, d1, d2 = (1 if kind == "2d" else axis()), axis(), axis()
        return {"kind": "nd", "d0": d0, "d1": d1, "d2": d2, "count": _log_int(rng, 1, max(1, (cap >> 1) // (d0 * d1 * d2))),
                "real": rng.random() < 0.5, "prec": prec, "inverse": inverse}
    if kind == "conv":
        n = _log_int(rng, 1 << 14, 1 << 20)
        return {"kind": "conv", "n": n, "taps": _log_int(rng, 33, 4097), "count": _log_int(rng, 1, max(1, (cap >> 1) // n)),
                "prec": prec}
    return {"kind": "uneven", "count": _log_int(rng, 200, 4000), "lengths_seed": rng.randrange(1, 1 << 20),
            "inverse": inverse}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _real(g, count, prec, uniform=False):
    dt = torch.float64 if prec else torch.float32
    if uniform:
        return torch.rand(count, generator=g, device="cuda", dtype=dt) * 2 - 1
    return torch.randn(count, generator=g, device="cuda", dtype=dt)


def _cplx(g, count, prec):
    return torch.view_as_complex(_real(g, 2 * count, prec).view(count, 2))


def _ctype(prec):
    return torch.complex128 if prec else torch.complex64


def _dims(case):
    return [d for d in (case["d0"], case["d1"], case["d2"]) if d > 1]


def _inputs(case, seed):
    """The input tensors of one pass, from the seed alone."""
    g = _gen(seed)
    kind, prec = case["kind"], case.get("prec", 0)
    if kind == "c2c":
        return [_cplx(g, case["n"] * case["count"], prec)]
    if kind == "real":
        return [_real(g, case["n"] * case["count"], prec, uniform=True)]
    if kind == "nd":
        d = _dims(case)
        total = math.prod(d) * case["count"]
        if not case["real"]:
            return [_cplx(g, total, prec)]
        x = _real(g, total, prec)
        if case["inverse"]:  # the spectrum of a real array
            ax = list(range(1, len(d) + 1))
            return [torch.fft.rfftn(x.view(case["count"], *d), dim=ax).contiguous().view(-1)]
        return [x]
    if kind == "conv":
        return [_real(g, case["n"] * case["count"], prec, uniform=True), _real(g, case["taps"], prec, uniform=True)]
    lengths = algofft.uneven_lengths(case["count"], seed=case["lengths_seed"])
    return [_cplx(g, int(lengths.sum()), 0)]


def prepare(case, seed):
    kind, prec = case["kind"], case.get("prec", 0)
    x = _inputs(case, seed)
    s = {"case": case, "x": x}
    if kind == "c2c":
        s["plan"] = algofft.NewPlanT(case["n"], prec)
        s["y"] = torch.empty_like(x[0])
    elif kind == "real":
        n, count = case["n"], case["count"]
        s["plan"] = algofft.NewPlanRealWithOptions(n, algofft.PlanOptions(Batch=count), prec)
        s["y"] = torch.empty(count * (n // 2 + 1), dtype=_ctype(prec), device="cuda")
        s["z"] = torch.empty_like(x[0])
    elif kind == "nd":
        d = _dims(case)
        s["plan"] = algofft.PlanND(d, prec, case["real"], algofft.PlanOptions(Batch=case["count"]))
        if not case["real"]:
            s["y"] = torch.empty_like(x[0])
        elif case["inverse"]:
            s["y"] = torch.empty(case["count"] * math.prod(d), dtype=torch.float64 if prec else torch.float32, device="cuda")
        else:
            s["y"] = torch.empty(case["count"] * math.prod(d[:-1]) * (d[-1] // 2 + 1), dtype=_ctype(prec), device="cuda")
    elif kind == "conv":
        s["y"] = torch.empty(case["count"] * (case["n"] + case["taps"] - 1), dtype=x[0].dtype, device="cuda")
    else:
        s["plan"] = algofft.PlanUneven(algofft.uneven_lengths(case["count"], seed=case["lengths_seed"]))
        s["y"] = torch.empty_like(x[0])
    return s


def run(s):
    case, x, y = s["case"], s["x"], s["y"]
    kind = case["kind"]
    if kind == "c2c":
        p = s["plan"]
        if case["count"] == 1:
            (p.Inverse if case["inverse"] else p.Forward)(y, x[0])
        else:
            (p.InverseBatch if case["inverse"] else p.ForwardBatch)(y, x[0], case["count"])
    elif kind == "real":
        s["plan"].Forward(y, x[0])
        s["plan"].Inverse(s["z"], y)
        return [y, s["z"]]
    elif kind == "conv":
        algofft.ConvolveRealBatch(y, x[0], case["n"], case["count"], x[1])
    else:  # N-D and uneven-length plans
        (s["plan"].Inverse if case["inverse"] else s["plan"].Forward)(y, x[0])
    return y


def exact(case, seed):
    kind = case["kind"]
    x = [v.to(torch.complex128 if v.is_complex() else torch.float64) for v in _inputs(case, seed)]
    if kind == "c2c":
        v = x[0].view(case["count"], case["n"])
        return (torch.fft.ifft(v, dim=1) if case["inverse"] else torch.fft.fft(v, dim=1)).reshape(-1)
    if kind == "real":
        return [torch.fft.rfft(x[0].view(case["count"], case["n"]), dim=1).reshape(-1), x[0]]
    if kind == "nd":
        d, c = _dims(case), case["count"]
        ax = list(range(1, len(d) + 1))
        if not case["real"]:
            v = x[0].view(c, *d)
            return (torch.fft.ifftn(v, dim=ax) if case["inverse"] else torch.fft.fftn(v, dim=ax)).reshape(-1)
        if case["inverse"]:
            return torch.fft.irfftn(x[0].view(c, *d[:-1], d[-1] // 2 + 1), s=d, dim=ax).reshape(-1)
        return torch.fft.rfftn(x[0].view(c, *d), dim=ax).reshape(-1)
    if kind == "conv":
        out, m = case["n"] + case["taps"] - 1, 1
        while m < out:
            m *= 2
        h = torch.fft.rfft(x[1], m)
        rows = x[0].view(case["count"], case["n"])
        return torch.cat([torch.fft.irfft(torch.fft.rfft(r, m) * h, m)[:out] for r in rows])
    lengths = algofft.uneven_lengths(case["count"], seed=case["lengths_seed"])
    v, out, at = x[0].cpu().numpy(), [], 0
    for n in lengths:
        r = v[at:at + n]
        out.append(np.fft.ifft(r) if case["inverse"] else np.fft.fft(r))
        at += n
    return np.concatenate(out)


def work(case):
    """Each input read once and each output written once; 5 n log2 n real
    operations per complex transform of n points (half of that for real
    input), as transforms are commonly counted."""
    kind, es = case["kind"], 16 if case.get("prec", 0) else 8
    if kind == "c2c":
        n, c = case["n"], case["count"]
        return {"bytes": 2 * es * n * c, "flops": 5 * n * math.log2(n) * c}
    if kind == "real":  # forward and inverse
        n, c = case["n"], case["count"]
        return {"bytes": 2 * c * (n * es // 2 + (n // 2 + 1) * es), "flops": 5 * n * math.log2(n) * c}
    if kind == "nd":
        d, c = _dims(case), case["count"]
        n = math.prod(d)
        if not case["real"]:
            return {"bytes": 2 * es * n * c, "flops": 5 * n * math.log2(n) * c}
        return {"bytes": c * (n * es // 2 + n // d[-1] * (d[-1] // 2 + 1) * es), "flops": 2.5 * n * math.log2(n) * c}
    if kind == "conv":
        n, t, c = case["n"], case["taps"], case["count"]
        out = n + t - 1
        return {"bytes": (c * n + t + c * out) * es // 2, "flops": c * (5 * out * math.log2(2 * t) + 3 * out)}
    lengths = algofft.uneven_lengths(case["count"], seed=case["lengths_seed"])
    total = int(lengths.sum())
    return {"bytes": 2 * 8 * total, "flops": float((5 * lengths * np.log2(lengths)).sum())}
