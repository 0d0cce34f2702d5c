"""The work that programs using mpsft_gb300 have it do, as measurable cases.

Each case is one call of a public entry point on inputs that the program
already holds (device-resident samples, a context, draws):

  bin      BinInTime::Run (mpsft_bin_in_time): the drop-in binner
  freq     BinInFreq::Run (mpsft_bin_in_freq): the other drop-in binner
  est, adj the coefficient estimate of a fixed set and its adjoint (gradients)
  iter     Iterate (mpsft_iterate_draws), as the adapter's IterateGPU calls it
  solve    Demo1::Run (mpsft_solve, mpsft_solve_batched_packed), one signal or
           many

Sizes follow this repository's configurations, tests and benchmark: lengths
2^16 .. 2^26 (powers of two and the primes below them), 51 .. 8001 bins,
window delta 1e-5 and 1e-6, complex64 and complex128, both precisions, one
and several trials. Results land in buffers that the caller holds (sized for
the most modes a call may return, zero past the last one) or in the arrays the
binding returns. Bins and single-iteration coefficients of FP32 precision are
kept as complex64, everything else as complex128.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import mpsft_gb300 as m

# the largest primes below 2^16 .. 2^26 (the reference's benchmark lengths)
_PRIMES = {16: 65521, 17: 131071, 18: 262139, 19: 524287, 20: 1048573, 21: 2097143,
           22: 4194301, 23: 8388593, 24: 16777213, 25: 33554393, 26: 67108859}
_CTX = None


def _ctx():
    """The context a program keeps for its lifetime."""
    global _CTX
    if _CTX is None:
        _CTX = m.Context(0)
    return _CTX


def _length(log2n: int, prime: bool) -> int:
    return _PRIMES[log2n] if prime else 1 << log2n


def _bits(n: int, bins: int) -> int:
    """NumBits: halvings of n while n >= bins."""
    if n < bins:
        return 1
    out = 0
    while n >= bins:
        n >>= 1
        out += 1
    return out


def listed():
    return [
        # one binner call of a small problem: nothing but latency
        {"name": "bin_small", "kind": "bin", "log2n": 16, "prime": True, "bins": 51,
         "bits": 11, "delta": 1e-5, "c128": False, "fp64": False, "device_out": False},
        # the reference's BinInTime benchmark shape, mixed precision
        {"name": "bin_bm_fp32", "kind": "bin", "log2n": 22, "prime": True, "bins": 501,
         "bits": 15, "delta": 1e-6, "c128": False, "fp64": False, "device_out": False},
        # the same, as the drop-in adapter runs it by default: FP64 throughout
        {"name": "bin_bm_fp64", "kind": "bin", "log2n": 22, "prime": True, "bins": 501,
         "bits": 15, "delta": 1e-6, "c128": True, "fp64": True, "device_out": False},
        # the first binning of the 512 MiB stress signal, bins left on the device
        {"name": "bin_large", "kind": "bin", "log2n": 26, "prime": False, "bins": 8001,
         "bits": 14, "delta": 1e-5, "c128": False, "fp64": False, "device_out": True},
        # the reference's BinInFreq benchmark shape
        {"name": "freq_bm", "kind": "freq", "log2n": 22, "prime": True, "bins": 501,
         "bits": 15, "delta": 1e-6, "modes": 100},
        # the differentiation workload: forward and backward
        {"name": "estimate", "kind": "est", "log2n": 20, "prime": False, "bins": 401,
         "delta": 1e-5, "modes": 200, "trials": 1, "c128": False},
        {"name": "adjoint", "kind": "adj", "log2n": 20, "prime": False, "bins": 401,
         "delta": 1e-5, "modes": 200, "trials": 1},
        # one mixed-precision Iterate of the headline signal, half of it found
        {"name": "iterate_fp32", "kind": "iter", "log2n": 22, "prime": False, "bins": 1001,
         "modes": 1000, "found": 500, "trials": 1, "c128": False, "fp64": False},
        # Iterate with three trials in FP64, the plain single-signal workload
        {"name": "iterate_fp64", "kind": "iter", "log2n": 20, "prime": False, "bins": 101,
         "modes": 50, "found": 10, "trials": 3, "c128": True, "fp64": True},
        # a whole recovery of one headline signal
        {"name": "solve_one", "kind": "solve", "count": 1, "lo": 22, "hi": 22,
         "modes_lo": 1000, "modes_hi": 1000, "unit": False, "c128": False, "fp64": False,
         "trials": 1, "shapes": 0},
        # the headline workload: 64 recoveries in one call
        {"name": "solve_batch", "kind": "solve", "count": 64, "lo": 22, "hi": 22,
         "modes_lo": 1000, "modes_hi": 1000, "unit": False, "c128": False, "fp64": False,
         "trials": 1, "shapes": 0},
        # an uneven batch of nearly noiseless signals (FP64 by the precision policy)
        {"name": "solve_uneven", "kind": "solve", "count": 24, "lo": 16, "hi": 24,
         "modes_lo": 10, "modes_hi": 2000, "unit": True, "c128": False, "fp64": False,
         "trials": 1, "shapes": 3},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bin", "bin", "bin", "freq", "est", "adj", "iter", "iter", "solve",
                       "solve"])
    prime = rng.random() < 0.4
    delta = rng.choice([1e-5, 1e-6])
    if kind == "bin":
        log2n = rng.randint(16, 26)
        fp64 = rng.random() < 0.4
        top = min(4001 if fp64 else 8001, (1 << log2n) // 64)
        bins = _log_int(rng, 51, top) | 1
        n = _length(log2n, prime)
        return {"kind": kind, "log2n": log2n, "prime": prime, "bins": bins,
                "bits": _bits(n, bins), "delta": delta,
                "c128": log2n <= 24 and rng.random() < (0.7 if fp64 else 0.2),
                "fp64": fp64, "device_out": rng.random() < 0.4}
    if kind == "freq":
        log2n = rng.randint(16, 26)
        bins = _log_int(rng, 51, min(4001, (1 << log2n) // 64)) | 1
        return {"kind": kind, "log2n": log2n, "prime": prime, "bins": bins,
                "bits": _bits(_length(log2n, prime), bins), "delta": delta,
                "modes": _log_int(rng, 10, 4000)}
    if kind in ("est", "adj"):
        log2n = rng.randint(16, 22)
        modes = _log_int(rng, 10, 1000)
        case = {"kind": kind, "log2n": log2n, "prime": prime,
                "bins": max(51, 2 * modes + 1), "delta": delta, "modes": modes,
                "trials": rng.choice([1, 1, 3])}
        if kind == "est":
            case["c128"] = rng.random() < 0.5
        return case
    if kind == "iter":
        log2n = rng.randint(16, 24)
        modes = _log_int(rng, 10, min(2000, (1 << log2n) // 128))
        found = rng.randint(0, modes - 1)
        fp64 = rng.random() < 0.5
        return {"kind": kind, "log2n": log2n, "prime": prime,
                "bins": max(51, 2 * (modes - found) + 1), "modes": modes, "found": found,
                "trials": rng.choice([1, 1, 3]),
                "c128": fp64 and rng.random() < 0.5, "fp64": fp64}
    lo = rng.randint(16, 22)
    hi = min(24, lo + rng.choice([0, 0, 2]))
    modes = _log_int(rng, 10, min(1000, (1 << lo) // 128))
    fp64 = rng.random() < 0.4
    return {"kind": "solve", "count": _log_int(rng, 1, 32), "lo": lo, "hi": hi,
            "modes_lo": max(10, modes // 2), "modes_hi": modes, "unit": rng.random() < 0.4,
            "c128": fp64 and rng.random() < 0.5, "fp64": fp64,
            "trials": rng.choice([1, 1, 1, 3]), "shapes": rng.randint(0, 1 << 20)}


# ------------------------------------------------------------------ inputs
def _modes(g: np.random.Generator, n: int, count: int, unit: bool):
    """Distinct positions, and coefficients of modulus 1 or log-uniform in
    [1e-2, 1] with uniform phase."""
    k = np.sort(g.choice(n, count, replace=False)).astype(np.int32)
    mag = np.ones(count) if unit else np.exp(g.uniform(math.log(1e-2), 0.0, count))
    return k, mag * np.exp(2j * np.pi * g.uniform(size=count))


def _sigma(c: np.ndarray, unit: bool) -> float:
    """1e-6 per sample with unit modes, else 60 dB SNR."""
    return 1e-6 if unit else float(1e-3 * np.sqrt(np.sum(np.abs(c) ** 2)))


def _samples(n: int, k, c, sigma: float, seed: int, c128: bool) -> torch.Tensor:
    """x_t = sum_j c_j e^{2 pi i k_j t / n} + complex Gaussian noise."""
    xh = torch.zeros(n, dtype=torch.complex128, device="cuda")
    xh[torch.from_numpy(k.astype(np.int64)).cuda()] = torch.from_numpy(c).cuda()
    x = torch.fft.ifft(xh, norm="forward")
    del xh
    g = torch.Generator(device="cuda").manual_seed(seed)
    noise = torch.randn(n, 2, generator=g, dtype=torch.float32, device="cuda")
    x += sigma / math.sqrt(2.0) * torch.view_as_complex(noise)
    return x if c128 else x.to(torch.complex64)


def _transform(g: np.random.Generator, n: int, trials: int):
    """(a, b, c, a_inv) with a invertible mod n, and the trials' q."""
    a, b, c = int(g.integers(1, n)), int(g.integers(0, n)), int(g.integers(0, n))
    if n & (n - 1) == 0:
        a |= 1
    return a, b, c, pow(a, -1, n), [int(v) for v in g.integers(0, n, trials)]


def _inputs(case, seed):
    """Everything of a single-signal case that depends on the seed."""
    n = _length(case["log2n"], case["prime"])
    g = np.random.default_rng([seed, n])
    d = {"n": n, "tf": _transform(g, n, case.get("trials", 1))}
    count = case.get("modes", max(1, case["bins"] // 2))
    unit = case["kind"] in ("est", "adj", "freq") or case.get("c128", False)
    d["k"], d["c"] = _modes(g, n, count, unit)
    d["sigma"] = _sigma(d["c"], unit)
    if case["kind"] == "freq":
        rows = 1 + 2 * case["bits"]
        shape = (rows, case["bins"])
        d["u"] = 0.1 * (g.standard_normal(shape) + 1j * g.standard_normal(shape))
    elif case["kind"] == "adj":
        d["g"] = g.standard_normal(count) + 1j * g.standard_normal(count)
    else:
        d["x"] = _samples(n, d["k"], d["c"], d["sigma"], seed, case["c128"])
    if case["kind"] == "iter":
        # the modes found so far (estimates, not exact values)
        f = np.sort(g.choice(count, case["found"], replace=False))
        d["fk"] = d["k"][f]
        d["fc"] = d["c"][f] + 0.1 * d["sigma"] / math.sqrt(n) * (
            g.standard_normal(f.size) + 1j * g.standard_normal(f.size))
        d["bin_thr"] = 3.0 * d["sigma"] / math.sqrt(case["bins"])
        d["sv_thr"] = d["sigma"] / math.sqrt(case["bins"])
    return d


def _wrap(ctx, x: torch.Tensor):
    return ctx.wrap_device(x.data_ptr(), x.numel(),
                           m.C128 if x.dtype == torch.complex128 else m.C64)


def prepare(case, seed):
    ctx = _ctx()
    s = {"case": case, "ctx": ctx}
    if case["kind"] == "solve":
        s.update(x=[], sig=[], opt=[], rng=[], seeds=[])
        shapes = np.random.default_rng([17, case["shapes"]])
        g = np.random.default_rng([seed, 91])
        for i in range(case["count"]):
            n = 1 << int(shapes.integers(case["lo"], case["hi"] + 1))
            count = int(shapes.integers(case["modes_lo"], case["modes_hi"] + 1))
            k, c = _modes(g, n, count, case["unit"])
            sigma = _sigma(c, case["unit"])
            x = _samples(n, k, c, sigma, int(g.integers(1 << 31)), case["c128"])
            s["x"].append(x)
            s["sig"].append(_wrap(ctx, x))
            s["opt"].append(ctx.solve_options(
                count, sigma, trials=case["trials"], min_bins=51, window_delta=1e-5,
                window_threshold=0.1, max_stale_iter=5,
                precision=m.FP64 if case["fp64"] else m.FP32))
            s["seeds"].append(int(g.integers(1, 1 << 30)))
            s["rng"].append(m.Rng(s["seeds"][-1]))
        # the arrays a C caller passes: handles, options, packed results
        count = case["count"]
        cap = sum(3 * o.k + 256 for o in s["opt"])
        s["sigs"] = (ctypes.c_void_p * count)(*[v._h.value for v in s["sig"]])
        s["rngs"] = (ctypes.c_void_p * count)(*[v._h.value for v in s["rng"]])
        s["opts"] = (m.SolveOptions * count)(*s["opt"])
        s["stats"] = (m.Stats * count)()
        s["seeds"] = np.array(s["seeds"], np.int32)
        s["k"], s["c"] = np.zeros(cap, np.int32), np.zeros(cap, np.complex128)
        s["offsets"], s["count"] = np.zeros(count + 1, np.int64), np.zeros(count, np.int32)
        torch.cuda.synchronize()
        return s
    s.update(_inputs(case, seed))
    if "x" in s:
        s["sig"] = _wrap(ctx, s["x"])
    if case["kind"] == "bin" and case["device_out"]:
        s["out"] = torch.empty(1 + 2 * case["bits"], case["bins"], dtype=torch.complex128,
                               device="cuda")
    if case["kind"] in ("est", "adj"):
        a, b, c, _, q = s["tf"]
        s["setup"] = ctx.estimate_setup(case["bins"], _bits(s["n"], case["bins"]),
                                        case["delta"], a, b, c, q)
    if case["kind"] == "iter":
        cap = s["fk"].size + case["bins"] + 16
        s["mm_k"], s["mm_c"] = np.zeros(cap, np.int32), np.zeros(cap, np.complex128)
        s["size"], s["found"] = np.zeros(1, np.int32), np.zeros(1, np.int32)
        s["q"] = np.array(s["tf"][4], np.int32)
        s["iopt"] = m.IterateOptions(case["bins"], 1e-5, case["trials"], s["bin_thr"], 0.1,
                                     s["sv_thr"], m.FP64 if case["fp64"] else m.FP32, 0.0)
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- run
def _check(rc):
    if rc != m.OK:
        raise m.MpsftError(rc, "call failed")


def _vp(a: np.ndarray):
    return a.ctypes.data_as(ctypes.c_void_p)


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "solve":
        lib = m.load_library()
        _check(lib.mpsft_rng_seed_many(s["rngs"], _vp(s["seeds"]), case["count"]))
        if case["count"] == 1:
            _check(lib.mpsft_solve(ctx._h, s["sigs"][0], s["opts"], s["rngs"][0], _vp(s["k"]),
                                   _vp(s["c"]), s["k"].size, _vp(s["count"]), s["stats"]))
            return {"k": s["k"], "c": s["c"], "count": s["count"]}
        _check(lib.mpsft_solve_batched_packed(
            ctx._h, s["sigs"], s["opts"], case["count"], s["rngs"], _vp(s["k"]), _vp(s["c"]),
            s["k"].size, _vp(s["offsets"]), _vp(s["count"]), s["stats"]))
        return {"k": s["k"], "c": s["c"], "count": s["count"]}
    if kind == "est":
        return ctx.estimate(s["sig"], s["setup"], s["k"])
    if kind == "adj":
        return ctx.adjoint(s["n"], s["setup"], s["k"], s["g"])
    a, b, c, a_inv, q = s["tf"]
    if kind == "freq":
        return ctx.bin_in_freq(s["u"], s["n"], case["bins"], case["bits"], case["delta"], a, b,
                               c, q[0], s["k"], s["c"])
    if kind == "bin":
        prec = m.FP64 if case["fp64"] else m.FP32
        if case["device_out"]:
            _check(m.load_library().mpsft_bin_in_time(
                ctx._h, s["sig"]._h, case["bins"], case["bits"], case["delta"], a, b, c, q[0],
                prec, ctypes.c_void_p(s["out"].data_ptr()), 1))
            u = s["out"]
            return u if case["fp64"] else u.to(torch.complex64)
        u = ctx.bin_in_time(s["sig"], case["bins"], case["bits"], case["delta"], a, b, c, q[0],
                            prec)
        return u if case["fp64"] else u.astype(np.complex64)
    # Iterate on outside draws; the mode map goes in and out
    f = s["fk"].size
    s["mm_k"][:f], s["mm_k"][f:] = s["fk"], 0
    s["mm_c"][:f], s["mm_c"][f:] = s["fc"], 0
    s["size"][0] = f
    _check(m.load_library().mpsft_iterate_draws(
        ctx._h, s["sig"]._h, ctypes.byref(s["iopt"]), a, b, c, a_inv, _vp(s["q"]),
        _vp(s["mm_k"]), _vp(s["mm_c"]), _vp(s["size"]), s["mm_k"].size, _vp(s["found"])))
    return {"k": s["mm_k"], "size": s["size"],
            "c": s["mm_c"] if case["fp64"] else s["mm_c"].astype(np.complex64)}


# -------------------------------------------------------------------- work
def _support(bins: int, delta: float) -> int:
    """Window support p (an odd number of folds of the bins)."""
    sq = math.sqrt(-math.log(delta))
    sigma_t = 1.0 / (2.0 * math.pi * (0.5 / (bins * 2.0 * math.sqrt(2.0) * sq)))
    f = math.ceil((2.0 * math.sqrt(2.0) * sigma_t * sq + 1.0) / bins)
    return (f | 1) * bins


def work(case):
    """Each sample that the rows' windows cover read once (at most the whole
    signal), results written once; a complex multiply-add per gathered sample
    and 5 B log2 B per size-B transform."""
    if case["kind"] == "solve":
        shapes = np.random.default_rng([17, case["shapes"]])
        by = fl = 0.0
        for _ in range(case["count"]):
            n = 1 << int(shapes.integers(case["lo"], case["hi"] + 1))
            k = int(shapes.integers(case["modes_lo"], case["modes_hi"] + 1))
            b = max(51, 2 * k + 1)
            rows = case["trials"] * (1 + 2 * _bits(n, b))
            p = _support(b, 1e-5)
            by += min(n, rows * p) * (16 if case["c128"] else 8) + 20 * k
            fl += rows * (8.0 * p + 5.0 * b * math.log2(b))
        return {"bytes": by, "flops": fl}
    n, b = _length(case["log2n"], case["prime"]), case["bins"]
    bits = case.get("bits", _bits(n, b))
    rows = case.get("trials", 1) * (1 + 2 * bits)
    if case["kind"] == "freq":
        return {"bytes": 32.0 * rows * b + 20.0 * case["modes"],
                "flops": 14.0 * rows * case["modes"]}
    p = _support(b, case.get("delta", 1e-5))
    fl = rows * (8.0 * p + 5.0 * b * math.log2(b))
    covered = min(n, rows * p)
    if case["kind"] == "adj":
        return {"bytes": 16.0 * n + 20.0 * case["modes"], "flops": fl}
    by = covered * (16 if case["c128"] else 8)
    if case["kind"] == "bin":
        by += 16 * rows * b
    else:
        by += 20 * case["modes"]
    return {"bytes": float(by), "flops": fl}


# ------------------------------------------------------------------- exact
def _unit(num: torch.Tensor, n: int) -> torch.Tensor:
    """e^{2 pi i num / n} for integers num, reduced exactly."""
    ph = (num % n).double() * (2.0 * math.pi / n)
    return torch.complex(torch.cos(ph), torch.sin(ph))


class _Window:
    def __init__(self, bins, delta):
        sq = math.sqrt(-math.log(delta))
        self.bins, self.p = bins, _support(bins, delta)
        self.p2 = (self.p - 1) // 2
        self.w = 1.0 / (2.0 * bins)
        self.sigma_f = 0.5 / (bins * 2.0 * math.sqrt(2.0) * sq)
        self.t = torch.arange(-self.p2, self.p2 + 1, device="cuda")
        t = self.t.double()
        self.wt = self.w * torch.sinc(t * self.w) * torch.exp(
            -2.0 * (math.pi * self.sigma_f * t) ** 2)

    def in_freq(self, xi):
        d = math.sqrt(2.0) / (2.0 * self.sigma_f)
        h = 0.5 * self.w
        return 0.5 * (torch.erf((xi + h) * d) - torch.erf((xi - h) * d))


def _offsets(bins, bits):
    out = [0]
    for s in range(bits):
        out += [bins << s, -(bins << s)]
    return out


def _bins_of(x, n, w, bits, a, b, c, q):
    """The (1 + 2 bits) x bins bin matrix in FP64."""
    rows = []
    roll = _unit(-w.t, 2 * w.bins)
    for off in _offsets(w.bins, bits):
        u = (q + off + w.t) % n
        y = x[(a * u + c) % n].to(torch.complex128) * w.wt
        y = y * _unit(b * ((off + w.t) % n), n) * roll
        fold = y.view(-1, w.bins).sum(0)
        rows.append(torch.roll(fold, int(-w.p2 % w.bins)))
    f = torch.fft.fft(torch.stack(rows))
    return f * _unit(torch.tensor([b * q], device="cuda"), n)


def _setup_modes(w, n, bins, a, b, k0):
    """k1, bin and window response of modes k0."""
    k1 = (a * k0 + b) % n
    beta = (k1 * bins) // n
    # k1/n - (beta + 1/2)/bins from its exact numerator
    xi = (2 * bins * k1 - (2 * beta + 1) * n).double() / (2.0 * n * bins)
    return k1, beta, w.in_freq(xi)


def exact(case, seed):
    if case["kind"] == "solve":
        return None  # dozens of adaptive iterations of many signals
    d = _inputs(case, seed)
    n, bins = d["n"], case["bins"]
    a, b, c, a_inv, q = d["tf"]
    bits = case.get("bits", _bits(n, bins))
    w = _Window(bins, case.get("delta", 1e-5))
    k0 = torch.from_numpy(d["k"].astype(np.int64)).cuda()
    off = torch.tensor(_offsets(bins, bits), device="cuda")
    if case["kind"] == "bin":
        return _bins_of(d["x"], n, w, bits, a, b, c, q[0]).cpu().numpy()
    if case["kind"] == "freq":
        u = torch.from_numpy(d["u"]).cuda()
        k1, beta, wf = _setup_modes(w, n, bins, a, b, k0)
        base = wf * torch.from_numpy(d["c"]).cuda() * _unit(q[0] * k1 + c * k0, n)
        u.index_add_(1, beta, base[None] * _unit(off[:, None] * k1[None], n), alpha=-1)
        return u.cpu().numpy()
    scale = 1.0 / (case["trials"] * (1 + 2 * bits))
    if case["kind"] == "est":
        k1, beta, wf = _setup_modes(w, n, bins, a, b, k0)
        acc = 0
        for qt in q:
            u = _bins_of(d["x"], n, w, bits, a, b, c, qt)[:, beta]
            acc = acc + (u * _unit(-(off[:, None] + qt) % n * k1[None], n)).sum(0)
        return (acc * _unit(-c * k0, n) * scale / wf).cpu().numpy()
    if case["kind"] == "adj":
        k1, beta, wf = _setup_modes(w, n, bins, a, b, k0)
        g = torch.from_numpy(d["g"]).cuda() * _unit(c * k0, n) * scale / wf
        dx = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
        for qt in q:
            for o in _offsets(bins, bits):
                row = torch.zeros(bins, dtype=torch.complex128, device="cuda")
                row.index_add_(0, beta, g * _unit((qt + o) % n * k1, n))
                h = torch.fft.ifft(row, norm="forward")
                u = (qt + o + w.t) % n
                v = h[w.t % bins] * w.wt * _unit(w.t, 2 * bins) * _unit(-b * u, n)
                dx.index_add_(0, (a * u + c) % n, torch.view_as_real(v))
        return torch.view_as_complex(dx).cpu().numpy()
    # Iterate: subtract the found modes, vote, estimate, merge
    fk = torch.from_numpy(d["fk"].astype(np.int64)).cuda()
    fc = torch.from_numpy(d["fc"]).cuda()
    k1, beta, wf = _setup_modes(w, n, bins, a, b, fk)
    us = []
    for qt in q:
        u = _bins_of(d["x"], n, w, bits, a, b, c, qt)
        base = wf * fc * _unit(qt * k1 + c * fk, n)
        us.append(u.index_add(1, beta, base[None] * _unit(off[:, None] * k1[None], n),
                              alpha=-1))
    u = torch.stack(us)
    ok = u[:, 0].abs().square().mean(0) >= d["bin_thr"] ** 2
    xs = torch.zeros(bins, dtype=torch.int64, device="cuda")
    for s in range(bits):
        u0, u1, u2 = u[:, 0], u[:, 2 * s + 1], u[:, 2 * s + 2]
        m01 = u0.conj() * u2 + u1.conj() * u0
        m00 = u0.abs().square() + u1.abs().square()
        m11 = u2.abs().square() + u0.abs().square()
        lmax = 0.5 * (m00 + m11) + torch.sqrt((0.5 * (m00 - m11)) ** 2 + m01.abs().square())
        det2 = (u0 * u0 - u1 * u2).abs().square()
        ok &= ~(det2 > 4.0 * d["sv_thr"] ** 2 * lmax).any(0)
        xs = 2 * xs + ((m01.imag > 0).sum(0) > case["trials"] // 2)
    ar = torch.arange(bins, device="cuda")
    k1 = torch.floor(n * (ar.double() + (2 * xs + 1).double() / 2.0 ** (bits + 1)) / bins
                     + 0.5).long()
    wf = w.in_freq((2 * bins * k1 - (2 * ar + 1) * n).double() / (2.0 * n * bins))
    ok &= wf.abs() >= 0.1
    acc = 0
    for t, qt in enumerate(q):
        acc = acc + (u[t] * _unit(-(off[:, None] + qt) % n * k1[None], n)).sum(0)
    new = a_inv * ((k1 - b) % n) % n
    coef = acc * _unit(-c * new, n) * scale / wf
    mm = dict(zip(d["fk"].tolist(), d["fc"].tolist()))
    for kk, cc in zip(new[ok].tolist(), coef[ok].tolist()):
        mm[kk] = mm.get(kk, 0) + cc
    out = np.zeros(d["fk"].size + bins + 16, np.complex128)
    out[:len(mm)] = [mm[v] for v in sorted(mm)]
    return {"k": None, "size": None, "c": out}
