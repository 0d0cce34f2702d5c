"""Contexts on several threads at once: calls whose kernels want different
amounts of shared memory (the limit is one per kernel for the whole process),
each with the results of a lone context."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import mpsft_gb300 as m

pytestmark = pytest.mark.gpu


def test_threads_with_different_sizes():
    n, bits = 1 << 20, 3
    rng = np.random.default_rng(3)
    calls = []
    for bins, modes in [(65, 10), (4001, 8000), (129, 300), (2001, 4000), (65, 9000)]:
        k = np.sort(rng.choice(n, modes, replace=False)).astype(np.int32)
        c = rng.standard_normal(modes) + 1j * rng.standard_normal(modes)
        u = rng.standard_normal((1 + 2 * bits, bins)) + 0j
        calls.append((u, n, bins, bits, 1e-5, 4097, 77, 5, 4099, k, c))
    ctx = m.Context(0)
    want = [ctx.bin_in_freq(*call) for call in calls]
    ctx.close()
    failures = []

    def work(first):
        try:
            c = m.Context(0)
            for i in range(250):
                j = (first + i) % len(calls)
                if not np.array_equal(c.bin_in_freq(*calls[j]), want[j]):
                    failures.append((first, i, "values"))
            c.close()
        except Exception as e:  # (reported by the test's own thread)
            failures.append((first, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:4]


def test_bucket_takes_bins_beyond_every_transform(ctx):
    """BinInFreq with the caller's responses has no transform: 24401 bins and 100
    modes, whose bucketing takes more shared memory than any bins with one."""
    n, bins, bits = 1 << 20, 24401, 1
    rng = np.random.default_rng(4)
    k = np.sort(rng.choice(n, 100, replace=False)).astype(np.int32)
    c = rng.standard_normal(100) + 1j * rng.standard_normal(100)
    a, b, cc, q = 4097, 77, 5, 4099
    got = ctx.bin_in_freq_wf(np.zeros((1 + 2 * bits, bins), np.complex128), n, bins, bits,
                             a, b, cc, q, k, c, np.ones(100))
    want = np.zeros_like(got)
    for kk, v in zip(k.astype(object), c):
        k1 = (a * kk + b) % n
        for r, off in enumerate((0, bins, -bins)):
            ph = ((q + off) * k1 + cc * kk) % n
            want[r, k1 * bins // n] -= v * np.exp(2j * np.pi * ph / n)
    assert np.abs(got - want).max() <= 1e-13


def test_tables_of_many_sizes_in_turn():
    """More bytes of tables than a context keeps (their memory is reused in turns,
    some calls' in two parts around its end): every call gives the bits that it
    gave first, in another order and between other sizes, and a new context's."""
    n = 1 << 16
    rng = np.random.default_rng(6)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    args = (1e-6, 4097, 77, 5, 4099)
    calls = [(3001 + 8 * i, m.FP64 if i % 3 else m.FP32) for i in range(120)]
    kept = m.Context(0)
    sig = kept.upload(x)
    want = [kept.bin_in_time(sig, b, 2, *args, precision=p) for b, p in calls]
    for i in [119, 0, 60, 119, 3, 3] + list(range(118, -1, -3)) + [0, 119]:
        got = kept.bin_in_time(sig, calls[i][0], 2, *args, precision=calls[i][1])
        assert np.array_equal(got, want[i]), i
    for i in (0, 1, 59, 119):
        c = m.Context(0)
        s = c.upload(x)
        got = c.bin_in_time(s, calls[i][0], 2, *args, precision=calls[i][1])
        assert np.array_equal(got, want[i]), i
        c.close()
    kept.close()
