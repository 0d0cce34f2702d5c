"""Who frees a signal's handle when a context and its signals are dropped in
any order, on a stand-in library that records the calls (no GPU)."""
from __future__ import annotations

import ctypes
import gc

import pytest

import mpsft_gb300 as m


class _Recorder:
    """The library's frees, in order."""

    def __init__(self):
        self.calls = []

    def mpsft_signal_free(self, h):
        self.calls.append(("signal", h.value))
        return m.OK

    def mpsft_ctx_destroy(self, h):
        self.calls.append(("ctx", h.value))
        return m.OK


def _context(lib):
    ctx = m.Context.__new__(m.Context)
    ctx._h, ctx._lib, ctx._signals = ctypes.c_void_p(1), lib, set()
    return ctx


EVERY_ONCE = [("signal", 10), ("signal", 11), ("signal", 12)]


def test_collected_cycle_frees_signals_before_their_context():
    """The module of a script holds both in one cycle (its functions' globals):
    they are finalized in any order, weak references cleared first."""
    lib = _Recorder()
    ctx = _context(lib)
    cycle = {"ctx": ctx, "sigs": [m.Signal(ctx, ctypes.c_void_p(10 + i), 1 << 12, m.C64)
                                  for i in range(3)]}
    cycle["self"] = cycle
    del ctx, cycle
    gc.collect()
    assert sorted(lib.calls[:3]) == EVERY_ONCE
    assert lib.calls[3:] == [("ctx", 1)]


@pytest.mark.parametrize("explicit", [False, True])
def test_signals_outlive_a_closed_context(explicit):
    lib = _Recorder()
    ctx = _context(lib)
    sigs = [m.Signal(ctx, ctypes.c_void_p(10 + i), 1 << 12, m.C64) for i in range(3)]
    if explicit:
        sigs[1].free()
    ctx.close()
    assert all(s._freed for s in sigs)
    sigs[0].free()
    del sigs
    gc.collect()
    assert sorted(lib.calls[:3]) == EVERY_ONCE and lib.calls[3:] == [("ctx", 1)]


def test_a_dropped_signal_is_freed_at_once():
    lib = _Recorder()
    ctx = _context(lib)
    s = m.Signal(ctx, ctypes.c_void_p(10), 1 << 12, m.C64)
    del s
    gc.collect()
    assert lib.calls == [("signal", 10)] and not ctx._signals
    ctx.close()
    assert lib.calls == [("signal", 10), ("ctx", 1)]
