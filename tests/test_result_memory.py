"""Memory of a download's per-PS vectors (host only: the library call is a stand-in
that fills what it is given): reused by the ordinary loop, never while a caller
still refers to it, and kept alive vector by vector."""
import ctypes
import gc
from types import SimpleNamespace

import numpy as np
import pytest

from pystamps_b200 import stage2 as S

KEYS = ("K_ps", "C_ps", "coh_ps", "N_opt", "coh_ps_save")


class Library:
    """ps2_download: every requested vector filled with the number of the call."""

    def __init__(self):
        self.calls = 0

    def ps2_download(self, _, ref):
        self.calls += 1
        o = ref._obj
        for k in KEYS:
            if getattr(o, k):
                ctypes.memset(getattr(o, k), 0, 8 * self.n)
                np.frombuffer((ctypes.c_double * self.n).from_address(getattr(o, k)))[:] = self.calls
        return 0

    def ps2_destroy(self, _):
        pass


@pytest.fixture
def ctx():
    c = S.Stage2Context.__new__(S.Stage2Context)
    lib = Library()
    fresh = S.Stage2Context.__init__
    real = S.lib
    S.lib = lambda: SimpleNamespace(ps2_create=lambda *a: 0, ps2_download=lib.ps2_download, ps2_destroy=lib.ps2_destroy)
    try:
        fresh(c)
    finally:
        S.lib = real

    def load(n):
        lib.n = n
        c.prepared = SimpleNamespace(n_ps=n, n_ifg=3, n_i=2, n_j=2, n_trial_wraps=1.0, grid_ij=None, grid_size=50.0,
                                     low_pass=None, nr_max_nz_ix=1.0)
    c.set = load
    load(1000)
    return c


@pytest.fixture
def allocated(monkeypatch):
    """Elements of the float64 vectors allocated so far."""
    empty, total = np.empty, []

    def counting(shape, dtype=float, **kw):
        if np.dtype(dtype) == np.float64 and np.size(shape) == 1:
            total.append(int(np.ravel(shape)[0]))
        return empty(shape, dtype=dtype, **kw)

    monkeypatch.setattr(np, "empty", counting)
    return lambda: sum(total)


def _address(v):
    return v.__array_interface__["data"][0]


def test_the_ordinary_loop_takes_two_blocks_in_turn(ctx, allocated):
    r = None
    for call in range(1, 11):
        r = ctx.download(KEYS)  # the previous result is dropped once this one is there
        assert all((r[k] == call).all() for k in KEYS)
    assert allocated() == 2 * 1000 * len(KEYS)


def test_what_a_caller_holds_is_not_handed_out_again(ctx):
    held = [ctx.download(KEYS) for _ in range(4)]
    tail = ctx.download(("K_ps",))["K_ps"][7:]
    tensor_like = memoryview(ctx.download(("K_ps",))["K_ps"])
    for _ in range(5):
        ctx.download(KEYS)
    gc.collect()
    for call, r in enumerate(held, 1):
        assert all((r[k] == call).all() and r[k].flags.writeable and r[k].flags.c_contiguous for k in KEYS)
    assert (tail == 5).all() and (np.asarray(tensor_like) == 6).all()


def test_a_kept_vector_keeps_itself_only(ctx):
    r = ctx.download(KEYS)
    coh = r["coh_ps"]
    spans = sorted((_address(r[k]), _address(r[k]) + r[k].nbytes) for k in KEYS)
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    del r
    again = ctx.download(KEYS)
    assert _address(again["coh_ps"]) != _address(coh)
    owner = coh
    while isinstance(owner, np.ndarray) and owner.base is not None:
        owner = owner.base
    assert memoryview(owner).nbytes == coh.nbytes


def test_calls_without_vectors_and_other_sizes(ctx, allocated):
    held = ctx.download(KEYS)
    assert "K_ps" not in ctx.download(("ph_grid",))
    given = np.zeros(1000)
    assert ctx.download(("K_ps",), out={"K_ps": given})["K_ps"] is given
    del held
    ctx.download(KEYS)
    assert allocated() == 1000 * len(KEYS)  # kept through both
    ctx.set(400)
    assert all(ctx.download(KEYS)[k].shape == (400,) for k in KEYS)
    ctx.set(1000)
    assert all(ctx.download(KEYS)[k].shape == (1000,) for k in KEYS)
