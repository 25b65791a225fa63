"""The stencils' straight-through arithmetic (hf_fast.cuh, compiled for the host) against the general
functions it stands in for: bit for bit wherever it says the item stayed in its window, and staying in it
wherever the values are ordinary.  The general functions are checked against the reference's fixtures
and the oracle elsewhere."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT

LIB = os.path.join(ROOT, "hyperflow_gb300", "libhf_hostmath.so")
P, D, I, N = C.c_void_p, C.c_double, C.c_int, C.c_int64


@pytest.fixture(scope="module")
def hm():
    if not os.path.exists(LIB):
        from hyperflow_gb300 import _build
        _build.build()
    L = C.CDLL(LIB)
    L.hm_predict.argtypes = [I, I, P, D, D, N, P, P, P]
    L.hm_face.argtypes = [I, P, D, D, N, P, P, P, P]
    L.hm_update.argtypes = [P, D, D, D, N, P, P, P]
    L.hm_uns.argtypes = [P, P, D, D, D, D, N, P, P, P, P, P, P]
    L.hm_godunov.argtypes = [I, P, D, D, N, P, P, P, P, P, P, P, P]
    return L


def states(kind, n=60_000):
    """[n][3][4] conservative states: a base state and its two neighbours at a distance between 0 (uniform
    flow) and order one, velocities of exactly zero among them."""
    rng = np.random.default_rng(11)
    base = np.stack([rng.uniform(0.1, 2, n), rng.uniform(-2, 2, n), rng.uniform(-2, 2, n), rng.uniform(0.1, 10, n)], 1)
    w = np.repeat(base[:, None], 3, 1)
    amp = rng.choice([0.0, 1e-15, 1e-8, 1e-5, 1e-3, 0.5], n)[:, None]
    w[:, :, 0] *= 1 + amp * rng.uniform(-1, 1, (n, 3))
    w[:, :, 1] += amp * rng.uniform(-1, 1, (n, 3))
    w[:, :, 2] += amp * rng.uniform(-1, 1, (n, 3))
    w[:, :, 3] *= 1 + amp * rng.uniform(-1, 1, (n, 3))
    w[rng.random(n) < 0.25, :, 1] = 0.0
    w[rng.random(n) < 0.25, :, 2] = 0.0
    if kind == "faint":        # velocities down to the subnormals: some at rest for all that matters
        w[:, :, 1] *= 2.0 ** -rng.integers(0, 1100, (n, 1)).astype(float)
    if kind == "unphysical":   # pressures below zero in some
        w[:, :, 3] -= rng.uniform(0, 2, (n, 3))
    if kind == "scaled":       # densities and pressures towards both ends of the range
        s = 2.0 ** rng.integers(-600, 600, (n, 1)).astype(float)
        w[:, :, 0] *= s
        w[:, :, 3] *= s
    with np.errstate(all="ignore"):
        c = np.stack([w[..., 0], w[..., 0] * w[..., 1], w[..., 0] * w[..., 2],
                      w[..., 3] / 0.4 + 0.5 * w[..., 0] * (w[..., 1] ** 2 + w[..., 2] ** 2)], -1)
    if kind == "special":      # one value of a state replaced
        odd = np.array([0.0, -0.0, 5e-324, -1e-310, 2.2e-308, 1e-300, 1e300, np.inf, -np.inf, np.nan, 2.0 ** 257,
                        2.0 ** -255, np.nextafter(2.0 ** -255, 0)])
        c[np.arange(n), rng.integers(0, 3, n), rng.integers(0, 4, n)] = rng.choice(odd, n)
    return np.ascontiguousarray(c)


def same(a, b):
    return (a.view(np.uint64) == b.view(np.uint64)) | (np.isnan(a) & np.isnan(b))


@pytest.mark.parametrize("kind", ["ordinary", "faint", "unphysical", "scaled", "special"])
@pytest.mark.parametrize("y", [0, 1])
def test_fast_functions_equal_the_general_ones(hm, kind, y):
    c = states(kind)
    n = len(c)
    g, g1 = 1.4, 1.4 - 1.0
    for lim, h in ((0, 0.173), (1, 0.05)):
        ok, fast, gen = np.empty(n, np.int32), np.zeros((n, 8)), np.empty((n, 8))
        hm.hm_predict(lim, y, c.ctypes.data, g1, h, n, ok.ctypes.data, fast.ctypes.data, gen.ctypes.data)
        assert same(fast, gen)[ok == 1].all()
        if kind == "ordinary":
            assert ok.mean() > 0.99
    ok, bad, fast, gen = np.empty(n, np.int32), np.empty(n, np.int32), np.zeros((n, 4)), np.empty((n, 4))
    hm.hm_face(y, c.ctypes.data, g, g1, n, ok.ctypes.data, bad.ctypes.data, fast.ctypes.data, gen.ctypes.data)
    assert same(fast, gen)[ok == 1].all() and not bad[ok == 1].any()
    if kind == "ordinary":
        assert ok.mean() > 0.99
    hm.hm_update(c.ctypes.data, 1.7e-4, 1365.0, 1000.3, n, ok.ctypes.data, fast.ctypes.data, gen.ctypes.data)
    assert same(fast, gen)[ok == 1].all()


@pytest.mark.parametrize("kind", ["ordinary", "faint", "unphysical", "scaled", "special"])
@pytest.mark.parametrize("y", [0, 1])
def test_godunov_functions_equal_the_general_ones(hm, kind, y):
    """cells, faces and TimeStep terms; and the faces against hllc on the conservative states"""
    c = states(kind)
    n = len(c)
    g, g1 = 1.4, 1.4 - 1.0
    ok, bad = np.empty(n, np.int32), np.empty(n, np.int32)
    out = [np.zeros((n, k)) for k in (10, 10, 4, 4, 2, 2)]
    hm.hm_godunov(y, c.ctypes.data, g, g1, n, ok.ctypes.data, bad.ctypes.data, *[o.ctypes.data for o in out])
    for bit, fast, gen in ((1, out[0], out[1]), (2, out[2], out[3]), (4, out[4], out[5])):
        assert same(fast, gen)[(ok & bit) != 0].all()
        if kind == "ordinary":
            assert ((ok & bit) != 0).mean() > 0.99
    assert not bad[(ok & 2) != 0].any()
    ok2, bad2, fast, gen = np.empty(n, np.int32), np.empty(n, np.int32), np.zeros((n, 4)), np.empty((n, 4))
    hm.hm_face(y, c.ctypes.data, g, g1, n, ok2.ctypes.data, bad2.ctypes.data, fast.ctypes.data, gen.ctypes.data)
    assert same(out[3], gen).all() and (bad == bad2).all()


@pytest.mark.parametrize("kind", ["ordinary", "faint", "unphysical", "scaled", "special"])
def test_unstructured_functions_equal_the_general_ones(hm, kind):
    """edges at any angle (along the axes among them, where a sine or cosine is zero) and cell updates"""
    c = states(kind)
    n = len(c)
    rng = np.random.default_rng(5)
    a = rng.uniform(-np.pi, np.pi, n)
    a[::5] = rng.integers(-2, 3, len(a[::5])) * (np.pi / 2)
    geo = np.stack([np.cos(a), np.sin(a), np.cos(-a), np.sin(-a), 10.0 ** rng.uniform(-4, 0, n)], 1)
    geo[::10, :4] = np.round(geo[::10, :4])
    ok, bad = np.empty(n, np.int32), np.empty(n, np.int32)
    out = [np.zeros((n, k)) for k in (4, 4, 5, 5)]
    hm.hm_uns(c.ctypes.data, geo.ctypes.data, 1.4, 1.4 - 1.0, 1e-3, 0.01, n, ok.ctypes.data, bad.ctypes.data,
              *[o.ctypes.data for o in out])
    assert same(out[0], out[1])[(ok & 1) != 0].all() and not bad[(ok & 1) != 0].any()
    assert same(out[2], out[3])[(ok & 2) != 0].all()
    if kind == "ordinary":
        assert ((ok & 1) != 0).mean() > 0.98 and ((ok & 2) != 0).mean() > 0.95


def test_fast_functions_leave_the_window_for_odd_constants(hm):
    """a zero step, a gamma of one and infinite spacings go to the general functions, or equal them"""
    c = states("ordinary", 4000)
    n = len(c)
    ok, fast, gen = np.empty(n, np.int32), np.zeros((n, 8)), np.empty((n, 8))
    for g1, h in ((0.4, 0.0), (0.0, 0.1), (1e-90, 0.1), (0.4, np.inf), (0.4, np.nan)):
        hm.hm_predict(0, 0, c.ctypes.data, g1, h, n, ok.ctypes.data, fast.ctypes.data, gen.ctypes.data)
        assert not ok.any()
    for dt, one in ((0.0, 10.0), (1e-3, np.inf), (np.nan, 1.0)):
        hm.hm_update(c.ctypes.data, dt, one, 1.0, n, ok.ctypes.data, fast.ctypes.data, gen.ctypes.data)
        assert not ok.any()
