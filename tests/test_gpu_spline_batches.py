"""Point sets and grids large enough for the parallel branches of the spline
level (more than 4096 points; host arrays of 16 MB and more): the same values
as small calls give, bit for bit, and the first bad point named."""

import numpy as np
import pytest

from vlasolve_b200 import _lib
from vlasolve_b200.spline import InterpolSpline, LocalSpline2

pytestmark = pytest.mark.gpu

N, PART = 30011, 997  # points; those of one small call


def _spline(ns=3, precision="fp64"):
    sp = LocalSpline2((0.01, -2.0), (25.0, 2.0), (40, 32), scale=("logarithmic", "linear"),
                      nslices=ns, precision=precision)
    g = np.random.default_rng(3)
    sp.assign(g.normal(size=(ns, 33, 41)))
    sp.build()
    return sp


def _parts(n):
    return [slice(k, min(k + PART, n)) for k in range(0, n, PART)]


@pytest.fixture(scope="module")
def points():
    g = np.random.default_rng(4)
    return dict(xx=np.exp(g.uniform(np.log(0.0101), np.log(24.9), N)), yy=g.uniform(-1.99, 1.99, N),
                sl=g.integers(0, 3, N), Nx=g.integers(0, 40, N).astype(np.int32),
                Ny=g.integers(0, 32, N).astype(np.int32), x=g.random(N), y=g.random(N))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_large_point_sets_match_small_ones(points, precision):
    sp, p = _spline(precision=precision), points
    for d, q in ((0, p["xx"]), (1, p["yy"])):
        I, F = sp.pos2Coord(q, d)
        for s in _parts(N):
            i, f = sp.pos2Coord(q[s], d)
            np.testing.assert_array_equal(I[s], i)
            np.testing.assert_array_equal(F[s], f)
    v = sp.evaluate(p["xx"], p["yy"], p["sl"])
    c = sp.evaluateC(p["Nx"], p["x"], p["Ny"], p["y"], p["sl"])
    w = sp.evaluateNxPy(p["Nx"], p["yy"], p["sl"])
    for s in _parts(N):
        np.testing.assert_array_equal(v[s], sp.evaluate(p["xx"][s], p["yy"][s], p["sl"][s]))
        np.testing.assert_array_equal(
            c[s], sp.evaluateC(p["Nx"][s], p["x"][s], p["Ny"][s], p["y"][s], p["sl"][s]))
        np.testing.assert_array_equal(w[s], sp.evaluateNxPy(p["Nx"][s], p["yy"][s], p["sl"][s]))


@pytest.mark.parametrize("n", [1000, N])
def test_first_bad_point_is_named(points, n):
    """Of bad points in any order, the first; at the same point the node comes
    before the slice.  Small and parallel calls alike."""
    sp = _spline()
    p = {k: v[:n].copy() for k, v in points.items()}
    k = n // 2

    def error():
        with pytest.raises(_lib.VlsError) as e:
            sp.evaluateC(p["Nx"], p["x"], p["Ny"], p["y"], p["sl"])
        assert e.value.code == _lib.VLS_EINVAL
        return str(e.value)

    p["sl"][n - 1] = 3
    assert "point %d: slice out of range" % (n - 1) in error()
    p["Ny"][k + 7] = 33
    assert "point %d lies outside the spline's nodes" % (k + 7) in error()
    p["sl"][k] = -1
    assert "point %d: slice out of range" % k in error()
    p["Nx"][k] = -1
    assert "point %d lies outside the spline's nodes" % k in error()
    ok = sp.evaluateC(points["Nx"][:n], points["x"][:n], points["Ny"][:n], points["y"][:n])
    assert np.isfinite(ok).all()


@pytest.mark.parametrize("use_log", [False, True])
def test_large_interpolations_match_small_ones(points, use_log):
    ini = InterpolSpline.createInit(0.01, 25.0, 40, -2.0, 2.0, 32, xscaleType="logarithmic",
                                    useLog=use_log)
    g = np.random.default_rng(9)
    sp = InterpolSpline(ini, g.uniform(0.5, 1.5, (ini.ny, ini.nx)))
    x, y = points["xx"], points["yy"]
    kw = {"grad": True} if use_log else {"hess": True}  # no Hessians of log values
    all_ = sp.evaluate(x, y, **kw)
    for s in _parts(N):
        for a, b in zip(all_, sp.evaluate(x[s], y[s], **kw)):
            np.testing.assert_array_equal(a[s], b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_large_grids_through_the_host_copies(precision):
    """2.2 M cells set and read through pageable arrays of 17.7 MB: every element
    comes back, rounded by FP32 storage."""
    from vlasolve_b200 import VlasovSolver21Spline
    g = np.random.default_rng(12)
    s = VlasovSolver21Spline({"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": 132,
                              "Pscale": "logarithmic", "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6),
                              "Ures": (160, 103), "Uscale": ("linear", "quadratic"), "dt": 0.01},
                             precision=precision)
    f = g.normal(size=s.shape)
    assert f.nbytes > 16 << 20 and f.nbytes % (4 << 20)
    want = f if precision == "fp64" else f.astype(np.float32).astype(np.float64)
    s.f = f
    np.testing.assert_array_equal(s.f, want)
    odd = np.empty(f.size + 3)[3:].reshape(f.shape)  # not on a page's start
    s.get_f_into(odd)
    np.testing.assert_array_equal(odd, want)
