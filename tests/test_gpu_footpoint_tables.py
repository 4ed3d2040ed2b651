"""The drift kernels' tables follow the footpoints: a handle whose footpoints are
replaced steps like one that was made with them, and each kind of trip, cell
and chunk is compared with the oracle in a case that is known to hold it."""

import ctypes

import numpy as np
import pytest

from oracle.vls_oracle import Oracle

from drift_tables import drift_tables

pytestmark = pytest.mark.gpu

LAYOUTS = [("fp64", "window"), ("fp32", "window"), ("fp32", "strip2"), ("fp32", "strip1")]


def _cfg(pres, ures, dt, **kw):
    cfg = {"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": pres, "Pscale": "logarithmic",
           "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6), "Ures": ures,
           "Uscale": ("linear", "quadratic"), "dt": dt}
    cfg.update(kw)
    return cfg


def _solver(cfg, precision, drift):
    from vlasolve_b200 import VlasovSolver21Spline
    s = VlasovSolver21Spline(cfg, precision=precision, layout={"drift": drift})
    assert s.layout()["drift"] == drift
    return s


def _set_footpoints(s, fp):
    i32, u8 = ctypes.POINTER(ctypes.c_int32), ctypes.POINTER(ctypes.c_uint8)
    d = ctypes.POINTER(ctypes.c_double)
    assert s._L.vls_set_footpoints(
        s._h, fp["rI"].ctypes.data_as(i32), fp["rF"].ctypes.data_as(d),
        fp["uI"].ctypes.data_as(i32), fp["uF"].ctypes.data_as(d),
        fp["out"].ctypes.data_as(u8), fp["driftR"].ctypes.data_as(d)) == 0


@pytest.mark.parametrize("precision,drift", LAYOUTS)
def test_tables_follow_new_footpoints(precision, drift):
    """Without gravity the kick's shift is zero whatever dt is, so a handle of
    time step a that is given the footpoints of time step b steps exactly as a
    handle of time step b.  From a to b regular trips become irregular, trips
    and chunks become empty, and the list of far cells grows from nothing; from
    b to a they turn back; c lies between."""
    shape = (96, (256, 5))
    dts = {"a": 0.005, "b": 0.3, "c": 0.1}
    handles = {k: _solver(_cfg(*shape, dt, kernelBufferSize=0, G=0.0), precision, drift)
               for k, dt in dts.items()}
    a = handles["a"]
    fps = {k: h.footpoints() for k, h in handles.items()}
    nr, nu, nj = a.nr, a.nu, a.nj
    tab = {k: drift_tables(fp, np.zeros(a.ncells, bool), nr, nu, nj) for k, fp in fps.items()}
    ta, tb, tc = tab["a"], tab["b"], tab["c"]
    assert not ta["far"].any() and tb["far"].sum() > tc["far"].sum() > 0
    assert (ta["regular"] & tb["others"]).any() and (ta["others"] & tb["empty"]).any()
    assert (tb["empty"] & tc["others"]).any() and (tb["empty_chunks"] & ~ta["empty_chunks"]).any()
    rng = np.random.default_rng(5)
    f0 = a.f * (1.0 + 0.1 * rng.random(a.f.shape))
    want = {}
    for k, h in handles.items():
        h.f = f0
        h.step(1)
        want[k] = h.f.copy(), h.last_mass()
    assert np.abs(want["a"][0] - want["b"][0]).max() > 1e-3 * np.abs(f0).max()
    for k in "bacab":
        _set_footpoints(a, fps[k])
        a.f = f0
        a.step(1)
        np.testing.assert_array_equal(a.f, want[k][0])
        assert a.last_mass() == want[k][1]
    a.sync()


def _compare(cfg, precision, drift, steps=3):
    s, o = _solver(cfg, precision, drift), Oracle(cfg)
    for _ in range(steps):
        s.step(1)
        o.step(1)
        ref = o.f
        d = s.f - ref
        if precision == "fp64":
            assert np.abs(d).max() <= 1e-12 * np.abs(ref).max()
        else:
            assert np.linalg.norm(d) <= 2e-6 * np.linalg.norm(ref)
            assert np.abs(d).max() <= 1e-5 * np.abs(ref).max()
    s.sync()


def _tables_of(cfg):
    o = Oracle(cfg)
    fp = o.footpoints()
    nr, nu = cfg["Pres"] + 1, cfg["Ures"][0] + 1
    chain = fp["driftR"] < o.kernel_radius()
    return drift_tables(fp, chain, nr, nu, chain.size // (nr * nu)), o.chains(), chain


@pytest.mark.parametrize("precision,drift", LAYOUTS)
@pytest.mark.parametrize("shape", [(96, (256, 5)), (70, (100, 5)), (33, (31, 7))],
                         ids=lambda s: "%dx%d" % (s[0] + 1, s[1][0] + 1))
def test_chains_and_far_cells_match_oracle(shape, precision, drift):
    """Delayed-kernel chains and cells whose taps leave their strip: FP64 to
    1e-12 of the largest value, FP32 to the storage modes' bounds (relative L2
    2e-6, largest error 1e-5 of the largest value)."""
    cfg = _cfg(*shape, 0.05, kernelBufferSize=8)
    t, ch, chain = _tables_of(cfg)
    assert len(ch["len"]) == chain.sum() > 20
    if shape[0] == 96:
        assert t["far"].any() and t["regular"].any() and t["empty_chunks"].any()
    _compare(cfg, precision, drift)


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
@pytest.mark.parametrize("nu", [33, 131])
def test_refilled_strip_buffers_match_oracle(nu, drift):
    """More strips than twice the buffers of 148 SMs, so that every block
    refills its buffers (131 v_r vertices; shorter strips have a block each),
    with all three kinds of trips."""
    cfg = _cfg(96, (nu - 1, 200), 0.05, kernelBufferSize=4)
    t, _, _ = _tables_of(cfg)
    assert t["regular"].shape[0] * t["regular"].shape[1] > 2 * 2 * 148
    assert t["regular"].any() and t["empty"].any() and t["others"].any()
    _compare(cfg, "fp32", drift)


@pytest.mark.parametrize("nr", [33, 65, 160, 192, 257])
def test_long_runs_of_strips_are_those_of_short_ones(nr):
    """More than 12 strips for each of 148 blocks are taken in another order than
    fewer; values and moments are those of batches of few slices, bit for bit."""
    from vlasolve_b200 import VlasovSolver21Spline
    ns = nr // 32 if nr % 32 == 1 else -(-nr // 32)
    nj = -(-12 * 148 // ns) + 7
    cfg = _cfg(nr - 1, (112, nj), 0.02, kernelBufferSize=3)
    a = VlasovSolver21Spline(cfg, precision="fp32", layout={"drift": "strip2"})
    b = VlasovSolver21Spline(cfg, precision="fp32",
                             layout={"drift": "strip2", "slices_per_batch": 61})
    for _ in range(2):
        a.step(1)
        b.step(1)
        assert a.last_mass() == b.last_mass()
        np.testing.assert_array_equal(a.f, b.f)
    a.sync()
    b.sync()
