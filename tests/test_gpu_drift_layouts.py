"""Drift layouts that a handle asks for, at the edges of what fits: FP64 strips
(two blocks of up to 253 v_r vertices per SM, one of up to 573), FP32 strips
(two buffers up to 573 vertices, one up to 1149; the tallest of each read the
moment weights in global memory), windows beyond.  Against the oracle, FP64 to
1e-12 of the largest value, FP32 to the storage modes' bounds (relative L2
2e-6, largest error 1e-5 of the largest value)."""

import numpy as np
import pytest

from oracle.vls_oracle import Oracle

pytestmark = pytest.mark.gpu


def _cfg(nr, nu, **kw):
    cfg = {"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": nr - 1, "Pscale": "logarithmic",
           "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6), "Ures": (nu - 1, 5),
           "Uscale": ("linear", "quadratic"), "dt": 0.05, "kernelBufferSize": 4}
    cfg.update(kw)
    return cfg


def _close(s, o, precision):
    ref = o.f
    d = s.f - ref
    if precision == "fp64":
        assert np.abs(d).max() <= 1e-12 * np.abs(ref).max()
    else:
        assert np.linalg.norm(d) <= 2e-6 * np.linalg.norm(ref)
        assert np.abs(d).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("precision,want,nr,nu,drift", [
    ("fp64", "strip2", 65, 33, "strip2"), ("fp64", "strip1", 65, 33, "strip1"),
    ("fp64", "strip2", 41, 253, "strip2"), ("fp64", "strip2", 41, 254, "window"),
    ("fp64", "strip1", 41, 254, "strip1"), ("fp64", "strip1", 33, 573, "strip1"),
    ("fp64", "strip1", 33, 574, "window"), ("fp64", "strip1", 9, 8, "strip1"),
    ("fp64", "auto", 65, 33, "window"),
    ("fp32", "strip2", 41, 567, "strip2"), ("fp32", "strip2", 65, 568, "strip2"),
    ("fp32", "auto", 41, 573, "strip2"), ("fp32", "auto", 41, 574, "strip1"),
    ("fp32", "strip2", 41, 574, "window"), ("fp32", "auto", 33, 1147, "strip1"),
    ("fp32", "strip1", 65, 1148, "strip1"), ("fp32", "auto", 41, 1149, "strip1"),
    ("fp32", "auto", 41, 1150, "window"), ("fp32", "strip1", 41, 1150, "window"),
])
def test_layout_is_the_one_asked_for(precision, want, nr, nu, drift):
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = _cfg(nr, nu)
    s = VlasovSolver21Spline(cfg, precision=precision, layout={"drift": want})
    assert s.layout()["drift"] == drift
    o = Oracle(cfg)
    for _ in range(2):
        s.step(1)
        o.step(1)
        _close(s, o, precision)
    s.sync()


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
def test_fp64_strip_wait_timeout_reports_and_falls_back(drift):
    """Waits that give up at once: reported, and the cells read C in global
    memory (the copies still land before the block ends)."""
    from vlasolve_b200 import VlasovSolver21Spline, _lib
    cfg = _cfg(65, 33)
    s = VlasovSolver21Spline(cfg, precision="fp64",
                             layout={"drift": drift, "drift_wait_spins": -1})
    o = Oracle(cfg)
    s.step(1)
    o.step(1)
    with pytest.raises(_lib.VlsError) as e:
        s.sync()
    assert e.value.code == _lib.VLS_ECUDA and "drift" in str(e.value)
    _close(s, o, "fp64")


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
def test_fp64_strips_in_batches_are_bit_identical(drift):
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = _cfg(65, 70)
    a = VlasovSolver21Spline(cfg, precision="fp64", layout={"drift": drift})
    b = VlasovSolver21Spline(cfg, precision="fp64",
                             layout={"drift": drift, "slices_per_batch": 2, "streams": 2})
    a.step(4)
    b.step(4)
    np.testing.assert_array_equal(a.f, b.f)


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
@pytest.mark.parametrize("nr,nu", [(65, 33), (130, 97), (34, 112), (720, 47)])
def test_short_fp32_strips_take_the_general_gather(nr, nu, drift):
    """FP32 strips of fewer than 15 trips run in blocks of one strip, whose cells
    take the general gather: the same bits as the windowed drift's."""
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = _cfg(nr, nu, kernelBufferSize=2)
    f = {}
    for k in ("window", drift):
        s = VlasovSolver21Spline(cfg, precision="fp32", layout={"drift": k})
        assert s.layout()["drift"] == k
        s.step(1)
        s.sync()
        f[k] = s.f
    np.testing.assert_array_equal(f[drift], f["window"])


@pytest.mark.parametrize("nr,nu", [(33, 33), (34, 112), (34, 113), (65, 97), (97, 129)])
@pytest.mark.parametrize("drift", ["strip2", "strip1"])
def test_strips_at_the_edge_of_the_block_form_match_oracle(nr, nu, drift):
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = _cfg(nr, nu, kernelBufferSize=8)
    a = VlasovSolver21Spline(cfg, precision="fp32", layout={"drift": drift})
    b = VlasovSolver21Spline(cfg, precision="fp32",
                             layout={"drift": drift, "slices_per_batch": 2, "streams": 2})
    o = Oracle(cfg)
    for _ in range(3):
        for s in (a, b, o):
            s.step(1)
        _close(a, o, "fp32")
    np.testing.assert_array_equal(a.f, b.f)


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
def test_fp32_strip_blocks_wait_timeout_reports_and_falls_back(drift):
    from vlasolve_b200 import VlasovSolver21Spline, _lib
    cfg = _cfg(65, 33)
    s = VlasovSolver21Spline(cfg, precision="fp32",
                             layout={"drift": drift, "drift_wait_spins": -1})
    o = Oracle(cfg)
    s.step(1)
    o.step(1)
    with pytest.raises(_lib.VlsError) as e:
        s.sync()
    assert e.value.code == _lib.VLS_ECUDA and "drift" in str(e.value)
    _close(s, o, "fp32")
