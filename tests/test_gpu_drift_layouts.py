"""Drift layouts that a handle asks for, at the edges of what fits: FP32 strips
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
