"""The strip drift's regular trips have a gather of their own.  One step from the
same grid: its error against FP64, beside that of the windowed drift, which
takes the general gather for every cell.  Both round the footpoints, the
coefficients and the value alike; the two forms' own roundings, emulated in
FP32 on smooth and rough taps, give the same rms error to 1 % wherever
neighbouring taps differ by less than their size."""

import numpy as np
import pytest

from drift_tables import drift_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
@pytest.mark.parametrize("init", ["UDF", "Plummer"])
def test_regular_trips_are_as_exact_as_the_general_gather(init, drift):
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = {"type": init, "Pmin": 0.01, "Pmax": 25.0, "Pres": 256, "Pscale": "logarithmic",
           "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6), "Ures": (256, 16),
           "Uscale": ("linear", "quadratic"), "dt": 0.005}
    s = {k: VlasovSolver21Spline(cfg, precision=p, layout={"drift": d})
         for k, p, d in (("ref", "fp64", "window"), ("general", "fp32", "window"),
                         ("strip", "fp32", drift))}
    assert s["strip"].layout()["drift"] == drift
    r = s["ref"]
    fp = r.footpoints()
    t = drift_tables(fp, np.zeros(r.ncells, bool), r.nr, r.nu, r.nj)
    assert t["regular"].mean() > 0.25
    f0 = s["general"].f  # values that FP32 holds
    err = {}
    for k, h in s.items():
        h.f = f0
        h.step(1)
    ref = r.f
    for k in ("general", "strip"):
        err[k] = np.linalg.norm(s[k].f - ref)
    assert err["strip"] <= 1.02 * err["general"], err
