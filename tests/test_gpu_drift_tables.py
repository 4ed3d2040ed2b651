"""The drift kernels' tables.  The FP32 strip drift's trips (8 rows of a 32-column strip): grids whose
last trip or last strip is partial, exactly full, or one row or column more,
both buffer layouts, with delayed-kernel chains and with footpoints that leave
their strip, against the oracle.  Tolerances are those of the FP32 storage
modes everywhere (relative L2 2e-6, largest error 1e-5 of the largest value
per saved step)."""

import numpy as np
import pytest

from oracle.vls_oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drift", ["strip2", "strip1"])
@pytest.mark.parametrize("shape", [(32, 7), (64, 8), (33, 15), (96, 256), (63, 272), (39, 1024)],
                         ids=lambda s: "%dx%d" % (s[0] + 1, s[1] + 1))
def test_strip_trips_match_oracle(shape, drift):
    from vlasolve_b200 import VlasovSolver21Spline
    if drift == "strip2" and shape[1] > 500:
        pytest.skip("two buffers of that height do not fit")
    cfg = {"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": shape[0],
           "Pscale": "logarithmic", "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6),
           "Ures": (shape[1], 5), "Uscale": ("linear", "quadratic"), "dt": 0.05,
           "kernelBufferSize": 2}
    s = VlasovSolver21Spline(cfg, precision="fp32", layout={"drift": drift})
    assert s.layout()["drift"] == drift
    o = Oracle(cfg)
    for _ in range(3):
        s.step(1)
        o.step(1)
        ref = o.f
        d = s.f - ref
        assert np.linalg.norm(d) <= 2e-6 * np.linalg.norm(ref)
        assert np.abs(d).max() <= 1e-5 * np.abs(ref).max()
    s.sync()
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(40, 15), (33, 16), (64, 47), (20, 700)],
                         ids=lambda s: "%dx%d" % (s[0] + 1, s[1] + 1))
def test_window_rows_match_oracle(shape, precision):
    """The windowed drift's chunks of 16 rows: full, one row more, empty ones
    (large steps leave the inner columns outside the box away from v_r = 0),
    and tap blocks hundreds of rows from their own chunk.  FP64 to 1e-12 of
    the largest value, FP32 as above."""
    from vlasolve_b200 import VlasovSolver21Spline
    cfg = {"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": shape[0],
           "Pscale": "logarithmic", "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6),
           "Ures": (shape[1], 5), "Uscale": ("linear", "quadratic"), "dt": 0.05,
           "kernelBufferSize": 1}
    s = VlasovSolver21Spline(cfg, precision=precision, layout={"drift": "window"})
    o = Oracle(cfg)
    for _ in range(3):
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
    s.close()
