"""The statistics' blocks take 16, 8, 4 or 2 rows of cells, as the grid needs to
fill the GPU: against the oracle's sums.  Both add up to 1e6 terms of one sign
per quantity, the oracle in plain FP64: 1e-11 of the quantity (of |Ek| + |Ep|
for the energy)."""

import numpy as np
import pytest

from oracle.vls_oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,rows", [((33, 8), 2), ((18, 3), 2), ((4, 1), 2), ((66, 20), 4),
                                        ((40, 33), 4), ((34, 75), 8), ((65, 60), 8),
                                        ((64, 80), 16), ((65, 75), 16)],
                         ids=lambda v: "%dx%d" % v if isinstance(v, tuple) else "%d" % v)
def test_statistics_match_oracle(shape, rows):
    from vlasolve_b200 import VlasovSolver21Spline
    nu, nj = shape
    want = 16
    while want > 2 and -(-(nu - 1) // want) * nj < 2 * 148:
        want //= 2
    assert want == rows
    cfg = {"type": "UDF", "Pmin": 0.01, "Pmax": 25.0, "Pres": 300, "Pscale": "logarithmic",
           "Umin": (-2.0, 0.0), "Umax": (2.0, 1.6), "Ures": (nu - 1, nj),
           "Uscale": ("linear", "quadratic"), "dt": 0.02}
    s, o = VlasovSolver21Spline(cfg), Oracle(cfg)
    f = o.f * (1.0 + 0.2 * np.random.default_rng(nu).random(o.f.shape))
    s.f = f
    o.f = f
    a, b = s.stats(), o.stats()
    for k in ("Mass", "Ek", "Ep", "S", "L1", "L2"):
        assert abs(a[k] - b[k]) <= 1e-11 * abs(b[k]), (k, a[k], b[k])
    assert abs(a["E"] - b["E"]) <= 1e-11 * (abs(b["Ek"]) + abs(b["Ep"]))
