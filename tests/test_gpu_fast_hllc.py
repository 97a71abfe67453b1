"""The fast mode's HLLC (one formula for every wave case) against the exact
mode's branches: one step without MOOD of a rough periodic state whose mean
flow puts every face in one of HLLC's cases -- supersonic to either side,
subsonic, near sonic, at rest -- in x and in y.  A step sums ~30 rounded terms
of the state's size per stage, so 1e-13 of the largest entry is ~450 ulp."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mord,ngp", [(5, 3), (3, 2)])
@pytest.mark.parametrize("mean", [(0, 0), (4, 0), (-4, 0), (0, 4), (0, -4), (4, -4), (1.18, 0), (0, -1.18), (0.3, 0.2)])
def test_fast_hllc_cases_equal_exact(pkg, mean, mord, ngp):
    lf, nf = 37, 29
    rng = np.random.default_rng(3)
    shape = (nf + 8, lf + 8)
    r, p = 1 + 0.2 * rng.uniform(-1, 1, shape), 1 + 0.2 * rng.uniform(-1, 1, shape)
    u, v = (m + 0.1 * rng.uniform(-1, 1, shape) for m in mean)
    U = np.ascontiguousarray(np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], axis=-1))
    out = {}
    for fp in (pkg.FP_EXACT, pkg.FP_FAST):
        with pkg.Solver(lf=lf, nf=nf, bc_type=18, mord=mord, ngp=ngp, method=pkg.GP_SE, fp_mode=fp) as s:
            V = U.copy()
            s.Boundary_C(V)
            out[fp] = np.empty_like(V)
            s.time_stepping(V, out[fp], 0.0, 1e-3)
    a, b = out[pkg.FP_EXACT], out[pkg.FP_FAST]
    assert np.isfinite(a).all()
    assert np.abs(a - b).max() <= 1e-13 * np.abs(a).max()
