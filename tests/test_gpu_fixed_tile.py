"""The fast first pass at the edges of its 32 x 4 tiles and of its number
range, against the exact mode: one step without MOOD."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(lf, nf, decades):
    """Rough flow whose density and energy grow by 10^decades per cell along x; momenta with exact zeros."""
    rng = np.random.default_rng(lf * 100 + nf)
    shape = (nf + 8, lf + 8)
    s = 10.0 ** (decades * np.arange(lf + 8.0))[None, :]
    r, p = s * (1 + 0.2 * rng.uniform(-1, 1, shape)), s * (1 + 0.2 * rng.uniform(-1, 1, shape))
    u = 0.3 * rng.uniform(-1, 1, shape) * (rng.uniform(size=shape) > 0.3)
    v = np.zeros(shape)
    v[:, ::3] = 0.1
    return np.ascontiguousarray(np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], axis=-1))


def _step(pkg, U, fp, mord=5, ngp=3):
    with pkg.Solver(lf=U.shape[1] - 8, nf=U.shape[0] - 8, bc_type=17, method=pkg.GP_SE, fp_mode=fp, mord=mord,
                    ngp=ngp) as s:
        V, out = U.copy(), np.empty_like(U)
        s.Boundary_C(V)
        s.time_stepping(V, out, 0.0, 1e-4)
        return out[4:-4, 4:-4]


@pytest.mark.parametrize("lf,nf", [(4, 4), (31, 5), (32, 4), (33, 9), (64, 7), (65, 33), (5, 70)])
@pytest.mark.parametrize("decades", [0.0, 0.15])
@pytest.mark.parametrize("mord,ngp", [(5, 3), (5, 2), (3, 3), (3, 2)])
def test_tile_edges_equal_exact(pkg, lf, nf, decades, mord, ngp):
    U = _state(lf, nf, decades)
    a, b = _step(pkg, U, pkg.FP_EXACT, mord, ngp), _step(pkg, U, pkg.FP_FAST, mord, ngp)
    # ~40 rounded operations on values of the cell's own density or energy (x10 for its neighbours'): 1e-13 of them
    assert np.isfinite(a).all()
    size = np.maximum(a[..., :1], a[..., 3:])
    assert np.all(np.abs(a - b) <= 1e-13 * (10.0 if decades else 1.0) * size), np.max(np.abs(a - b) / size)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("var", [0, 3])
def test_non_finite_cells_spread_as_in_exact(pkg, bad, var):
    U = _state(40, 11, 0.0)
    U[9, 36, var] = bad  # next to a tile's right edge
    a, b = _step(pkg, U, pkg.FP_EXACT), _step(pkg, U, pkg.FP_FAST)
    fa, fb = np.isfinite(a).all(axis=-1), np.isfinite(b).all(axis=-1)
    assert not fa.all() and np.array_equal(fa, fb)
