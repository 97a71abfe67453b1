"""Exact mode with infinite energies in the state: such a cell's sides are
admissible (p = +inf), its wave speeds are infinite and the contact speed NaN,
and HLLC_Flux then takes its last branch, the right state's physical flux
(every comparison with NaN is false), so a finite cell to the right stays
finite.  One step against the oracle, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import nan_equal

pytestmark = pytest.mark.gpu


def states(oracle, lf, nf, flow, mord, ngp):
    p = oracle.make_params(lf, nf, bc=18, tmax=0.8, mord=mord, ngp=ngp)
    y, x = np.meshgrid(np.arange(nf + 8), np.arange(lf + 8), indexing="ij")
    r = 1 + 0.1 * np.sin(0.3 * x) * np.cos(0.2 * y)
    u, v = flow[0] + 0 * r, flow[1] + 0 * r
    U = np.ascontiguousarray(np.stack([r, r * u, r * v, 1 / 0.4 + 0.5 * r * (u * u + v * v)], axis=-1))
    for j, i in ((15, 14), (22, 30), (23, 30)):
        U[j, i, 3] = np.inf
    oracle.boundary(p, U, 0.0)
    return p, U


@pytest.mark.parametrize("mord,ngp", [(5, 3), (3, 2), (1, 1)])
@pytest.mark.parametrize("flow", [(0.0, 0.0), (0.3, -0.2), (4.0, -4.0), (-4.0, 4.0)])
def test_infinite_energies_equal_the_oracle(pkg, oracle, flow, mord, ngp):
    lf, nf = 45, 36
    p, U = states(oracle, lf, nf, flow, mord, ngp)
    ref = np.empty_like(U)
    oracle.Stepper(p).time_stepping(U.copy(), ref, 0.0, 1e-3)
    kw = dict(bc_type=18, tmax=0.8, mord=mord, ngp=ngp, fp_mode=pkg.FP_EXACT)
    with pkg.Solver(lf=lf, nf=nf, **kw) as s:
        out = np.empty_like(U)
        s.time_stepping(U.copy(), out, 0.0, 1e-3)
    assert np.isfinite(ref).all(axis=-1).sum() < ref[..., 0].size
    assert nan_equal(out, ref)
