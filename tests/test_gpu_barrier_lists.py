"""A MOOD loop whose grid barrier ran out leaves no list behind: the step's later
stages list their own cells only.  Nearly every cell is troubled in every stage
here, so lists added up over the three stages would be three times as long as
they may be.  Afterwards the context steps as the oracle does, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import nan_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lf,nf", [(64, 48), (257, 130)])
def test_lists_of_a_timed_out_step_do_not_add_up(pkg, oracle, lf, nf):
    p = oracle.make_params(lf, nf, bc=18, tmax=0.8)
    rng = np.random.default_rng(lf)
    U = np.empty((nf + 8, lf + 8, 4))
    r = rng.uniform(0.2, 5.0, U.shape[:2])
    u, v = rng.uniform(-3, 3, r.shape), rng.uniform(-3, 3, r.shape)
    U[..., 0], U[..., 1], U[..., 2], U[..., 3] = r, r * u, r * v, 1 / 0.4 + 0.5 * r * (u * u + v * v)
    oracle.boundary(p, U, 0.0)
    dt = oracle.setdt(p, U, p.tmax)
    # one unlimited Euler step of the long dt: a cell it leaves inadmissible is troubled in the first stage's first
    # pass, and then, starting from there, in the later stages'
    far = np.empty_like(U)
    oracle.Stepper(oracle.make_params(lf, nf, bc=18, tmax=0.8, method=202, integrator=8)).time_stepping(
        U.copy(), far, 0.0, 50 * dt)
    f = far[4:-4, 4:-4]
    press = 0.4 * (f[..., 3] - 0.5 * (f[..., 1] ** 2 + f[..., 2] ** 2) / f[..., 0])
    assert (~((f[..., 0] > 0) & (press > 0))).mean() > 0.6
    ref = np.empty_like(U)
    oracle.Stepper(p).time_stepping(U.copy(), ref, 0.0, dt)
    with pkg.Solver(lf=lf, nf=nf, bc_type=18, tmax=0.8, fp_mode=pkg.FP_EXACT) as s:
        for _ in range(2):
            out = np.empty_like(U)
            s.set_wait_limit(1)
            with pytest.raises(pkg.GpmoodError) as e:
                s.time_stepping(U.copy(), out, 0.0, 50 * dt)
            assert e.value.code == -2 and "barrier" in str(e.value)
            s.set_wait_limit(0)
            s.time_stepping(U.copy(), out, 0.0, dt)
            assert nan_equal(out, ref)
