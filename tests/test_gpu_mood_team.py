"""MOOD passes on one cluster over lists of every size class: cross cells of up
to and beyond the four-lane update's, lists up to and beyond the shared-cell
scan's, and lists that the all-SM passes hand over.  m spots of dense, fast gas
in a smooth flow give lists of about that length.  Exact mode: bit for bit
against the oracle.  Fast mode: the prepared crosses against one thread per
cross cell with nothing prepared, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spots(pkg, lf, nf, m, fp):
    rng = np.random.default_rng(100 + m)
    y, x = np.meshgrid(np.arange(nf + 8), np.arange(lf + 8), indexing="ij")
    r = 1 + 0.1 * np.sin(2 * np.pi * x / lf) * np.cos(2 * np.pi * y / nf)
    u, v, p = 0.5 + 0 * r, 0.2 + 0 * r, 1 + 0 * r
    at = rng.choice(lf * nf, m, replace=False)
    j, i = at // lf + 4, at % lf + 4
    r[j, i] *= 4
    u[j, i] = 3 * rng.choice([-1.0, 1.0], m)
    v[j, i] = 3 * rng.choice([-1.0, 1.0], m)
    U = np.ascontiguousarray(np.stack([r, r * u, r * v, p / 0.4 + 0.5 * r * (u * u + v * v)], axis=-1))
    s = pkg.Solver(lf=lf, nf=nf, bc_type=18, tmax=0.5, fp_mode=fp)
    s.Boundary_C(U)
    return s, U


@pytest.mark.parametrize("m", [1, 2, 4, 8, 20, 60])
def test_team_passes_equal_oracle(pkg, oracle, m):
    lf, nf = 61, 47
    s, U = spots(pkg, lf, nf, m, pkg.FP_EXACT)
    p = oracle.make_params(lf, nf, bc=18, tmax=0.5)
    st = oracle.Stepper(p)
    with s:
        s.set_state(U, 0.0)
        assert s.advance(2) == 2
        got, t, _ = s.get_state()
        assert s.counters().max_passes_stage > 2
    ref = U.copy()
    assert st.run(ref, 0.0, 2) == (t, 2)
    assert np.array_equal(got[4:-4, 4:-4], ref[4:-4, 4:-4])


@pytest.mark.parametrize("m", [1, 4, 20, 60])
def test_prepared_crosses_agree(pkg, m, monkeypatch):
    out = []
    for split in ("1", "0"):
        monkeypatch.setenv("GPMOOD_SOLO_SPLIT", split)
        s, U = spots(pkg, 61, 47, m, pkg.FP_FAST)
        with s:
            s.set_state(U, 0.0)
            assert s.advance(2) == 2
            V, t, _ = s.get_state()
            out.append((V, t, s.counters().detected_total))
    assert out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])
