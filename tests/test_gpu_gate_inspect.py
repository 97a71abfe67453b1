"""Looking at the gate between steps (nn_predict, nn_gate_logits) leaves the next
step as it would have been: those calls list the gated cells as a step does, and
a step's own lists start empty.  With few gated cells and the extras repair on a
leftover list would take each cell off the a-priori count twice; with every cell
gated it would outgrow the list.  Bits, orders and counters against a solver that
made no such call."""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GATE = Path(__file__).resolve().parents[1] / "gp-mood_gb300" / "gates" / "gate_sedov_rp2d3.txt"
LF, NF = 77, 53


def state(oracle):
    """2DRP3 after five steps with a ripple, so that no stencil is constant."""
    p = oracle.make_params(LF, NF, bc=17, tmax=0.8)
    U = oracle.initial_condition(p, "rp2d3")
    oracle.Stepper(p).run(U, 0.0, 5)
    y, x = np.meshgrid(np.arange(NF + 8), np.arange(LF + 8), indexing="ij")
    U *= 1 + 1e-3 * (np.sin(1.1 * x) * np.cos(0.7 * y))[..., None]
    return U


def run(pkg, U, fp, threshold, repair, look, resident):
    from gpmood_gb300 import nn_train as T
    params = T.load_text(str(GATE))
    with pkg.Solver(lf=LF, nf=NF, bc_type=17, tmax=0.8, method=pkg.NN_GP_MOOD, fp_mode=fp) as s:
        s.Boundary_C(U, 0.0)
        s.set_nn(params)
        s.set_nn_threshold(threshold)
        s.set_nn_repair(repair)
        s.set_state(U, 0.0)
        out, counts = [], []
        gated = 0
        for _ in range(2):
            if look:
                z = torch.empty(LF * NF, dtype=torch.float32, device="cuda")
                s.nn_gate_logits(z.data_ptr())
                gated = s.nn_predict()[1]
            if resident:
                assert s.advance(1) == 1
                out.append(s.get_state()[0])
            else:
                V = np.empty_like(U)
                s.time_stepping(U, V, 0.0, 1e-4)
                out.append(V)
                s.set_state(U, 0.0)
            out += [s.stage_orders(k) for k in range(3)]
            c = s.counters()
            counts += [c.a_priori_last_step, c.detected_last_step, c.mood_passes_last_step]
    return out, counts, gated


@pytest.mark.parametrize("resident", [True, False])
@pytest.mark.parametrize("repair", [False, True])
@pytest.mark.parametrize("threshold", [0.0, -1e30])
@pytest.mark.parametrize("fp", [0, 1])
def test_a_look_at_the_gate_does_not_change_the_next_step(pkg, oracle, fp, threshold, repair, resident):
    U = state(oracle)
    ref, nref, _ = run(pkg, U.copy(), fp, threshold, repair, False, resident)
    got, ngot, gated = run(pkg, U.copy(), fp, threshold, repair, True, resident)
    assert 0 < gated < LF * NF // 2 if threshold == 0.0 else gated == LF * NF
    assert ngot == nref
    assert min(nref) >= 0
    for a, b in zip(got, ref):
        assert np.array_equal(a.view(np.int64) if a.dtype == np.float64 else a,
                              b.view(np.int64) if b.dtype == np.float64 else b)
