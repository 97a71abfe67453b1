"""The gate's features narrow FP64 states to FP32 in integer instructions: the
same floats as a conversion, for ties, values next to them, zeros, results that
are subnormal or overflow, and infinities."""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nno(oracle):
    import nn_oracle
    return nn_oracle


def values(kind, shape):
    rng = np.random.default_rng(17)
    mant = rng.integers(0, 1 << 52, shape, dtype=np.uint64)
    low = np.uint64((1 << 29) - 1)
    if kind != "any":  # the part below a float's last place: half, just below, just above, or none
        tail = rng.choice(np.array([1 << 28, (1 << 28) - 1, (1 << 28) + 1, 0], dtype=np.uint64), shape)
        mant = (mant & ~low) | tail
        mant = np.where(rng.random(shape) < 0.1, (np.uint64((1 << 52) - 1) & ~low) | tail, mant)  # carries out
    lo, hi = {"any": (-60, 60), "ties": (-60, 60), "edges": (-160, 128)}[kind]
    e = rng.integers(lo, hi, shape)
    if kind == "edges":
        e = np.where(rng.random(shape) < 0.5, rng.choice([-150, -149, -127, -126, 126, 127, 128, 1000], shape), e)
    x = ((e + 1023).astype(np.uint64) << np.uint64(52) | mant).view(np.float64) * rng.choice([-1.0, 1.0], shape)
    if kind == "edges":
        x = np.where(rng.random(shape) < 0.05, rng.choice([0.0, -0.0, np.inf, 5e-324], shape), x)
    return x


@pytest.mark.parametrize("kind", ["any", "ties", "edges"])
def test_features_are_the_converted_states(pkg, nno, kind):
    lf, nf = 67, 45
    U = np.ascontiguousarray(values(kind, (nf + 8, lf + 8, 4)))
    with pkg.Solver(lf=lf, nf=nf, bc_type=17) as s:
        s.set_state(U, 0.0)
        x = torch.empty((lf * nf, 36), dtype=torch.float32, device="cuda")
        c = torch.empty((lf * nf,), dtype=torch.int8, device="cuda")
        s.nn_features(x.data_ptr(), c.data_ptr())
    with np.errstate(all="ignore"):
        xr, cr = nno.features(U, lf, nf)
    assert np.array_equal(x.cpu().numpy(), xr, equal_nan=True)
    assert np.array_equal(c.cpu().numpy().astype(bool), cr)
