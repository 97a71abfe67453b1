"""Device memory of a destroyed adjoint recording: a small one's block is kept
for the solver's next recording and freed with the solver, a large one's (over
64 MB) is freed at once, so that another allocation can have it."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("n,kept", [(64, True), (640, False)])
def test_a_destroyed_recording_gives_its_memory_back(pkg, n, kept):
    from gpmood_gb300 import ic
    U = ic.isentropic_vortex(n, n, 10.0, 10.0, beta=5.0)
    size = (n + 8) ** 2 * (6 * 32 + 3 * 32 + 7 * 32 + 640)  # adjoint buffers, checkpoints, stage inputs, faces
    with pkg.Solver(lf=n, nf=n, lx=10.0, ly=10.0, bc_type=pkg.PERIODIC, tmax=1e30, fp_mode=0) as s:
        s.Boundary_C(U, 0.0)
        for _ in range(2):
            s.set_state(U, 0.0)
            before = free_bytes()
            rec = s.adj_record(6, 2)
            held = before - free_bytes()
            rec.close()
            after = free_bytes()
            if not kept:
                assert held >= 0.9 * size
                assert before - after <= 0.1 * size, (before, after, size)
        if kept:
            assert before - after <= 4 << 20  # the second recording took the first one's block
        outlives = s.adj_record(6, 2)
        start = free_bytes()
    outlives.close()
    assert free_bytes() - start >= 0.9 * size
