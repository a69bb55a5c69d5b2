"""Restart lengths at which the shared memory of the back substitution (407
columns) and of the classical Gram-Schmidt update (from 612) first passes what
a launch gets without opting in, its static part included (needs a B200): the
restart cycle still runs on the device.  A solve that converges inside its first
cycle launches the same kernels whatever the restart length; the host-driven
cycle launches others."""
import numpy as np
import pytest

from helpers import mode_n_solver, mode_r_case, mode_r_solver, rand_c, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu

RESTARTS = (300, 407, 612, 620)


def test_mode_r():
    g, st = mode_r_case(10, 4, 3)
    f = rand_c(g.shape_zyx, seed=3)
    seen = set()
    for m in RESTARTS:
        s = mode_r_solver(g, st, tol=1e-11, restart=m, max_iter=3000)
        before = s.kernel_launches
        u = s.solve(f)
        assert np.linalg.norm(st.apply_a(u) - f) / np.linalg.norm(f) < 1e-9
        seen.add((s.last_stats.iterations, s.kernel_launches - before))
        s.close()
    assert len(seen) == 1 and min(seen)[0] < min(RESTARTS), seen


def test_classical_gram_schmidt(monkeypatch):
    monkeypatch.setenv("HELM3D_GS", "cgs2")
    p = small_problem(12, 11, 9, pml=3, seed=41)
    on = mode_n.setup(p, factor=False)
    f = rand_c(p.shape, seed=50)
    seen = set()
    for m in RESTARTS:
        s = mode_n_solver(p, precision=1, tol=1e-10, restart=m)
        before = s.kernel_launches
        u = s.solve(f)
        assert np.linalg.norm(on.apply_a(u) - f) / np.linalg.norm(f) < 2e-10
        seen.add((s.last_stats.iterations, s.kernel_launches - before))
        s.close()
    assert len(seen) == 1 and min(seen)[0] < min(RESTARTS), seen
