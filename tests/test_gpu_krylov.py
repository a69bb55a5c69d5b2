"""The Gram-Schmidt passes and the bookkeeping they end with, at the sizes where
they can go wrong: cycles longer than the 64 vectors a block keeps sums of, and
than the 32 columns the back substitution stages; one-step cycles; grids smaller
than a tile and not a multiple of it; batches whose right-hand sides stop at
different steps, one of them zero (needs a B200).  The solutions are held to the
requested residual by the oracle's operator, and graph cycles to host-driven
ones (solutions as in test_gpu_parity: 1e-8 relative)."""
import numpy as np
import pytest

from helpers import mode_n_solver, mode_r_case, mode_r_solver, rand_c, rel, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,restart", [((12, 11, 9), 1), ((12, 11, 9), 90), ((21, 17, 13), 33), ((21, 17, 13), 70)])
@pytest.mark.parametrize("gs", ["dcgs2", "cgs2"])
def test_cycle_lengths(shape, restart, gs, monkeypatch):
    p = small_problem(*shape, pml=3, seed=41)
    on = mode_n.setup(p, factor=False)
    F = np.stack([rand_c(p.shape, seed=50), np.zeros(p.shape, complex), p.rhs(0) + 0j])
    monkeypatch.setenv("HELM3D_GS", gs)
    # one step per cycle: what such a cycle can reach, the same by graphs and by the host
    tol, it = (1e-10, 4000) if restart > 1 else (1e-30, 6)
    out = []
    for graph in ("1", "0"):
        monkeypatch.setenv("HELM3D_GRAPH", graph)
        s = mode_n_solver(p, precision=1, tol=tol, restart=restart, max_iter=it)
        U = s.solve(F, nrhs=3, allow_not_converged=restart == 1)
        s.close()
        assert not np.any(U[1])
        if restart > 1:
            for r in (0, 2):
                assert np.linalg.norm(on.apply_a(U[r]) - F[r]) / np.linalg.norm(F[r]) < 2e-10
        out.append(U)
    assert rel(out[0], out[1]) < 1e-8


def test_mode_r_long_cycle():
    g, st = mode_r_case(10, 4, 3)
    f = rand_c(g.shape_zyx, seed=3)
    u = [mode_r_solver(g, st, tol=1e-11, restart=m, max_iter=3000).solve(f) for m in (30, 100)]
    for x in u:
        assert np.linalg.norm(st.apply_a(x) - f) / np.linalg.norm(f) < 1e-9
    assert rel(u[0], u[1]) < 1e-8
