"""The two-ended block factor and sweep (half chains meeting at the middle
y-line) where the halves can go wrong: one or two lines in all (a half without
lines), even and odd line counts, every factor and sweep kernel, one and
several right-hand sides, forward and adjoint, against the FP64 oracle (needs
a B200).  Tolerances as in test_gpu_parity: 1e-9 (complex128 preconditioner),
5e-5 (complex64)."""
import numpy as np
import pytest

from helpers import mode_n_solver, rand_c, rel, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,pml", [(9, 2, 0), (20, 3, 1), (33, 4, 1), (64, 5, 2), (130, 2, 0), (150, 3, 1), (100, 7, 3)])
@pytest.mark.parametrize("prec", [0, 1])
def test_half_chains(nx, ny, pml, prec, monkeypatch):
    nz, nrhs = 6, 3
    p = small_problem(nx, ny, nz, pml=pml, seed=nx + ny)
    on = mode_n.setup(p, beta_prec=0.25)
    X = np.stack([rand_c(p.shape, seed=7 + r) for r in range(nrhs)])
    ref = [on.apply_prec(x) for x in X]
    refh = [on.apply_prec_adjoint(x) for x in X]
    tol = 5e-5 if prec else 1e-9
    for factor in (0, 1, 2):
        monkeypatch.setenv("HELM3D_FORCE_FACTOR", str(factor))
        s = mode_n_solver(p, precision=prec, beta_prec=0.25)
        for sweep in (0, 1, 6, 9):
            monkeypatch.setenv("HELM3D_FORCE_SWEEP", str(sweep))
            for k in (1, nrhs):
                Y, Yh = s.apply_prec_batch(X[:k]), s.apply_prec_batch(X[:k], adjoint=True)
                for r in range(k):
                    assert rel(Y[r], ref[r]) < tol, (factor, sweep, k, r)
                    assert rel(Yh[r], refh[r]) < tol, (factor, sweep, k, r)
        s.close()
