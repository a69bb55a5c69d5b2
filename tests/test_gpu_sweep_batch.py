"""Batches of right-hand sides in the block sweep, at the edges of its splits:
rows per warp and warps per line (8, 16 or 32 rows; odd counts, whose last
thread owns one row), one and several stages to a line, right-hand sides below,
at and above the padded counts 4, 8 and 16 (above 8 in two groups: complex128, and
complex64 where that fills the last wave),
forward and adjoint, against the FP64 oracle (needs a B200).  Tolerances as in
test_gpu_parity: 1e-9 (complex128 preconditioner), 5e-5 (complex64)."""
import numpy as np
import pytest

from helpers import mode_n_solver, rand_c, rel, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu


def check(nx, ny, nz, batches, prec):
    p = small_problem(nx, ny, nz, pml=1, seed=nx)
    on = mode_n.setup(p, beta_prec=0.25)
    X = np.stack([rand_c(p.shape, seed=300 + r) for r in range(max(batches))])
    ref = [on.apply_prec(x) for x in X]
    refh = [on.apply_prec_adjoint(x) for x in X]
    s = mode_n_solver(p, precision=prec, beta_prec=0.25)
    tol = 5e-5 if prec else 1e-9
    for k in batches:
        Y, Yh = s.apply_prec_batch(X[:k]), s.apply_prec_batch(X[:k], adjoint=True)
        for r in range(k):
            assert rel(Y[r], ref[r]) < tol, (k, r)
            assert rel(Yh[r], refh[r]) < tol, (k, r)
    s.close()


@pytest.mark.parametrize("nx,batches", [(5, (3, 16)), (31, (5, 9)), (33, (4, 8)), (64, (5, 16)), (65, (3, 8)), (96, (16,)),
                                        (97, (4, 9)), (128, (16,)), (129, (3, 16)), (193, (8,)), (240, (9,)), (255, (5, 16))])
@pytest.mark.parametrize("prec", [0, 1])
def test_batches_match_the_oracle(nx, batches, prec):
    check(nx, 3, 4, batches, prec)


@pytest.mark.parametrize("prec", [0, 1])
def test_groups_of_right_hand_sides(prec):
    check(70, 3, 80, (9, 16), prec)
