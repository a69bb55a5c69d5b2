"""The operator and its adjoint at the grids where each of its launch shapes is
the default one (1, 4, 6 and 8 planes per block) with ragged edges in x, y and z
(needs a B200).  Tolerance as in test_gpu_parity: 1e-13."""
import numpy as np
import pytest

from helpers import mode_n_solver, rand_c, rel, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(31, 7, 3), (33, 9, 13), (50, 51, 53), (65, 63, 151), (70, 66, 203)])
def test_operator_shapes(nx, ny, nz):
    p = small_problem(nx, ny, nz, pml=1, seed=nx)
    on = mode_n.setup(p, factor=False)
    s = mode_n_solver(p, precision=1)
    x, y = rand_c(p.shape, seed=1), rand_c(p.shape, seed=2)
    ax, ahy = s.apply_op(x), s.apply_op_adjoint(y)
    s.close()
    assert rel(ax, on.apply_a(x)) < 1e-13
    lhs, rhs = np.vdot(y, on.apply_a(x)), np.vdot(ahy, x)
    assert abs(lhs - rhs) < 1e-12 * np.linalg.norm(y) * np.linalg.norm(ax)
