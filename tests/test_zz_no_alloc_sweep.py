"""helm3d_apply_prec_noalloc launches the sweep that helm3d_apply_prec does before
any solve was tuned: bit for bit the same result, at block sizes whose lines are
several stages of the sweep's ring (needs a B200)."""
import ctypes

import pytest

from helpers import mode_n_solver, rand_c, small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,nx,ny,nz", [(1, 94, 20, 16), (1, 150, 10, 8), (0, 57, 20, 16), (0, 130, 10, 8), (0, 20, 12, 9)])
def test_same_sweep(prec, nx, ny, nz):
    import torch

    import helm3d
    fn = helm3d.lib.helm3d_apply_prec_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    p = small_problem(nx, ny, nz, pml=3, seed=nx)
    s = mode_n_solver(p, precision=prec)
    x = torch.from_numpy(rand_c(p.shape, seed=2)).cuda()
    y = torch.full_like(x, float("nan"))
    ref = s.apply_prec(x)
    assert fn(s.h, x.data_ptr(), y.data_ptr()) == helm3d.OK
    assert torch.equal(y, ref)
    s.close()
