"""The first solve of a batch times each sweep that is another launch once (one
warm-up and three timed launches), and none twice under two numbers (needs a
B200)."""
import pytest

from cuda_kernels import kernels
from helpers import mode_n_solver, rand_c, small_problem

pytestmark = pytest.mark.gpu


# complex128: the six shapes of the CUDA-core kernel; complex64 beyond 128 rows
# two of the tensor-core kernel more, up to 128 rows four
@pytest.mark.parametrize("prec,nx,own", [(0, 23, 6), (1, 131, 8), (1, 23, 10)])
def test_sweeps_timed(prec, nx, own, tmp_path, monkeypatch):
    import torch
    monkeypatch.delenv("HELM3D_TUNE_CACHE", raising=False)
    p = small_problem(nx, 13, 11, pml=3, seed=8)
    f = torch.from_numpy(rand_c(p.shape, seed=4)).cuda()
    s = mode_n_solver(p, precision=prec, tol=1e-6)
    first, again = [sum("sweep" in n for n, _ in kernels(lambda: s.solve(f), tmp_path)) for _ in range(2)]
    s.close()
    assert first - again == 4 * own
