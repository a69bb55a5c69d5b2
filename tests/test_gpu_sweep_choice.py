"""The first solve of a batch times each sweep that is another launch once (one
warm-up and three timed launches), and none twice under two numbers (needs a
B200)."""
import pytest

from cuda_kernels import in_child

pytestmark = pytest.mark.gpu


def test_sweeps_timed():
    got = in_child("""
        out = []
        for prec, nx in ((0, 23), (1, 131), (1, 23)):
            p = small_problem(nx, 13, 11, pml=3, seed=8)
            f = torch.from_numpy(rand_c(p.shape, seed=4)).cuda()
            s = mode_n_solver(p, precision=prec, tol=1e-6)
            first, again = [sum("sweep" in n for n, _ in kernels(lambda: s.solve(f))) for _ in range(2)]
            out.append(first - again)
        """)
    # complex128: the six shapes of the CUDA-core kernel; complex64 beyond 128
    # rows two of the tensor-core kernel more, up to 128 rows four
    assert got == [4 * 6, 4 * 8, 4 * 10]
