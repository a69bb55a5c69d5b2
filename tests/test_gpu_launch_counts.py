"""The launch counts that the library reports for a new medium are the kernels
that ran: the factor's halves and middle lines, and for complex64 the block
scales and the packing (needs a B200)."""
import pytest

from cuda_kernels import kernels
from helpers import mode_n_solver, small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_factor_launches(prec, tmp_path):
    p = small_problem(20, 12, 8, pml=3, seed=5)
    s = mode_n_solver(p, precision=prec)
    s.profile(True)
    s.profile_read()
    before = s.kernel_launches
    ran = [n for n, _ in kernels(lambda: s.set_medium(p.s2), tmp_path)]
    mine = [n for n in ran if "factor" in n or "gscale" in n or "gpack" in n]
    assert len(mine) == (4 if prec else 2), ran
    assert s.profile_read()["factor"][1] == len(mine)
    assert s.kernel_launches - before == len(ran), ran
    s.close()
