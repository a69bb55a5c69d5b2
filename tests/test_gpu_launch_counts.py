"""The launch counts that the library reports for a new medium are the kernels
that ran: the factor's halves and middle lines, and for complex64 the block
scales and the packing (needs a B200)."""
import pytest

from cuda_kernels import in_child

pytestmark = pytest.mark.gpu


def test_factor_launches():
    got = in_child("""
        out = []
        for prec in (0, 1):
            p = small_problem(20, 12, 8, pml=3, seed=5)
            s = mode_n_solver(p, precision=prec)
            s.profile(True)
            s.profile_read()
            before = s.kernel_launches
            ran = [n for n, _ in kernels(lambda: s.set_medium(p.s2))]
            out.append((ran, s.profile_read()["factor"][1], s.kernel_launches - before))
        """)
    for (ran, factor, launches), expected in zip(got, (2, 4)):
        mine = [n for n in ran if "factor" in n or "gscale" in n or "gpack" in n]
        assert len(mine) == expected, ran
        assert factor == len(mine)
        assert launches == len(ran), ran
