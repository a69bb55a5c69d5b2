"""The register factor of the smallest blocks leaves room for a second CTA on an
SM (complex128, 256 threads) and for a fourth (complex64, 128 threads): at most
128 registers in the kernel of the halves and in that of the middle lines (needs a
B200)."""
import pytest

from cuda_kernels import in_child

pytestmark = pytest.mark.gpu


def test_registers():
    got = in_child("""
        out = []
        for prec in (0, 1):
            p = small_problem(20, 12, 8, pml=3, seed=6)
            s = mode_n_solver(p, precision=prec)
            out.append([k for k in kernels(lambda: s.set_medium(p.s2)) if "factor_kernel" in k[0]])
        """, HELM3D_FORCE_FACTOR="0")
    for ran in got:
        assert len(ran) == 2 and all(regs <= 128 for _, regs in ran), ran
