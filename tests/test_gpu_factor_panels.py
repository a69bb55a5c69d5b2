"""The complex64 factors at the edges of their panels of 16 columns: one panel
and a partial one, the last panel full and partial, the first size with two and
with three panels (columns left of, right of and between panels p and p + 1),
both sides of 128 rows (one CTA, a CTA pair) and the largest; and more chains
than the GPU holds at once, two CTAs to an SM.  Every factor variant against the
FP64 oracle (needs a B200).  Tolerance as in test_gpu_parity: 5e-5."""
import pytest

from helpers import mode_n_solver, rand_c, rel, small_problem
from oracle import mode_n

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(5, 5, 4), (15, 6, 4), (16, 5, 4), (17, 5, 4), (32, 5, 4), (33, 6, 4), (48, 5, 4),
                                      (49, 4, 4), (96, 5, 4), (97, 4, 4), (112, 5, 4), (113, 5, 4), (127, 5, 4),
                                      (128, 6, 4), (129, 5, 4), (144, 5, 4), (208, 5, 4), (209, 4, 4), (224, 5, 4),
                                      (40, 4, 320), (136, 4, 160)])
def test_every_variant(nx, ny, nz, monkeypatch):
    p = small_problem(nx, ny, nz, pml=1, seed=nx + nz)
    v = rand_c(p.shape, seed=5)
    on = mode_n.setup(p, beta_prec=0.25)
    ref, refh = on.apply_prec(v), on.apply_prec_adjoint(v)
    for var in range(4):
        monkeypatch.setenv("HELM3D_FORCE_FACTOR", str(var))
        s = mode_n_solver(p, precision=1, beta_prec=0.25)
        assert rel(s.apply_prec(v), ref) < 5e-5, var
        assert rel(s.apply_prec_adjoint(v), refh) < 5e-5, var
        s.close()
