"""Which launch shape the operator takes outside the batch that a solve was tuned
for (needs a B200): on a grid that a single vector does not fill the SMs of, the
default rule's register kernel, whatever a batched solve was tuned or another
family forced to; a forced shape everywhere."""
import pytest

from cuda_kernels import in_child

pytestmark = pytest.mark.gpu

BODY = """
    p = small_problem(20, 20, 20, pml=4, seed=11)
    F = torch.from_numpy(np.stack([rand_c(p.shape, seed=r) for r in range(16)])).cuda()
    s = mode_n_solver(p, precision=1)
    solve = [n for n, _ in kernels(lambda: s.solve(F, nrhs=16)) if "stencil" in n]
    apply = [n for n, _ in kernels(lambda: s.apply_op(F[0]))]
    out = (solve, apply)
    """
DEFAULT = "stencil_kernel<false, double2, 1>"


@pytest.mark.parametrize("env", [{}, {"HELM3D_TUNE": "0"}, {"HELM3D_TUNE": "0", "HELM3D_FORCE_REDUCE": "0"}])
def test_one_vector_after_a_batch(env):
    _, (name,) = in_child(BODY, **env)
    assert DEFAULT in name


def test_forced():
    solve, (name,) = in_child(BODY, HELM3D_FORCE_STENCIL="5")
    assert solve and all(", 12>" in n for n in solve), solve
    assert "stencil_block_kernel<false, double2, 12>" in name
