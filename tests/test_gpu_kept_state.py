"""What a context keeps between calls: group cycles (captured once, used while
nothing they hold has moved), the gradient's wavefields, the cleared status word
(needs a B200).  Each call's results are those of a fresh context, whatever was
called before (solutions 1e-8 relative, gradients 1e-6, as elsewhere)."""
import numpy as np
import pytest

from helpers import mode_n_solver, rand_c, rel, small_problem

pytestmark = pytest.mark.gpu


def test_group_cycles_follow_their_contexts():
    """The same group again, with another medium, after one of its contexts has
    solved a larger batch (its workspace moves) and after one was replaced."""
    import helm3d
    probs = [small_problem(16, 14, 12, pml=3, seed=61), small_problem(20, 17, 15, pml=4, seed=62)]
    ss = [mode_n_solver(p, precision=1, tol=1e-10, z_transform=helm3d.ZT_PML_EIGEN) for p in probs]
    F = [rand_c(p.shape, seed=70 + i) for i, p in enumerate(probs)]

    def check(media):
        U = helm3d.solve_group(ss, F)
        for p, m, f, u in zip(probs, media, F, U):
            fresh = mode_n_solver(p, precision=1, tol=1e-10, z_transform=helm3d.ZT_PML_EIGEN)
            fresh.set_medium(m)
            assert rel(u, fresh.solve(f)) < 1e-8
            fresh.close()

    media = [p.s2 for p in probs]
    check(media)
    media = [p.s2 * 1.02 for p in probs]
    for s, m in zip(ss, media):
        s.set_medium(m)
    check(media)
    ss[1].solve(np.stack([F[1]] * 3), nrhs=3)
    check(media)
    ss[1].close()
    ss[1] = mode_n_solver(probs[1], precision=1, tol=1e-10, z_transform=helm3d.ZT_PML_EIGEN)
    check([media[0], probs[1].s2])
    for s in ss:
        s.close()


def test_skipped_modes_follow_the_medium():
    """kz_skip_ratio: another medium skips other modes; solves before and after."""
    p = small_problem(18, 16, 24, pml=3, seed=63)
    f = rand_c(p.shape, seed=5)
    s = mode_n_solver(p, precision=1, tol=1e-9, kz_skip_ratio=1.0)
    for scale in (1.0, 4.0, 0.3):
        s.set_medium(p.s2 * scale)
        fresh = mode_n_solver(p, precision=1, tol=1e-9, kz_skip_ratio=1.0)
        fresh.set_medium(p.s2 * scale)
        a, b = (x.solve(f, allow_not_converged=True) for x in (s, fresh))
        assert s.last_stats.iterations == fresh.last_stats.iterations
        assert rel(a, b) < 1e-7
        fresh.close()
    s.close()


def test_gradient_wavefields_are_reused():
    """Gradients of 2, 5 and again 2 sources, solves between them."""
    p = small_problem(18, 16, 14, pml=3, seed=64)
    s = mode_n_solver(p, precision=1, tol=1e-10)
    recv = np.arange(700, 1100, 37, dtype=np.int64)
    for k in (2, 5, 2):
        F = np.stack([rand_c(p.shape, seed=80 + r) for r in range(k)])
        d = np.stack([rand_c((recv.size,), seed=90 + r) for r in range(k)])
        J, g = s.misfit_grad(F, recv, d)
        fresh = mode_n_solver(p, precision=1, tol=1e-10)
        J1, g1 = fresh.misfit_grad(F, recv, d)
        assert abs(J - J1) <= 1e-8 * abs(J1) and rel(g, g1) < 1e-6
        assert rel(s.solve(F[0]), fresh.solve(F[0])) < 1e-8
        fresh.close()
    s.close()
