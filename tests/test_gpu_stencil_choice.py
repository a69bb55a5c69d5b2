"""Which launch shape the operator takes outside the batch that a solve was tuned
for (needs a B200): on a grid that a single vector does not fill the SMs of, the
default rule's register kernel, whatever a batched solve was tuned or another
family forced to."""
import numpy as np
import pytest

from cuda_kernels import kernels
from helpers import mode_n_solver, rand_c, small_problem

pytestmark = pytest.mark.gpu

DEFAULT = "stencil_kernel<false, double2, 1>"


def stencils(run, tmp_path):
    return [n for n, _ in kernels(run, tmp_path) if "stencil" in n]


def test_other_family_forced(tmp_path, monkeypatch):
    import torch
    monkeypatch.setenv("HELM3D_TUNE", "0")
    monkeypatch.setenv("HELM3D_FORCE_REDUCE", "0")
    p = small_problem(20, 20, 20, pml=4, seed=11)
    s = mode_n_solver(p, precision=0)
    x = torch.from_numpy(rand_c(p.shape, seed=1)).cuda()
    s.solve(x)
    (name,) = stencils(lambda: s.apply_op(x), tmp_path)
    assert DEFAULT in name
    s.close()


def test_after_a_batched_solve(tmp_path, monkeypatch):
    import torch
    nrhs = 16
    p = small_problem(20, 20, 20, pml=4, seed=12)
    F = torch.from_numpy(np.stack([rand_c(p.shape, seed=r) for r in range(nrhs)])).cuda()
    s = mode_n_solver(p, precision=1)
    s.solve(F, nrhs=nrhs)
    (name,) = stencils(lambda: s.apply_op(F[0]), tmp_path)
    assert DEFAULT in name
    s.close()
    # a forced shape holds for every batch
    s = mode_n_solver(p, precision=1)
    monkeypatch.setenv("HELM3D_FORCE_STENCIL", "5")
    ran = stencils(lambda: s.solve(F, nrhs=nrhs), tmp_path)
    assert ran and all(", 12>" in n for n in ran), ran
    (name,) = stencils(lambda: s.apply_op(F[0]), tmp_path)
    assert "stencil_block_kernel<false, double2, 12>" in name
    s.close()
