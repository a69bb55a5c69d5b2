"""A gradient gives back the device memory of its wavefields: what it leaves
allocated is what the solves of its batch leave (needs a B200)."""
import numpy as np
import pytest

from helpers import mode_n_solver, rand_c, small_problem

pytestmark = pytest.mark.gpu


def test_wavefields_are_given_back():
    import torch
    nsrc = 8
    p = small_problem(64, 64, 64, pml=6, seed=7)
    F = torch.from_numpy(np.stack([rand_c(p.shape, seed=r) for r in range(nsrc)])).cuda()
    recv = np.arange(0, p.nx * p.ny * p.nz, 9973, dtype=np.int64)
    d = rand_c((nsrc, recv.size), seed=3)
    s = mode_n_solver(p, precision=1, tol=1e-6)
    s.solve(F, nrhs=nsrc)
    s.solve_adjoint(F[0])
    held, free = s.device_bytes, torch.cuda.mem_get_info()[0]
    s.misfit_grad(F, recv, d)
    wavefields = 3 * F.numel() * F.element_size()
    assert s.device_bytes == held
    # (the adjoint batch's cycle graph and the allocator's granularity remain)
    assert free - torch.cuda.mem_get_info()[0] < wavefields // 2
    s.close()
