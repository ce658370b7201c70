"""The direct y solve on fields long in both directions (the largest chunk lengths with
many columns) against the CPU oracle; tolerance 1e-13, the operator-level solve bar."""
import numpy as np
import pytest

from fixtures import rel_l2
from test_gpu_dense_cg import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(600, 648), (540, 1000), (1000, 576), (810, 768), (1024, 1024)])
def test_solves_match_oracle(ib, orc, nx, ny):
    prob = _problem(ib, 4, nx=nx, ny=ny, L=2)
    s = ib.create_solver(ib.State(prob), cg=dict(maxiter=1))
    lam = orc.lap_eigs(nx, ny)
    rng = np.random.default_rng(nx + ny)
    mode = np.outer(np.sin(np.pi * np.arange(1, nx) / nx), np.sin(np.pi * np.arange(1, ny) / ny))
    for b in (rng.standard_normal((nx - 1, ny - 1)), mode):
        assert rel_l2(s.diag_solve(0, 1, b), orc.lap_inv(nx, ny, lam, b)) < 1e-13
        for lev in (1, 2):
            h = prob.grid.gridstep(lev)
            den = 1 + lam * prob.scheme.dt / (2 * prob.fluid.Re * h ** 2)
            assert rel_l2(s.diag_solve(2, lev, b), orc.lap_inv(nx, ny, den, b)) < 1e-13
