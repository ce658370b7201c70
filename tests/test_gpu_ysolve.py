"""The direct y solve of the DST-diagonalised operators (csrc/ytri.cuh) against
the CPU oracle at the edges of its layouts: every compiled chunk length, rows
that fill the last chunk or leave it nearly empty, the full mode sum (at most 32
rows) and the first size past it, extreme aspect ratios, and diffusion numbers
from none to dominant.  Tolerance 1e-13, the operator-level solve bar."""
import ctypes as C
import importlib

import numpy as np
import pytest

from fixtures import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _lap_inv(ib, b):
    import torch

    lib = importlib.import_module(ib.__name__ + "._abi").load()
    nx, ny = b.shape[0] + 1, b.shape[1] + 1
    bd = torch.from_numpy(np.asfortranarray(b).ravel(order="F")).cuda()
    xd = torch.empty_like(bd)
    rc = lib.ibpm_lap_inv_noalloc(nx, ny, C.c_void_p(bd.data_ptr()), C.c_void_p(xd.data_ptr()),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0, lib.ibpm_noalloc_last_error().decode()
    return xd.cpu().numpy().reshape(b.shape, order="F")


@pytest.mark.parametrize("nx,ny", [(24, 8), (1024, 8), (8, 1024), (96, 32), (1000, 36), (64, 64), (20, 72), (54, 128),
                                   (16, 144), (30, 192), (128, 200), (10, 256), (36, 320), (40, 324), (18, 384),
                                   (200, 400), (300, 512), (12, 540), (24, 640), (48, 648), (60, 768), (80, 800),
                                   (32, 810), (24, 900), (250, 1000), (200, 1024)])
def test_lap_inv_matches_oracle(ib, orc, nx, ny):
    lam = orc.lap_eigs(nx, ny)
    rng = np.random.default_rng(nx * ny)
    mode = np.outer(np.sin(np.pi * np.arange(1, nx) / nx), np.sin(np.pi * np.arange(1, ny) / ny))
    edge = np.zeros((nx - 1, ny - 1))
    edge[0, 0] = edge[-1, -1] = edge[nx // 2, 0] = 1.0
    for b in (rng.standard_normal((nx - 1, ny - 1)), mode, edge):
        x = _lap_inv(ib, b)
        assert rel_l2(x, orc.lap_inv(nx, ny, lam, b)) < TOL


@pytest.mark.parametrize("c", [1e-9, 0.3, 40.0, 1e5])
@pytest.mark.parametrize("n", [24, 72])
def test_implicit_diffusion_matches_oracle(ib, orc, n, c):
    prob = ib.configs.small_cylinder(n, 1, npts=16)
    h = prob.grid.gridstep(1)
    prob.fluid.Re = prob.scheme.dt / (2 * c * h * h)
    s = ib.create_solver(ib.State(prob), cg=dict(maxiter=1))
    b = np.random.default_rng(n).standard_normal((n - 1, n - 1))
    lam = orc.lap_eigs(n, n)
    den = 1 + lam * prob.scheme.dt / (2 * prob.fluid.Re * h ** 2)
    assert rel_l2(s.diag_solve(2, 1, b), orc.lap_inv(n, n, den, b)) < TOL
    assert rel_l2(s.diag_solve(1, 1, b), orc.lap_inv(n, n, 1 / (1 - lam * c), b)) < TOL
