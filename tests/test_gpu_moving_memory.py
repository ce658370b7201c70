"""Column work of a moving-body handle: two columns until a step whose CG may
assemble B, then at most 1 GB more, and a handle that finds no room steps on with
what it has."""
import numpy as np
import pytest

from test_gpu_dense_cg import _problem

pytestmark = pytest.mark.gpu


def test_a_new_handle_holds_two_columns(ib):
    # 225 points never assemble B, so never have more than two columns; their panels
    # take the more memory, but for B itself
    few, many = (ib.GpuCnabSolver(ib.State(_problem(ib, n, nx=512, ny=512, L=4))) for n in (101, 225))
    assert few.info().device_bytes <= many.info().device_bytes + 8 * 202 ** 2
    # the rebuilds' batch of all columns, which the steps do not widen
    few.set_warm_start(None, mode="preconditioned_extrapolated", depth=8)
    held = few.info().device_bytes
    few.advance_()
    assert few.info().device_bytes == held


@pytest.mark.parametrize("nx,ny,L", [(1024, 1024, 2), (1024, 1024, 4), (256, 256, 3)])
def test_steps_add_at_most_one_gigabyte(ib, nx, ny, L):
    s = ib.GpuCnabSolver(ib.State(_problem(ib, 101, nx=nx, ny=ny, L=L)))
    ng, nq = (nx - 1) * (ny - 1), (nx + 1) * ny + nx * (ny + 1)
    column = 8 * ((2 * L + 1) * ng + nq + 2 * (nx + 1) * (ny + 1))
    # two columns, the state's fields (q and q0; psi, two each of Gamma and the nonlinear
    # term, and the right-hand side), a few single-level scratch fields and the tables
    assert s.info().device_bytes <= 2 * column + 8 * (2 * nq * L + (6 * L + 6) * ng) + (32 << 20)
    held = s.info().device_bytes
    s.advance_()
    assert s.info().device_bytes - held <= 1 << 30


def test_no_room_for_columns(ib):
    """A 512 x 512 x 4 handle beside other programs' data: 16 columns are some 436 MB."""
    import torch

    prob = _problem(ib, 101, nx=512, ny=512, L=4)
    a = ib.GpuCnabSolver(ib.State(prob))
    for _ in range(2):
        a.advance_()
    fb = a.state.fb.copy()
    a.close()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (384 << 20), dtype=torch.uint8, device="cuda")
    try:
        b = ib.GpuCnabSolver(ib.State(prob))
        for _ in range(2):
            b.advance_()
        assert np.abs(b.state.fb - fb).max() <= 1e-6 * np.abs(fb).max()
    finally:
        del hold
        torch.cuda.empty_cache()
