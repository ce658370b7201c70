"""The direct y solve's tables (4 MB of them at 1024 points, whatever the rows) are
held by the engines that solve so, and not by the FP32 and mixed ones."""
import pytest

from test_gpu_dense_cg import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts", [1, 16])
def test_fp32_handle_holds_no_direct_solve_tables(ib, npts):
    nx, ny = 1024, 16
    prob = _problem(ib, npts, nx=nx, ny=ny, L=1)
    fp32 = ib.GpuCnabSolver(ib.State(prob), precision="fp32").info().device_bytes
    fp64 = ib.GpuCnabSolver(ib.State(prob)).info().device_bytes
    table = 8 * (nx // 2) * (nx - 1)
    assert fp64 > table
    # its fields: some forty arrays of a level's size in 64 bits, and the panels
    assert fp32 < 40 * 8 * nx * ny
