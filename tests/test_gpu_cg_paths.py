"""Which form a moving body's CG takes -- B assembled for the step, or applied in
every iteration -- seen through the kernels it launches."""
import numpy as np
import pytest

from test_gpu_dense_cg import _problem

pytestmark = pytest.mark.gpu


def _steps(ib, prob, cg, eager=False, steps=2):
    """kernels, CG iterations and forces of each step"""
    s = ib.GpuCnabSolver(ib.State(prob), cg=cg)
    s.profile(eager)  # a profiled handle launches kernel by kernel, without graphs
    out = []
    for _ in range(steps):
        before = s.kernel_launches()
        s.advance_()
        out.append((s.kernel_launches() - before, s.info().last_cg_iters, s.state.fb.copy()))
    return out


def _first_iteration(ib, prob, **cg):
    """kernels that a step's first CG iteration adds: one application of B and two
    more, or all the applications that assemble B and one more"""
    (without, none, _), = _steps(ib, prob, dict(cg, maxiter=0), steps=1)
    (with_one, one, _), = _steps(ib, prob, dict(cg, maxiter=1), steps=1)
    assert (none, one) == (0, 1)
    return with_one - without


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("npts,cg,assembled", [(101, {}, True), (224, {}, True), (225, {}, False),
                                               (40, dict(reltol=0.2), False)])
def test_path_taken(ib, npts, cg, assembled):
    loop = _first_iteration(ib, _problem(ib, 400))  # more points than the assembled form takes
    assert (_first_iteration(ib, _problem(ib, npts), **cg) > loop) == assembled


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("npts,cg,assembled", [(201, {}, True), (201, dict(reltol=1e-2), False),
                                               (13, dict(reltol=1e-2), True)])
def test_a_large_grid_assembles_only_for_many_iterations(ib, npts, cg, assembled):
    size = dict(nx=640, ny=640, L=1)
    loop = _first_iteration(ib, _problem(ib, 400, **size))
    assert (_first_iteration(ib, _problem(ib, npts, **size), **cg) > loop) == assembled


@pytest.mark.parametrize("npts,cg", [(13, {}), (101, {}), (225, {}), (40, dict(reltol=0.2)),
                                     (40, dict(reltol=0.0, abstol=1e-10))])
def test_graph_and_eager_steps_launch_the_same_kernels(ib, npts, cg):
    prob = _problem(ib, npts)
    for g, e in zip(_steps(ib, prob, cg), _steps(ib, prob, cg, eager=True)):
        assert g[:2] == e[:2]
        assert np.array_equal(g[2], e[2])
