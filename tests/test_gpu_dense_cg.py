"""Moving-body CG with the step's B assembled (taken where the first residual is
well above the tolerance) against the CPU oracle's CG, at the edges of its layout:
fewer rows than blocks, rows that do not divide by the blocks, the largest size,
and the first size past it (B applied each iteration); a loose tolerance, where
the plain loop stays; maxiter.  Two CGs that stop at the same residual agree to the
tolerance times B's condition number (up to 1e5): 1e-6, the bar the other CG starts
are held to."""
import math

import numpy as np
import pytest

from fixtures import rel_l2

pytestmark = pytest.mark.gpu


def _problem(ib, npts, nx=480, ny=40, L=2):
    h = 0.0625
    fluid = ib.Fluid(grid=ib.fluid_grid(h=h, xlims=(0.0, nx * h), ylims=(0.0, ny * h), nlevel=L), Re=100.0,
                     freestream_vel=lambda t: (1.0, 0.0))
    # a plate along the channel, points a cell apart
    xb = np.column_stack([nx * h / 2 + h * (np.arange(npts) - (npts - 1) / 2), np.full(npts, ny * h / 2 + 0.3 * h)])

    def motion(t):
        return ib.RigidBodyTransform(pos=(0.02 * math.sin(t), 0.0), vel=(0.02 * math.cos(t), 0.0), angle=0.0,
                                     angular_vel=0.0)

    body = ib.MovingRigidBody(motion, ib.Panels(xb, np.full(npts, h)))
    return ib.Problem(fluid=fluid, bodies=ib.Bodies(b=body), scheme=ib.CNAB(dt=0.2 * h))


@pytest.mark.parametrize("npts,cg", [(1, {}), (3, {}), (13, {}), (101, {}), (224, {}), (225, {}),
                                     (40, dict(reltol=0.0, abstol=1e-10)), (40, dict(reltol=0.2)),
                                     (40, dict(maxiter=7))])
def test_forces_match_oracle(ib, orc, npts, cg):
    prob = _problem(ib, npts)
    sg, so = ib.State(prob), ib.State(prob)
    gpu, cpu = ib.GpuCnabSolver(sg, cg=cg), orc.OracleSolver(so, cg=cg)
    for _ in range(3):
        gpu.advance_()
        cpu.advance_()
        assert np.abs(sg.fb - so.fb).max() <= 1e-6 * np.abs(so.fb).max()
        if "maxiter" in cg:
            assert gpu.info().last_cg_iters == cg["maxiter"]
    gpu.getstate()
    assert rel_l2(sg.Gamma, so.Gamma) <= 1e-6
