"""vort2flux across nested levels (the boundary values between levels enter in
the y solve, csrc/kernels.cuh RingOut) against the CPU oracle where its layouts
change: one, two and five levels, sizes that are not multiples of four,
non-square grids, odd chunk lengths; and bodies whose support reaches the
level-1 boundary, where E reads faces that come from the coarser level.
Tolerances: the operator-level and drop-in bars."""
import math

import numpy as np
import pytest

from fixtures import rel_l2

pytestmark = pytest.mark.gpu


def _problem(ib, nx, ny, L, body, moving=False, Re=100.0):
    h = 0.0625
    fluid = ib.Fluid(grid=ib.fluid_grid(h=h, xlims=(0.0, nx * h), ylims=(0.0, ny * h), nlevel=L), Re=Re,
                     freestream_vel=lambda t: (1.0, 0.0))
    xb = np.asarray(body(nx * h, ny * h, h))
    panels = ib.Panels(xb, np.full(len(xb), h))
    if moving:
        def motion(t):
            return ib.RigidBodyTransform(pos=(0.02 * math.sin(t), 0.0), vel=(0.02 * math.cos(t), 0.0), angle=0.0,
                                         angular_vel=0.0)

        b = ib.MovingRigidBody(motion, panels)
    else:
        b = ib.StaticBody(panels)
    return ib.Problem(fluid=fluid, bodies=ib.Bodies(b=b), scheme=ib.CNAB(dt=0.01))


def _middle(w, v, h):
    return [(w / 2 + h * k, v / 2 + 0.3 * h * k) for k in range(-6, 7)]


def _edges(w, v, h):
    # panels 3.1 cells from the left, bottom and right edges and 3.2 from the top
    ks = np.arange(0, 12)
    return ([(3.1 * h, v / 2 + 1.3 * h * k) for k in ks[:4]] + [(w / 3 + 1.3 * h * k, 3.1 * h) for k in ks[:4]]
            + [(w - 4.2 * h, v / 3 + 1.3 * h * k) for k in ks[:4]] + [(w / 2 + 1.3 * h * k, v - 4.2 * h) for k in ks[:4]])


@pytest.mark.parametrize("nx,ny,L", [(64, 64, 1), (64, 40, 2), (54, 50, 3), (150, 90, 3), (90, 150, 4), (200, 72, 2),
                                     (256, 64, 3), (96, 128, 5), (72, 250, 2), (30, 20, 3)])
def test_vort2flux_matches_oracle(ib, orc, nx, ny, L):
    prob = _problem(ib, nx, ny, L, _middle)
    g, o = ib.create_solver(ib.State(prob)), orc.OracleSolver(ib.State(prob))
    G = np.random.default_rng(nx + ny).standard_normal((prob.grid.inds.nGamma, L))
    ga, pa, qa = g.diag_vort2flux(G)
    gb, pb, qb = o.vort2flux(G)
    assert rel_l2(ga, gb) < 1e-15
    assert rel_l2(pa, pb) < 1e-13
    assert rel_l2(qa, qb) < 1e-12
    z = np.random.default_rng(L).standard_normal(2 * prob.bodies.npanel)
    assert rel_l2(g.diag_apply_B(z), o.apply_B(z)) < 1e-12


@pytest.mark.parametrize("body", [_middle, _edges])
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("nx,ny,L", [(64, 64, 1), (64, 80, 2), (50, 54, 3), (128, 64, 4)])
def test_steps_match_oracle(ib, orc, nx, ny, L, moving, body):
    prob = _problem(ib, nx, ny, L, body, moving)
    sg, so = ib.configs.seed_vorticity(ib.State(prob)), ib.configs.seed_vorticity(ib.State(prob))
    gpu, cpu = ib.create_solver(sg), orc.OracleSolver(so)
    for _ in range(3):
        gpu.advance_()
        cpu.advance_(pull=False)
    cpu.pull()
    gpu.getstate()
    assert rel_l2(sg.Gamma, so.Gamma) <= 1e-10
    assert rel_l2(sg.q, so.q) <= 1e-10
    assert rel_l2(sg.psi, so.psi) <= 1e-10
    assert np.abs(sg.fb - so.fb).max() <= 1e-9 * np.abs(so.fb).max()


@pytest.mark.parametrize("prec,bar", [("mixed", 1e-4), ("fp32", 1e-4)])
@pytest.mark.parametrize("L", [1, 2, 3])
def test_reduced_precision_follows_fp64(ib, prec, bar, L):
    prob = _problem(ib, 96, 64, L, _edges)
    s64, sx = ib.configs.seed_vorticity(ib.State(prob)), ib.configs.seed_vorticity(ib.State(prob))
    a, b = ib.create_solver(s64), ib.create_solver(sx, precision=prec)
    for _ in range(3):
        a.advance_()
        b.advance_()
    a.getstate()
    b.getstate()
    assert rel_l2(sx.Gamma, s64.Gamma) <= bar
    assert rel_l2(sx.q, s64.q) <= bar
