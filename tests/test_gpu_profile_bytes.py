"""The profile's algorithmic bytes: what the kernels of a step read and write, in the
engine's element size, and inside the body's window where only that is covered."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _profiled_step(ib, prob, prec, q=None):
    st = ib.configs.seed_vorticity(ib.State(prob))
    if q is not None:
        st.q[...] = q
    s = ib.create_solver(st, precision=prec)
    s.profile(True)
    s.advance_()
    return {k: s.profile_read(k) for k in ("nonlinear", "curl", "xpass")}


@pytest.mark.parametrize("n,L", [(64, 1), (150, 3)])
@pytest.mark.parametrize("prec,size", [("fp64", 8), ("fp32", 4)])
def test_nonlinear_term(ib, n, L, prec, size):
    prob = ib.configs.small_cylinder(n, L)
    ng, nq = (n - 1) ** 2, 2 * n * (n + 1)
    # psi, Gamma, the last term in; the term and the right-hand side out
    assert _profiled_step(ib, prob, prec)["nonlinear"][2] == size * 5 * ng * L
    q = 1e-3 * np.random.default_rng(3).standard_normal(ib.State(prob).q.shape)  # a q of the caller's: read itself
    assert _profiled_step(ib, prob, prec, q)["nonlinear"][2] == size * (nq + 4 * ng) * L


@pytest.mark.parametrize("n,L", [(64, 1), (150, 3)])
def test_windowed_launches(ib, n, L):
    prob = ib.configs.small_cylinder(n, L)
    h, xb = prob.grid.gridstep(1), np.concatenate([b.panels.xb for _, b, _ in prob.bodies.preset])
    # the body's box: three faces around the panels' cells (rounded as the library does)
    ix, iy = (np.rint((xb[:, k] - x0) / h + 0.75) for k, x0 in ((0, -1.0), (1, -2.0)))
    w, v = int(np.ptp(ix)) + 7, int(np.ptp(iy)) + 7
    got = _profiled_step(ib, prob, "fp64")
    assert got["curl"][2] == 8 * (2 * w * v + (w + 1) * (v + 1))
    ng = (n - 1) ** 2
    rows = (v + 1) * (n - 1)  # the curl of faces j0 .. j1 reads psi's rows j0 - 1 .. j1
    # trial solve; vort2flux to level 1's window, with the lines between the levels;
    # projection, whose last pass reads its target; vort2flux of every level
    lines = (L - 1) * ng / 2
    want = 4 * ng * L + (2 * ng * L + lines + 2 * rows) + (rows + ng + 3 * ng) + (4 * ng * L + lines)
    assert got["xpass"][2] == 8 * want
