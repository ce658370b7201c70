"""The flux between steps: the steps read q as psi's curl and keep none, so a
caller's q that is not psi's curl must still be what the next step reads, in every
engine and in an ensemble, and q read back must be the last step's."""
import numpy as np
import pytest

from fixtures import rel_l2

pytestmark = pytest.mark.gpu


def _state(ib, prob, scale):
    st = ib.configs.seed_vorticity(ib.State(prob))
    st.q[...] = scale * np.random.default_rng(5).standard_normal(st.q.shape)
    return st


@pytest.mark.parametrize("n,L", [(40, 1), (64, 3), (150, 2)])
def test_a_set_flux_is_read_once(ib, orc, n, L):
    prob = ib.configs.small_cylinder(n, L)
    h = prob.grid.gridstep()
    sg, so = _state(ib, prob, 0.1 * h), _state(ib, prob, 0.1 * h)
    gpu, cpu = ib.create_solver(sg), orc.OracleSolver(so)
    for _ in range(3):
        gpu.advance_()
        cpu.advance_(pull=False)
    cpu.pull()
    gpu.getstate()
    assert rel_l2(sg.Gamma, so.Gamma) <= 1e-10
    assert rel_l2(sg.q, so.q) <= 1e-10


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
def test_set_and_restored_states_agree(ib, prec):
    """A state read back and set again (q is psi's curl then) steps on as the run
    it came from; one with another q steps on differently, alone as in an ensemble."""
    prob = ib.configs.small_cylinder(96, 3)
    a = ib.create_solver(ib.configs.seed_vorticity(ib.State(prob)), precision=prec)
    a.advance_many(3)
    mid = a.sync()
    back = ib.State(prob)
    for k in ("q", "q0", "Gamma", "psi", "Fbt"):
        getattr(back, k)[...] = getattr(mid, k)
    for k in range(2):
        back.nonlin[k][...] = mid.nonlin[k]
    back.index = mid.index
    b = ib.create_solver(back, precision=prec)
    a.advance_many(2)
    b.advance_many(2)
    sa, sb = a.sync(), b.sync()
    assert np.array_equal(sa.Gamma, sb.Gamma) and np.array_equal(sa.q, sb.q)
    other = [_state(ib, prob, 1e-3) for _ in range(2)] + [ib.configs.seed_vorticity(ib.State(prob))]
    sols = [ib.create_solver(s, precision=prec) for s in other]
    alone = ib.create_solver(_state(ib, prob, 1e-3), precision=prec)
    ens = ib.Ensemble(sols[1:])
    ens.advance_(2)
    alone.advance_many(2)
    assert np.array_equal(sols[1].sync().Gamma, alone.sync().Gamma)
    assert not np.array_equal(sols[1].state.Gamma, sols[2].sync().Gamma)
