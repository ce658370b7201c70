"""Reading output fields: the first read of a handle, alone or in an ensemble, before
and after its first step, allocates nothing, and gives what the state holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _all_fields(s, levels):
    return [f(lev) for f in (s.vorticity, s.x_velocity, s.y_velocity) for lev in range(1, levels + 1)]


@pytest.mark.parametrize("prec", ["fp64", "fp32", "mixed"])
@pytest.mark.parametrize("n,L", [(24, 1), (150, 3)])
@pytest.mark.parametrize("steps", [0, 2])
def test_first_read(ib, prec, n, L, steps):
    def make(k):
        st = ib.configs.seed_vorticity(ib.State(ib.configs.small_cylinder(n, L, npts=16)), seed=k)
        st.q[...] = 1e-3 * np.random.default_rng(k).standard_normal(st.q.shape)
        return ib.create_solver(st, precision=prec)

    alone, grouped = [make(k) for k in range(3)], [make(k) for k in range(3)]
    ens = ib.Ensemble(grouped)
    if steps:
        ens.advance_(steps)
        for s in alone:
            s.advance_many(steps)
    for a, g in zip(alone, grouped):
        held = a.info().device_bytes, g.info().device_bytes
        fa, fg = _all_fields(a, L), _all_fields(g, L)
        assert (a.info().device_bytes, g.info().device_bytes) == held
        for x, y in zip(fa, fg):
            assert np.array_equal(x, y)
        s = a.sync()
        h = a.state.prob.grid.gridstep(1)
        # the state's level 1 through the same division in 64 bits (mixed: level 1 is FP64)
        assert np.array_equal(fa[0].ravel(order="F"), s.Gamma[:, 0] / (h * h))
        # reads between steps leave no trace in them
        a.advance_many(1)
    ens.advance_(1)
    for a, g in zip(alone, grouped):
        assert np.array_equal(a.sync().Gamma, g.sync().Gamma)
