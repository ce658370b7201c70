"""A grouped case stepped on its own, an odd or an even number of times, between the
ensemble's steps: every case's state stays that of the same steps without an ensemble."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("own", [1, 2, 3])
def test_steps_alone_and_together(ib, prec, own):
    def make(k):
        return ib.create_solver(ib.configs.seed_vorticity(ib.State(ib.configs.small_cylinder(64, 3)), seed=k),
                                precision=prec)

    alone, grouped = [make(k) for k in range(3)], [make(k) for k in range(3)]
    ens = ib.Ensemble(grouped)
    for n in (1, 2, 1):
        ens.advance_(n)
        grouped[1].advance_many(own)
        for k, s in enumerate(alone):
            s.advance_many(n + own * (k == 1))
        for a, g in zip(alone, grouped):
            x, y = a.sync(), g.sync()
            assert x.index == y.index
            for name in ("Gamma", "psi", "q", "Fbt"):
                assert np.array_equal(getattr(x, name), getattr(y, name)), name
            assert np.array_equal(x.nonlin[1], y.nonlin[1])
