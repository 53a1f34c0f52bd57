"""Lattices of at most ten sites on either side of the choice between the column kernel and the
pair kernel, against the oracle."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (3, 2, 1), (2, 2, 2), (5, 2, 1)])
@pytest.mark.parametrize("B", [1, 149, 301, 1500])
def test_small_systems(dims, B):
    T = cf.hopping(cf.distances(cf.grid_positions(*dims)), [(1.0, -1.0)] if dims != (1, 1, 1) else [])
    n = T.shape[0]
    rng = np.random.default_rng(n)
    U, X = np.diag(rng.uniform(1.0, 4.0, n)), np.diag(rng.uniform(-1, 1, n))
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    obs = E.OBS_DEFAULT | E.OBS_WHOLE
    ref = orc.run(orc.System(T, U, None, X, orc.COUL_ONSITE, False), 0, 0.01, 2, 3, rho, obs)
    for prec in (E.PREC_FP64, E.PREC_FP32):
        eng = E.Engine()
        eng.set_system(T, U, None, X, E.COUL_ONSITE)
        eng.set_initial_samples(rho)
        r = eng.run(E.METHOD_FTWA, prec, 0.01, 2, 3, obs)
        state = eng.get_state()
        eng.close()
        if prec == E.PREC_FP64:
            assert np.array_equal(state, ref["final"])
            tol = B * 8 * 2.0 ** -52          # sums of B values of at most 8 in another order
        else:
            # six steps of four stages, h |Delta| <= 0.1, a few ulp of |rho| <= 2 per stage, compensated update
            tol = 24 * 0.1 * 8 * 2.0 * 2.0 ** -24 + 2.0 * 2.0 ** -24
            assert np.max(np.abs(state - ref["final"])) < tol
        for k in ("niiu", "niid", "n2iiu", "n2iid", "nund", "whole_u", "whole_d"):
            assert np.max(np.abs(getattr(r, k) - ref[k])) < 4 * tol, k
