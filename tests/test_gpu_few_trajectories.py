"""Ensembles on either side of the choice between four SMs and two for a trajectory (33 4-CTA
clusters run at a time), against the oracle."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,dims", [(E.PREC_FP64, (10, 8)), (E.PREC_FP64, (10, 10)), (E.PREC_FP32, (12, 12))])
@pytest.mark.parametrize("B", [1, 30, 33, 34, 38])
def test_few_trajectories(prec, dims, B):
    T = cf.hopping(cf.distances(cf.grid_positions(*dims)), [(1.0, -1.0)])
    n = T.shape[0]
    rng = np.random.default_rng(n)
    U, X = np.diag(rng.uniform(1.0, 4.0, n)), np.diag(rng.uniform(-1, 1, n))
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, None, X, orc.COUL_ONSITE, False), 0, 0.01, 1, 2, rho)
    eng = E.Engine()
    eng.set_system(T, U, None, X, E.COUL_ONSITE)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, prec, 0.01, 1, 2)
    assert r.path_used == E.PATH_RESIDENT
    state = eng.get_state()
    eng.close()
    if prec == E.PREC_FP64:
        assert np.array_equal(state, ref["final"])
    else:
        # two steps of four stages, h |Delta| <= 0.1, a few ulp of |rho| <= 2 per stage, compensated update
        assert np.max(np.abs(state - ref["final"])) < 8 * 0.1 * 8 * 2.0 * 2.0 ** -24
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
        tol = B * 4 * 2.0 ** -52 if prec == E.PREC_FP64 else 8 * 2.0 * 2.0 ** -24
        assert np.max(np.abs(getattr(r, k) - ref[k])) < tol, k
