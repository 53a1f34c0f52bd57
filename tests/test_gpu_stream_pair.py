"""k_stream_pair (matrices beyond shared memory with an offset pattern) against the oracle, at
the ends of its tiles and offsets."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,coulomb,whole", [
    ((169, 1, 1), E.COUL_ONSITE, False),      # one offset, odd
    ((16, 16, 1), E.COUL_ONSITE, True),
    ((13, 15, 1), E.COUL_DISTANCE, False),
    ((6, 6, 5), E.COUL_ONSITE, False),        # three offsets
    ((11, 13, 1), E.COUL_ONSITE, False),      # a matrix that fits shared memory too
])
def test_stream_pair_matches_oracle(dims, coulomb, whole):
    T = cf.hopping(cf.distances(cf.grid_positions(*dims)), [(1.0, -1.0)])
    n = T.shape[0]
    rng = np.random.default_rng(n)
    D = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :])
    U = 2.0 / (1.0 + D) if coulomb == E.COUL_DISTANCE else np.diag(rng.uniform(1.0, 4.0, n))
    V = U - np.diag(np.diag(U)) if coulomb == E.COUL_DISTANCE else None
    X = np.diag(rng.uniform(-1, 1, n))
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, 2, 11, occ, 1.0 - occ)
    obs = E.OBS_DEFAULT | (E.OBS_WHOLE if whole else 0)
    ref = orc.run(orc.System(T, U, V, X, coulomb, False), 0, 0.01, 1, 2, rho, obs)
    for prec in (E.PREC_FP64, E.PREC_FP32):
        eng = E.Engine()
        eng.set_system(T, U, V, X, coulomb)
        eng.set_initial_samples(rho)
        r = eng.run(E.METHOD_FTWA, prec, 0.01, 1, 2, obs, path=E.PATH_STREAM)
        state = eng.get_state()
        eng.close()
        if prec == E.PREC_FP64:
            assert np.array_equal(state, ref["final"])
            for k in ("niiu", "niid", "n2iiu", "nund"):
                assert np.array_equal(getattr(r, k), ref[k]), k
            assert np.allclose(r.energies, ref["energies"], rtol=1e-13, atol=1e-12)
            if whole:
                assert np.allclose(r.whole_u, ref["whole_u"], rtol=0, atol=1e-14)
        else:
            # two steps of four stages, h |Delta| <= 0.3, |rho| <= 2, plain FP32 update
            assert np.max(np.abs(state - ref["final"])) < 2 * (4 * 0.3 * 8 + 2) * 2.0 * 2.0 ** -24


@pytest.mark.parametrize("prec", [E.PREC_FP64, E.PREC_FP32])
@pytest.mark.parametrize("coulomb", [E.COUL_ONSITE, E.COUL_DISTANCE])
def test_batch_members_equal_runs_alone(prec, coulomb):
    """Batch systems past the resident kernels run in one launch of their own; each gives the
    bits of the same system run alone, which takes k_stream_pair."""
    desc = []
    for k, dims in enumerate([(13, 13, 1), (16, 16, 1), (6, 6, 5)]):
        T = cf.hopping(cf.distances(cf.grid_positions(*dims)), [(1.0, -1.0)])
        n = T.shape[0]
        rng = np.random.default_rng(n)
        D = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :])
        U = 2.0 / (1.0 + D) if coulomb == E.COUL_DISTANCE else np.diag(rng.uniform(1.0, 4.0, n))
        occ = (rng.random(n) < 0.5).astype(float)
        desc.append({"tM": T, "U": U, "V": U - np.diag(np.diag(U)) if coulomb == E.COUL_DISTANCE else None,
                     "ext": np.diag(rng.uniform(-1, 1, n)), "coulomb": coulomb, "n_traj": 3, "seed": 5 + k,
                     "occ_up": occ, "occ_dn": 1.0 - occ})
    eng = E.Engine()
    res, _ = eng.run_batch(desc, E.METHOD_FTWA, prec, 0.01, 2, 4)
    for d, r in zip(desc, res):
        eng.set_system(d["tM"], d["U"], d["V"], d["ext"], coulomb=coulomb)
        eng.sample(3, d["seed"], d["occ_up"], d["occ_dn"])
        one = eng.run(E.METHOD_FTWA, prec, 0.01, 2, 4)
        assert r.path_used == one.path_used == E.PATH_STREAM
        for key in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
            assert np.array_equal(getattr(r, key), getattr(one, key)), key
    eng.close()
