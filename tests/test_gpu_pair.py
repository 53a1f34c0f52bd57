"""k_pair (offset-pattern lattices) against the oracle, at the sizes where its slot order,
masks and dispatch change: tiles of 32 rows and their remainders, odd and even n, one, two
and three offsets, sites without neighbours, one matrix per CTA and many, split and not."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def lattice(nx, ny, nz, t):
    return cf.hopping(cf.distances(cf.grid_positions(nx, ny, nz)), [(1.0, t)] if t else [])


def compare(T, coulomb, ext, B, S=2, Tp=4, dt=0.01, seed=3):
    n = T.shape[0]
    rng = np.random.default_rng(seed)
    if coulomb == E.COUL_DISTANCE:
        D = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :])
        U = 2.0 / (1.0 + D)
        V = U - np.diag(np.diag(U))
    else:
        U, V = np.diag(rng.uniform(1.0, 4.0, n)), None
    X = np.diag(rng.uniform(-1, 1, n)) if ext else None
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, V, X, coulomb, X is None), 0, dt, S, Tp, rho)
    out = {}
    for prec in (E.PREC_FP64, E.PREC_FP32):
        eng = E.Engine()
        eng.set_system(T, U, V, X, coulomb)
        eng.set_initial_samples(rho)
        r = eng.run(E.METHOD_FTWA, prec, dt, S, Tp)
        assert r.path_used == E.PATH_RESIDENT
        out[prec] = (r, eng.get_state())
        eng.close()
    return ref, out


@pytest.mark.parametrize("dims,t,coulomb,ext,B", [
    ((1, 1, 1), 0.0, E.COUL_ONSITE, False, 5),      # one site, no offsets
    ((2, 1, 1), -1.0, E.COUL_ONSITE, True, 40),
    ((7, 1, 1), -0.7, E.COUL_ONSITE, False, 300),   # a chain: one offset, several matrices per CTA
    ((31, 1, 1), -1.0, E.COUL_DISTANCE, True, 3),   # one partial tile
    ((8, 4, 1), -1.3, E.COUL_ONSITE, True, 3),      # exactly one tile of 32
    ((11, 3, 1), -1.0, E.COUL_ONSITE, False, 3),    # a tile and one row
    ((7, 9, 1), -1.0, E.COUL_DISTANCE, False, 3),   # 63: odd last column beside a full tile
    ((8, 8, 1), 0.9, E.COUL_ONSITE, True, 4),       # 64: two tiles
    ((4, 4, 4), -1.0, E.COUL_ONSITE, False, 3),     # three offsets
    ((3, 4, 5), -0.3, E.COUL_DISTANCE, True, 3),
    ((3, 9, 3), -1.0, E.COUL_ONSITE, True, 2),      # 81, three offsets
])
def test_pair_matches_oracle(dims, t, coulomb, ext, B):
    ref, out = compare(lattice(*dims, t), coulomb, ext, B)
    r, state = out[E.PREC_FP64]
    assert np.array_equal(state, ref["final"])
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund", "energies"):
        assert np.allclose(getattr(r, k), ref[k], rtol=1e-13, atol=1e-13), k
    # FP32: 8 steps of 4 stages round |rho| <= 2 (samples included) to 2^-24 a few times each, the
    # update itself compensated: h |Delta| <= 0.2 of a few ulp per stage
    r, state = out[E.PREC_FP32]
    assert np.max(np.abs(state - ref["final"])) < 32 * 0.2 * 8 * 2.0 * 2.0 ** -24 * 4


def test_pattern_needs_one_value():
    """Hopping of two values has no offset pattern: the column kernels run it, to the same bits."""
    T = cf.hopping(cf.distances(cf.grid_positions(5, 4)), [(1.0, -1.0)])
    T[0, 1] = T[1, 0] = -1.5
    ref, out = compare(T, E.COUL_ONSITE, True, 3)
    assert np.array_equal(out[E.PREC_FP64][1], ref["final"])


@pytest.mark.parametrize("dims,coulomb,ext,B,fp32", [
    ((10, 7, 1), E.COUL_ONSITE, True, 3, False),     # 70: past the single-CTA and 2-CTA FP64 kernels
    ((5, 5, 4), E.COUL_DISTANCE, False, 2, False),   # 100, three offsets
    ((10, 10, 1), E.COUL_ONSITE, True, 35, False),   # more trajectories than clusters
    ((11, 10, 1), E.COUL_ONSITE, True, 2, True),     # FP32 past k_pair
    ((11, 11, 1), E.COUL_DISTANCE, False, 2, True),
    ((12, 12, 1), E.COUL_ONSITE, False, 2, True),    # past k_pair_packed
    ((101, 1, 1), E.COUL_ONSITE, False, 2, False),   # FP64 past it
])
def test_packed_matches_oracle(dims, coulomb, ext, B, fp32):
    """k_pair_packed: FP64 to the bit, FP32 within the bound above; past it, the kernels of
    two CTAs per spin."""
    T = lattice(*dims, -1.0)
    n = T.shape[0]
    ref, out = compare(T, coulomb, ext, B, S=1, Tp=3) if not fp32 else compare_fp32(T, coulomb, ext, B)
    if not fp32:
        r, state = out[E.PREC_FP64]
        assert np.array_equal(state, ref["final"])
        for k in ("niiu", "n2iid", "nund", "energies"):
            assert np.allclose(getattr(r, k), ref[k], rtol=1e-13, atol=1e-13), k
    r, state = out[E.PREC_FP32]
    assert np.max(np.abs(state - ref["final"])) < 12 * 0.2 * 8 * 2.0 * 2.0 ** -24 * 4
    assert np.allclose(r.energies, ref["energies"], rtol=1e-6, atol=1e-6 * n)


def compare_fp32(T, coulomb, ext, B):
    """compare() without the FP64 run, which may be past the resident kernels."""
    n = T.shape[0]
    rng = np.random.default_rng(5)
    D = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :])
    U = 2.0 / (1.0 + D) if coulomb == E.COUL_DISTANCE else np.diag(rng.uniform(1.0, 4.0, n))
    V = U - np.diag(np.diag(U)) if coulomb == E.COUL_DISTANCE else None
    X = np.diag(rng.uniform(-1, 1, n)) if ext else None
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, V, X, coulomb, X is None), 0, 0.01, 1, 3, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, X, coulomb)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, E.PREC_FP32, 0.01, 1, 3)
    assert r.path_used == E.PATH_RESIDENT
    state = eng.get_state()
    eng.close()
    return ref, {E.PREC_FP32: (r, state)}


@pytest.mark.parametrize("prec,sizes", [(0, [(10, 10), (9, 10), (9, 9)]), (1, [(10, 10), (9, 10), (9, 9)]),
                                        (1, [(12, 12), (11, 11), (11, 10)]), (0, [(5, 4), (4, 4), (3, 3)])])
def test_batch_members_of_one_configuration(prec, sizes):
    # systems of falling size that take the same kernel: the shared memory that the last one
    # needs must not be the limit of the first one's launch
    eng = E.Engine()
    desc = []
    for k, (nx, ny) in enumerate(sizes):
        pos = cf.grid_positions(nx, ny, 1)
        n = nx * ny
        occ = (np.arange(n) % 2).astype(float)
        desc.append({"tM": cf.hopping(cf.distances(pos), [(1.0, -1.0)]), "U": 4.0 * np.eye(n), "V": None, "ext": None,
                     "coulomb": E.COUL_ONSITE, "n_traj": 9, "seed": 5 + k, "occ_up": occ, "occ_dn": 1.0 - occ})
    res, _ = eng.run_batch(desc, E.METHOD_FTWA, prec, 0.01, 1, 3, obs=1 | 2 | 4 | 16)
    for d, r in zip(desc, res):
        eng.set_system(d["tM"], d["U"], None, None, coulomb=E.COUL_ONSITE)
        eng.sample(9, d["seed"], d["occ_up"], d["occ_dn"])
        one = eng.run(E.METHOD_FTWA, prec, 0.01, 1, 3, obs=1 | 2 | 4 | 16)
        assert r.path_used == one.path_used == E.PATH_RESIDENT
        for key in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
            assert np.array_equal(getattr(r, key), getattr(one, key)), key
    eng.close()
