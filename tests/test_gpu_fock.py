"""The cluster kernel of HF with the Fock term against the oracle, at the sizes where its
chunks, clusters and the place of Delta change."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,B,S,Tp", [
    ((1, 1), 1, 1, 3), ((2, 1), 3, 2, 3), ((3, 3), 12, 1, 4), ((8, 4), 1, 2, 3), ((11, 3), 2, 1, 3),
    ((8, 8), 1, 1, 3),
    ((9, 9), 1, 1, 2),       # Delta still in shared memory
    ((10, 9), 1, 1, 2),      # Delta in global memory
    ((17, 7), 1, 1, 2),      # the largest X
    ((12, 10), 1, 1, 2),     # beyond: the per-stage kernel
])
def test_fock_matches_oracle(dims, B, S, Tp):
    D = cf.distances(cf.grid_positions(*dims))
    n = D.shape[0]
    T = cf.hopping(D, [(1.0, -1.0)])
    U = 2.0 / (1.0 + D)
    V = U - np.diag(np.diag(U))
    rng = np.random.default_rng(n)
    ext = np.diag(rng.uniform(-1, 1, n))
    rho = np.zeros((B, 2, n, n), dtype=complex)
    for b in range(B):
        for s in range(2):
            _, R = np.linalg.eigh(T + np.diag(rng.uniform(-1, 1, n)))
            rho[b, s] = R[:, : (n + 1 - s) // 2] @ R[:, : (n + 1 - s) // 2].T
    rho = (rho + np.conj(np.swapaxes(rho, 2, 3))) / 2
    ref = orc.run(orc.System(T, U, V, ext, orc.COUL_DISTANCE, False), 1, 0.01, S, Tp, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, ext, E.COUL_DISTANCE)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_HF, E.PREC_FP64, 0.01, S, Tp)
    assert r.path_used == E.PATH_STREAM
    assert np.array_equal(eng.get_state(), ref["final"])
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
        assert np.array_equal(getattr(r, k), ref[k]), k
    # sums of n^2 terms of order 1 in another order
    assert np.max(np.abs(r.energies - ref["energies"])) < 4 * n * n * 2.0 ** -52 * np.abs(ref["energies"]).max()
    eng.set_initial_samples(rho)
    r32 = eng.run(E.METHOD_HF, E.PREC_FP32, 0.01, S, Tp)
    # FP32: S (Tp - 1) steps of 4 stages, |h Delta| <= 0.1, n-term sums of |X| <= 1, the state rounded every step
    bound = S * (Tp - 1) * (4 * 0.1 * 4 * np.sqrt(n) + 4) * 2.0 ** -24 * 4
    assert np.max(np.abs(r32.niiu - ref["niiu"])) < bound
    eng.close()


def small_system(n, seed=5):
    rng = np.random.default_rng(seed)
    D = np.abs(np.arange(n)[:, None] - np.arange(n)[None, :]).astype(float)
    T = -1.0 * (D == 1)
    U = 2.0 / (1.0 + D)
    return T, U, U - np.diag(np.diag(U)), np.diag(rng.uniform(-1, 1, n)), rng


def hf_states(T, B, rng):
    """Projectors on half of the eigenstates of the hopping in random potentials."""
    n = T.shape[0]
    rho = np.zeros((B, 2, n, n), dtype=complex)
    for b in range(B):
        for s in range(2):
            R = np.linalg.eigh(T + np.diag(rng.uniform(-1, 1, n)))[1][:, : (n + 1 - s) // 2]
            rho[b, s] = R @ R.T
    return (rho + np.conj(np.swapaxes(rho, 2, 3))) / 2


def test_fock_more_snapshots_than_a_grid_dimension():
    """65 538 snapshots, recorded by many launches and reduced in more than one go."""
    T, U, V, ext, rng = small_system(2)
    Tp, dt = 65538, 1e-3
    rho = hf_states(T, 1, rng)
    pulse = {"n_bins": 3, "amp": rng.normal(0, 0.5, 3), "bin_width": 30.0, "t0": 30.0, "td": 20.0, "proj": np.array([-0.5, 0.5])}
    ref = orc.run(orc.System(T, U, V, ext, orc.COUL_DISTANCE, False, pulse), 1, dt, 1, Tp, rho, nthreads=1)
    eng = E.Engine()
    eng.set_system(T, U, V, ext, E.COUL_DISTANCE)
    eng.set_pulse(pulse["amp"], pulse["bin_width"], pulse["t0"], pulse["td"], pulse["proj"])
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_HF, E.PREC_FP64, dt, 1, Tp)
    assert np.array_equal(eng.get_state(), ref["final"])
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
        assert np.array_equal(getattr(r, k), ref[k]), k
    # sums of n^2 terms of order 1 in another order
    assert np.max(np.abs(r.energies - ref["energies"])) < 4 * 4 * 2.0 ** -52 * np.abs(ref["energies"]).max()
    eng.close()


def test_fock_without_room_for_all_records():
    """Under a memory cap that holds one snapshot's records but not all of them, the run is the
    per-stage kernel's."""
    T, U, V, ext, rng = small_system(3)
    Tp = 4001
    rho = hf_states(T, 2, rng)
    ref = orc.run(orc.System(T, U, V, ext, orc.COUL_DISTANCE, False), 1, 0.005, 1, Tp, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, ext, E.COUL_DISTANCE)
    eng.set_initial_samples(rho)
    # the sums of all snapshots take 19 doubles each; with every record there are 19 + 2 (3 + 4) 2 more
    eng.set_memory_cap(8 * Tp * 19 + (1 << 18))
    r = eng.run(E.METHOD_HF, E.PREC_FP64, 0.005, 1, Tp)
    assert np.array_equal(eng.get_state(), ref["final"])
    # the mean of two trajectories, each value exact: the order of the sum does not matter
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
        assert np.array_equal(getattr(r, k), ref[k]), k
    eng.close()


@pytest.mark.parametrize("n,B", [(4, 14), (4, 15), (4, 300), (30, 28), (30, 29), (64, 63), (64, 75)])
def test_fock_ensembles(n, B):
    """Ensembles on either side of the choice between the cluster kernel, round after round, and
    the per-stage kernel: the same bits."""
    T, U, V, ext, rng = small_system(n)
    rho = hf_states(T, B, rng)
    ref = orc.run(orc.System(T, U, V, ext, orc.COUL_DISTANCE, False), 1, 0.01, 1, 3, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, ext, E.COUL_DISTANCE)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_HF, E.PREC_FP64, 0.01, 1, 3)
    assert np.array_equal(eng.get_state(), ref["final"])
    # means of B values of at most 1, summed in another order
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund"):
        assert np.max(np.abs(getattr(r, k) - ref[k])) < B * 2.0 ** -52, k
    eng.close()
