"""k_pair_packed in FP64 with more trajectories than 4-CTA clusters run at a time (fewer take
k_resident_quad_hp), against the oracle: three, four and five slots a thread, one, two and three
offsets, dense Coulomb rows, a pulse, whole matrices, Hartree-Fock.  And FP32 past its shared
memory."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def system(dims, coulomb):
    pos = cf.grid_positions(*dims)
    D = cf.distances(pos)
    n = D.shape[0]
    rng = np.random.default_rng(n)
    T = cf.hopping(D, [(1.0, -1.0)])
    U = 2.0 / (1.0 + D) if coulomb == E.COUL_DISTANCE else np.diag(rng.uniform(1.0, 4.0, n))
    V = U - np.diag(np.diag(U)) if coulomb == E.COUL_DISTANCE else None
    X = np.diag(rng.uniform(-1, 1, n))
    pulse = {"n_bins": 3, "amp": rng.normal(0, 0.5, 3), "bin_width": 0.02, "t0": 0.02, "td": 0.02,
             "proj": pos[:, 0] - pos[:, 0].mean()}
    return T, U, V, X, pulse, rng


@pytest.mark.parametrize("dims,coulomb,pulsed,whole,method", [
    ((67, 1, 1), E.COUL_ONSITE, False, False, E.METHOD_FTWA),   # one offset, three slots
    ((9, 8, 1), E.COUL_ONSITE, True, True, E.METHOD_FTWA),
    ((8, 9, 1), E.COUL_DISTANCE, True, False, E.METHOD_FTWA),
    ((4, 4, 5), E.COUL_DISTANCE, False, True, E.METHOD_FTWA),   # three offsets, four slots
    ((11, 8, 1), E.COUL_ONSITE, True, False, E.METHOD_HF),
    ((9, 11, 1), E.COUL_ONSITE, False, True, E.METHOD_HF),      # odd, five slots
    ((5, 5, 4), E.COUL_DISTANCE, True, False, E.METHOD_FTWA),
])
def test_packed_fp64(dims, coulomb, pulsed, whole, method):
    T, U, V, X, pulse, rng = system(dims, coulomb)
    n, B = T.shape[0], 38
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    obs = E.OBS_DEFAULT | (E.OBS_WHOLE if whole else 0)
    ref = orc.run(orc.System(T, U, V, X, coulomb, False, pulse if pulsed else None), method, 0.01, 2, 3, rho, obs)
    eng = E.Engine()
    eng.set_system(T, U, V, X, coulomb)
    if pulsed:
        eng.set_pulse(pulse["amp"], pulse["bin_width"], pulse["t0"], pulse["td"], pulse["proj"])
    eng.set_initial_samples(rho)
    r = eng.run(method, E.PREC_FP64, 0.01, 2, 3, obs)
    assert r.path_used == E.PATH_RESIDENT
    assert np.array_equal(eng.get_state(), ref["final"])
    # sums of B values of at most 8 (and n^2 of them in the energies) in another order
    for k in ("niiu", "niid", "n2iiu", "n2iid", "nund") + (("whole_u", "whole_d") if whole else ()):
        assert np.max(np.abs(getattr(r, k) - ref[k])) < B * 8 * 2.0 ** -52, k
    assert np.max(np.abs(r.energies - ref["energies"])) < B * n * n * 8 * 2.0 ** -52
    eng.set_initial_samples(rho)
    t = 0.0
    steps = 4 if method == E.METHOD_HF else 6
    for m in (1, steps - 1):                      # in pieces: the same bits
        eng.advance(method, E.PREC_FP64, 0.01, 2, m, t_start=t)
        t += m * 0.005
    if not pulsed:                                # (a pulse's times add up in another order)
        assert np.array_equal(eng.get_state(), ref["final"])
    eng.close()


@pytest.mark.parametrize("dims,path", [((16, 9, 1), E.PATH_RESIDENT), ((150, 1, 1), E.PATH_STREAM)])
def test_fp32_past_packed(dims, path):
    """An offset too large for the triangle with its sub-diagonals in shared memory: the kernel of
    two CTAs per spin; too many slots: the stream path."""
    T, U, V, X, _, rng = system(dims, E.COUL_ONSITE)
    n = T.shape[0]
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, 40, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, V, X, orc.COUL_ONSITE, False), 0, 0.01, 1, 3, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, X, E.COUL_ONSITE)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, E.PREC_FP32, 0.01, 1, 3)
    assert r.path_used == path
    # three steps of four stages, h |Delta| <= 0.2, |rho| <= 2, eight roundings a stage; the plain
    # update of the stream path adds one of |rho| per step
    bound = 12 * 0.2 * 8 * 2.0 * 2.0 ** -24 + 3 * 2.0 * 2.0 ** -24
    assert np.max(np.abs(eng.get_state() - ref["final"])) < bound
    eng.close()
