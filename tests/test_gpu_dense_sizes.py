"""The dense path over the number of matrices: the diagonals formed by the stage kernel or by a
launch of their own, the snapshot records at sizes where their blocks and warps change, and what
the path needs under a memory cap."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NP = 256


def system(n, coulomb, ext=True):
    rng = np.random.default_rng(n)
    D = np.abs(rng.permutation(n)[:, None] - np.arange(n)[None, :]).astype(float)
    D = D + D.T
    T = -np.exp(-0.5 * D) * (1.0 - np.eye(n))
    U = 1.0 / (1.0 + D) + np.eye(n) if coulomb == E.COUL_DISTANCE else np.diag(rng.uniform(1.0, 4.0, n))
    V = U - np.diag(np.diag(U)) if coulomb == E.COUL_DISTANCE else None
    X = np.diag(rng.uniform(-1, 1, n)) if ext else None
    occ = (rng.random(n) < 0.5).astype(float)
    return T, U, V, X, occ


@pytest.mark.parametrize("prec", [E.PREC_SPLIT_BF16X3, E.PREC_SPLIT_TF32X3])
@pytest.mark.parametrize("coulomb", [E.COUL_ONSITE, E.COUL_DISTANCE])
def test_a_trajectory_does_not_depend_on_the_others(coulomb, prec):
    """One matrix per CTA, several, and more than five (own launch for dense rows): the same sums in
    the same order, so the same bits."""
    T, U, V, X, occ = system(30, coulomb)
    eng = E.Engine()
    eng.set_system(T, U, V, X, coulomb)
    states = []
    for B in (3, 75, 400):
        eng.sample(B, 5, occ, 1.0 - occ)
        eng.advance(E.METHOD_FTWA, prec, 0.005, 1, 3)
        states.append(eng.get_state()[:3])
    eng.close()
    assert np.array_equal(states[0], states[1]) and np.array_equal(states[0], states[2])


@pytest.mark.parametrize("n", [1, 3, 31, 33, 100, 255, 256])
@pytest.mark.parametrize("coulomb,ext", [(E.COUL_ONSITE, True), (E.COUL_DISTANCE, False), (E.COUL_DISTANCE, True)])
def test_records(n, coulomb, ext):
    """The first snapshot's records against the oracle's.  The state is the sample rounded to FP32:
    each term of an energy is off by a few ulp of products of |rho| <= 2 and a weight in FP32."""
    T, U, V, X, occ = system(n, coulomb, ext)
    rho = orc.sample(n, 3, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, V, X, coulomb, X is None), 0, 0.005, 1, 1, rho)
    eng = E.Engine()
    eng.set_system(T, U, V, X, coulomb)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, E.PREC_SPLIT_BF16X3, 0.005, 1, 1)
    eng.close()
    eps = 2.0 ** -24
    for k in ("niiu", "niid"):
        assert np.max(np.abs(getattr(r, k) - ref[k])) <= 2 * eps, k
    for k in ("n2iiu", "n2iid", "nund"):
        assert np.max(np.abs(getattr(r, k) - ref[k])) <= 16 * eps, k
    weight = np.abs(T).sum() + (0 if X is None else np.abs(X).sum()) + 4 * np.abs(U).sum()
    assert np.max(np.abs(r.energies - ref["energies"])) <= 2 * 2.0 * 4 * eps * weight


def smallest_cap(T, U, V, X, coulomb, B, occ):
    """The smallest memory cap (to 4 KB) that holds the system and its samples."""
    def fits(cap):
        eng = E.Engine()
        try:
            eng.set_memory_cap(cap)
            eng.set_system(T, U, V, X, coulomb)
            eng.sample(B, 5, occ, 1.0 - occ)
            return True
        except E.FpsgError:
            return False
        finally:
            eng.close()
    lo, hi = 1, 1 << 26
    while hi - lo > 4096:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(mid) else (mid, hi)
    return hi


@pytest.mark.parametrize("B,coulomb,record", [(40, E.COUL_ONSITE, False), (380, E.COUL_DISTANCE, False),
                                              (1, E.COUL_ONSITE, True)])
def test_memory(B, coulomb, record):
    """Four copies of the state in planes, tM, its tiles, dense U and V, the snapshot buffers and a
    packed copy for the records: nothing else."""
    n = 16
    T, U, V, X, occ = system(n, coulomb)
    ne, M, W, Tp = n * (n + 1) // 2, 2 * B, 5 * n + 4, 3
    need = 4 * M * 2 * NP * NP * 4 + NP * NP * 4 + 2 * NP * NP * 4 + 4
    if coulomb == E.COUL_DISTANCE:
        need += 2 * NP * NP * 4
    if record:
        need += 8 * (Tp * W + M * n + M * 4 + W) + 8 * M * ne
    eng = E.Engine()
    eng.set_memory_cap(smallest_cap(T, U, V, X, coulomb, B, occ) + need + 4096)
    eng.set_system(T, U, V, X, coulomb)
    eng.sample(B, 5, occ, 1.0 - occ)
    ref = E.Engine()
    ref.set_system(T, U, V, X, coulomb)
    ref.sample(B, 5, occ, 1.0 - occ)
    if record:
        a = eng.run(E.METHOD_FTWA, E.PREC_SPLIT_BF16X3, 0.005, 1, Tp)
        b = ref.run(E.METHOD_FTWA, E.PREC_SPLIT_BF16X3, 0.005, 1, Tp)
        assert np.array_equal(a.niiu, b.niiu) and np.array_equal(a.nund, b.nund)
        # energies from a packed copy add up in another order, and, after a step, from one triangle of
        # planes that are Hermitian to rounding only: the first snapshot's are comparable
        assert np.allclose(a.energies[:, 0], b.energies[:, 0], rtol=1e-12, atol=1e-12)
    else:
        for e in (eng, ref):
            e.advance(E.METHOD_FTWA, E.PREC_SPLIT_BF16X3, 0.005, 1, 2)
    assert np.array_equal(eng.get_state(), ref.get_state())
    eng.close()
    ref.close()
