"""k_resident_quad_hp with one CTA per spin in FP64, and its empty rounds: lattices with more
neighbours on a side than k_resident takes, at the sizes where a configuration ends."""
import numpy as np
import pytest

from fermiphasespace_b200 import engine as E
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def ring(n, reach):
    """A ring where every site hops to its `reach` nearest on each side, with values of its own."""
    T = np.zeros((n, n))
    for i in range(n):
        for d in range(1, reach + 1):
            j = (i + d) % n
            if i != j:
                T[i, j] = T[j, i] = -1.0 / d
    return T


@pytest.mark.parametrize("n,reach,B", [(20, 6, 40), (32, 6, 40), (44, 5, 40), (45, 5, 40), (63, 5, 31), (64, 6, 31),
                                       (71, 5, 31), (77, 2, 31), (78, 2, 2), (79, 2, 31), (96, 2, 31)])
def test_one_cta_per_spin_matches_oracle(n, reach, B):
    T = ring(n, reach)
    rng = np.random.default_rng(n)
    U = np.diag(rng.uniform(1.0, 4.0, n))
    X = np.diag(rng.uniform(-1, 1, n))
    occ = (rng.random(n) < 0.5).astype(float)
    rho = orc.sample(n, B, 11, occ, 1.0 - occ)
    ref = orc.run(orc.System(T, U, None, X, orc.COUL_ONSITE, False), 0, 0.01, 1, 3, rho)
    eng = E.Engine()
    eng.set_system(T, U, None, X)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 3)
    assert r.path_used == E.PATH_RESIDENT
    assert np.array_equal(eng.get_state(), ref["final"])
    assert np.allclose(r.nund, ref["nund"], rtol=1e-13, atol=1e-13)
    assert np.allclose(r.energies, ref["energies"], rtol=1e-13, atol=1e-12)
    eng.set_initial_samples(rho)
    r = eng.run(E.METHOD_FTWA, E.PREC_FP32, 0.01, 1, 3)
    # three steps of four stages, h |Delta| <= 0.3, |rho| <= 2
    assert np.max(np.abs(eng.get_state() - ref["final"])) < 3 * (4 * 0.3 * 12 + 2) * 2.0 * 2.0 ** -24
    eng.close()
