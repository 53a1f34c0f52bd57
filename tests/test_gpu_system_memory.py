"""fpsg_set_system under a memory cap: a system whose tables do not fit is refused and leaves none
behind, and one whose dense Coulomb rows do not fit runs from its index lists."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E

pytestmark = pytest.mark.gpu


def lattice(nx, ny):
    D = cf.distances(cf.grid_positions(nx, ny))
    n = nx * ny
    U = 2.0 / (1.0 + D)
    occ = (np.arange(n) % 2).astype(float)
    return cf.hopping(D, [(1.0, -1.0)]), U, U - np.diag(np.diag(U)), occ


def test_a_refused_system_is_not_run():
    T, U, V, occ = lattice(3, 2)
    eng = E.Engine()
    eng.set_system(T, U, V, None, E.COUL_DISTANCE)
    eng.sample(4, 1, occ, 1.0 - occ)
    ref = eng.run(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
    eng.set_memory_cap(1)
    big = lattice(8, 8)
    with pytest.raises(E.FpsgError) as ei:
        eng.set_system(*big[:3], None, E.COUL_DISTANCE)
    assert ei.value.code == E.ERR_OOM
    for call in (lambda: eng.run(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2), lambda: eng.sample(4, 1, occ, 1.0 - occ),
                 lambda: eng.set_pulse([1.0], 1.0, 0.0, 1.0, np.zeros(6))):
        with pytest.raises(E.FpsgError) as ei:
            call()
        assert ei.value.code == E.ERR_STATE
    eng.set_memory_cap(0)
    eng.set_system(T, U, V, None, E.COUL_DISTANCE)
    eng.sample(4, 1, occ, 1.0 - occ)
    r = eng.run(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
    assert np.array_equal(r.nund, ref.nund)
    eng.close()


def test_no_room_for_dense_rows():
    T, U, V, occ = lattice(12, 12)

    def run(cap):
        eng = E.Engine()
        try:
            eng.set_memory_cap(cap)
            eng.set_system(T, U, V, None, E.COUL_DISTANCE)
            eng.set_memory_cap(0)
            eng.sample(2, 1, occ, 1.0 - occ)
            eng.advance(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
            return eng.get_state()
        except E.FpsgError:
            return None
        finally:
            eng.close()

    # the smallest cap that the tables fit under; both precisions' U and V once more take 24 n^2 bytes
    lo, hi = 1, 1 << 24
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if run(mid) is not None else (mid, hi)
    assert run(0) is not None
    assert hi < (12 + 12 + 8 + 8 + 4 + 4 + 1) * 144 * 144 + (64 << 10)   # lists of U and V, orders, masks
    assert np.array_equal(run(hi), run(0))
