"""Device memory after fpsg_run_batch: what the systems of a batch held must not stand in the way
of later calls, under a memory cap or without one."""
import numpy as np
import pytest

from fermiphasespace_b200 import configs as cf
from fermiphasespace_b200 import engine as E

pytestmark = pytest.mark.gpu


def system(nx, ny, traj, seed=5):
    n = nx * ny
    occ = (np.arange(n) % 2).astype(float)
    return {"tM": cf.hopping(cf.distances(cf.grid_positions(nx, ny, 1)), [(1.0, -1.0)]), "U": 4.0 * np.eye(n), "V": None,
            "ext": None, "coulomb": E.COUL_ONSITE, "n_traj": traj, "seed": seed, "occ_up": occ, "occ_dn": 1.0 - occ}


def state_bytes(d):
    n = d["tM"].shape[0]
    return d["n_traj"] * 2 * (n * (n + 1) // 2) * 16


@pytest.mark.parametrize("traj,after", [(1500, 1600), (1500, 100)])
def test_sample_after_a_batch_under_a_cap(traj, after):
    """Two systems whose states take 3/4 of the cap each (each is checked by itself), then another
    system whose state takes most of it, or little."""
    d = [system(6, 6, traj, seed=k) for k in range(2)]
    one = dict(system(6, 6, after), n_traj=after)
    eng = E.Engine()
    eng.set_memory_cap(state_bytes(d[0]) * 4 // 3)
    eng.run_batch(d, E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
    ref = E.Engine()
    out = []
    for e in (eng, ref):
        e.set_system(one["tM"], one["U"], None, None, coulomb=E.COUL_ONSITE)
        e.sample(after, 9, one["occ_up"], one["occ_dn"])
        out.append((e.run(E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2), e.get_state()))
        e.close()
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0].nund, out[1][0].nund)


def test_pool_after_batches_of_falling_size():
    """Only the last batches' states stay allocated, at most twice the last one's."""
    import torch
    eng = E.Engine()
    eng.run_batch([system(6, 6, 200)], E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
    free0 = torch.cuda.mem_get_info()[0]
    for traj in (40000, 15000, 6000, 2000):        # 852, 320, 128 and 43 MB of states
        eng.run_batch([system(6, 6, traj)], E.METHOD_FTWA, E.PREC_FP64, 0.01, 1, 2)
    held = free0 - torch.cuda.mem_get_info()[0]
    # beside them tables and record scratch, and the 2 MB granularity of the driver's blocks
    assert held < 2 * 2000 * 2 * 666 * 16 + (64 << 20), held
    eng.close()
