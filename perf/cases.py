"""The engine's work as its users have it done, for timing and comparison.

A pass is what a program does for one simulation through `fermiphasespace_b200.engine`: draw or
hand over the initial samples, integrate, read the observables (or the gradient).  The system
(hopping, Coulomb and potential matrices, pulse) is set once, in prepare().  Observables of FP64
trajectories are returned as FP64; those of FP32 and split-precision trajectories as FP32, the
type the trajectories have.

exact() restates the same simulation with dense FP64 torch operations: the engine's documented
sample stream (Philox4x32-10, Box-Muller), the mean-field equations and the 3/8-rule RK4 step.
"""
import math

import numpy as np
import torch

from fermiphasespace_b200 import engine as E

PRECISION = {"fp64": E.PREC_FP64, "fp32": E.PREC_FP32, "bf16x3": E.PREC_SPLIT_BF16X3,
             "tf32x3": E.PREC_SPLIT_TF32X3}
DIAGONALS = ("niiu", "niid", "n2iiu", "n2iid", "nund")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest calls: the 3x2 grid of the repository's CPU-runnable configuration, Neel state,
        # ten steps per snapshot; latency of a stage and of the call
        {"name": "ftwa_grid3x2_fp64", "kind": "ftwa", "lattice": "grid", "nx": 3, "ny": 2, "nz": 1,
         "precision": "fp64", "traj": 1000, "snapshots": 41, "steps": 10, "dt": 0.01, "coulomb": "onsite",
         "U": 4.0, "W": 0.0, "state": "neel", "whole": False, "energies": True},
        # the headline benchmark: 10x10 grid, random site potential, domain wall, densities and doublons
        {"name": "ftwa_grid10x10_fp32", "kind": "ftwa", "lattice": "grid", "nx": 10, "ny": 10, "nz": 1,
         "precision": "fp32", "traj": 16384, "snapshots": 41, "steps": 1, "dt": 0.005, "coulomb": "onsite",
         "U": 4.0, "W": 2.0, "state": "wall", "whole": False, "energies": False},
        # the same system in FP64, every default observable
        {"name": "ftwa_grid10x10_fp64", "kind": "ftwa", "lattice": "grid", "nx": 10, "ny": 10, "nz": 1,
         "precision": "fp64", "traj": 4096, "snapshots": 41, "steps": 1, "dt": 0.005, "coulomb": "onsite",
         "U": 8.0, "W": 2.0, "state": "wall", "whole": False, "energies": True},
        # an odd lattice with the distance Coulomb interaction (U and same-spin V everywhere)
        {"name": "ftwa_grid7x9_fp32_distance", "kind": "ftwa", "lattice": "grid", "nx": 7, "ny": 9, "nz": 1,
         "precision": "fp32", "traj": 777, "snapshots": 81, "steps": 2, "dt": 0.01, "coulomb": "distance",
         "U": 2.0, "W": 0.0, "state": "random", "whole": False, "energies": True},
        # a large lattice (the site count of the moire configuration on a grid)
        {"name": "ftwa_grid16x16_fp32", "kind": "ftwa", "lattice": "grid", "nx": 16, "ny": 16, "nz": 1,
         "precision": "fp32", "traj": 512, "snapshots": 21, "steps": 1, "dt": 0.005, "coulomb": "onsite",
         "U": 4.0, "W": 1.0, "state": "wall", "whole": False, "energies": True},
        # from the rotated (tight-binding ground) state, whole density matrices, as `fps` runs a quench
        # from an eigenstate and reports occupations of eigenstates
        {"name": "ftwa_kagome48_rotated_fp64", "kind": "ftwa", "lattice": "kagome", "nx": 4, "ny": 4, "nz": 1,
         "precision": "fp64", "traj": 2048, "snapshots": 21, "steps": 2, "dt": 0.01, "coulomb": "onsite",
         "U": 2.0, "W": 1.0, "state": "ground", "whole": True, "energies": True},
        # Hartree-Fock: one deterministic trajectory, on-site interaction, the 10x10 grid
        {"name": "hf_grid10x10_fp64", "kind": "hf", "lattice": "grid", "nx": 10, "ny": 10, "nz": 1,
         "precision": "fp64", "traj": 1, "snapshots": 401, "steps": 1, "dt": 0.005, "coulomb": "onsite",
         "U": 4.0, "W": 2.0, "state": "ground", "whole": False, "energies": True},
        # Hartree-Fock with the distance Coulomb interaction (Fock term: a dense complex Hamiltonian)
        {"name": "hf_grid8x8_distance_fp64", "kind": "hf", "lattice": "grid", "nx": 8, "ny": 8, "nz": 1,
         "precision": "fp64", "traj": 1, "snapshots": 201, "steps": 1, "dt": 0.01, "coulomb": "distance",
         "U": 2.0, "W": 1.0, "state": "ground", "whole": False, "energies": True},
        # long-range hopping and Coulomb: the 256-site twisted bilayer on the tensor-core path
        {"name": "ftwa_moire256_bf16x3", "kind": "ftwa", "lattice": "moire", "nx": 8, "ny": 8, "nz": 1,
         "precision": "bf16x3", "traj": 1024, "snapshots": 11, "steps": 1, "dt": 0.005, "coulomb": "distance",
         "U": 1.0, "W": 0.0, "state": "random", "whole": False, "energies": True},
        # several lattices of uneven size in one call (a quarter of the repository's batch configuration)
        {"name": "batch_uneven_fp32", "kind": "batch", "precision": "fp32", "snapshots": 41, "steps": 1,
         "dt": 0.01, "U": 4.0, "members": "kagome:6:6:1:512,honeycomb:3:4:1:256,fcc:3:3:3:256,grid:8:8:1:512,"
                                          "grid:12:12:1:512"},
        # gradients of the time-integrated doublon occupancy: 8x8 grid with a pulse
        {"name": "grad_grid8x8_fp32", "kind": "grad", "lattice": "grid", "nx": 8, "ny": 8, "nz": 1,
         "precision": "fp32", "traj": 1024, "snapshots": 101, "steps": 1, "dt": 0.01, "U": 4.0, "bins": 50,
         "checkpoint": 16},
        # gradients in FP64 on a small odd lattice (the reference gradient of a fit)
        {"name": "grad_grid5x5_fp64", "kind": "grad", "lattice": "grid", "nx": 5, "ny": 5, "nz": 1,
         "precision": "fp64", "traj": 300, "snapshots": 41, "steps": 2, "dt": 0.01, "U": 3.0, "bins": 7,
         "checkpoint": 10},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


#: Work (flops) that a drawn case of each kind may take at most, so that none costs more than the listed ones.
CEILING = {"fp64": 3.0e11, "fp32": 1.2e12, "bf16x3": 6e12, "tf32x3": 6e12, "hf": 3e9, "grad": 1.2e11, "batch": 2e11,
           "large": 1.5e11}


def _lattice(rng, largest):
    kind = rng.choice(["grid", "grid", "grid", "honeycomb", "kagome", "fcc"])
    while True:
        if kind == "fcc":
            d = [rng.randint(1, 3) for _ in range(3)]
        else:
            d = [rng.randint(2, 16), rng.randint(2, 16), 1]
        n = d[0] * d[1] * d[2] * {"grid": 1, "honeycomb": 2, "kagome": 3, "fcc": 4}[kind]
        if 4 <= n <= largest:
            return {"lattice": kind, "nx": d[0], "ny": d[1], "nz": d[2]}


def draw(rng):
    kind = rng.choice(["ftwa", "ftwa", "ftwa", "ftwa", "hf", "hf", "moire", "batch", "grad", "grad"])
    if kind == "batch":
        parts = []
        for _ in range(rng.randint(2, 5)):
            c = _lattice(rng, 144)
            parts.append("%s:%d:%d:%d:%d" % (c["lattice"], c["nx"], c["ny"], c["nz"], _log_int(rng, 64, 512)))
        c = {"kind": "batch", "precision": rng.choice(["fp32", "fp32", "fp64"]), "snapshots": rng.randint(5, 41),
             "steps": rng.choice([1, 1, 2]), "dt": 0.01, "U": rng.choice([2.0, 4.0, 8.0]),
             "members": ",".join(parts)}
        while work(c)["flops"] > CEILING["batch"]:
            c["snapshots"] = max(2, c["snapshots"] * 2 // 3)
            if c["snapshots"] == 2:
                break
        return c
    if kind == "grad":
        c = dict(_lattice(rng, 64), kind="grad", precision=rng.choice(["fp32", "fp32", "fp64"]),
                 traj=_log_int(rng, 32, 1024), snapshots=rng.randint(11, 101), steps=rng.choice([1, 1, 2, 3]),
                 dt=0.01, U=rng.choice([2.0, 3.0, 4.0]), bins=rng.randint(3, 50), checkpoint=rng.choice([8, 10, 16]))
        top = CEILING["grad"]
    elif kind == "hf":
        c = dict(_lattice(rng, 128), kind="hf", precision=rng.choice(["fp64", "fp64", "fp32"]), traj=1,
                 snapshots=_log_int(rng, 21, 401), steps=rng.choice([1, 1, 2]), dt=0.005,
                 coulomb=rng.choice(["onsite", "distance"]), U=rng.choice([1.0, 2.0, 4.0]),
                 W=rng.choice([0.0, 1.0, 2.0]), state=rng.choice(["ground", "neel", "wall"]), whole=False,
                 energies=True)
        top = CEILING["hf"]
    elif kind == "moire":
        c = {"kind": "ftwa", "lattice": "moire", "nx": rng.randint(5, 8), "ny": rng.randint(5, 8), "nz": 1,
             "precision": rng.choice(["bf16x3", "bf16x3", "tf32x3"]), "traj": _log_int(rng, 64, 1024),
             "snapshots": rng.randint(3, 11), "steps": rng.choice([1, 1, 2]), "dt": 0.005,
             "coulomb": rng.choice(["onsite", "distance"]), "U": rng.choice([1.0, 2.0]), "W": 0.0, "state": "random",
             "whole": False, "energies": True}
        top = CEILING[c["precision"]]
    else:
        c = dict(_lattice(rng, 256), kind="ftwa", precision=rng.choice(["fp32", "fp32", "fp64"]),
                 traj=_log_int(rng, 64, 16384), snapshots=_log_int(rng, 5, 201), steps=rng.choice([1, 1, 2, 5]),
                 dt=rng.choice([0.005, 0.01]), coulomb=rng.choice(["onsite", "onsite", "distance"]),
                 U=rng.choice([1.0, 2.0, 4.0, 8.0]), W=rng.choice([0.0, 1.0, 2.0]),
                 state=rng.choice(["neel", "wall", "random", "ground"]), whole=False, energies=rng.random() < 0.7)
        n = sites(c)
        if n <= 100 and rng.random() < 0.3:
            c["whole"] = True
        if c["state"] == "ground":
            c["traj"] = min(c["traj"], 4096)
        if n > 100:
            c["traj"] = min(c["traj"], 1024)
        top = CEILING["large"] if n > 100 else CEILING[c["precision"]]
        c["traj"] = max(32, min(c["traj"], int(4e9 / (32 * n * n))))
        if c["steps"] > 2 and n > 64:
            c["steps"] = 2
    while work(c)["flops"] > top:
        if c["snapshots"] > 5:
            c["snapshots"] = max(5, c["snapshots"] * 2 // 3)
        elif c["traj"] > 32:
            c["traj"] = max(32, c["traj"] * 2 // 3)
        else:
            break
    return c


# ------------------------------------------------------------------ systems
def positions(kind, nx, ny, nz):
    """Site positions with nearest neighbours at distance 1 (moire: in units of the hopping's length)."""
    if kind == "grid":
        return np.array([(x, y, z) for z in range(nz) for y in range(ny) for x in range(nx)], dtype=float)
    if kind == "honeycomb":
        a, basis = [(math.sqrt(3), 0, 0), (math.sqrt(3) / 2, 1.5, 0), (0, 0, 0)], [(0, 0, 0), (0, 1, 0)]
    elif kind == "kagome":
        a, basis = [(2, 0, 0), (1, math.sqrt(3), 0), (0, 0, 0)], [(0, 0, 0), (1, 0, 0), (0.5, math.sqrt(3) / 2, 0)]
    elif kind == "fcc":
        s = math.sqrt(2)
        a, basis = [(s, 0, 0), (0, s, 0), (0, 0, s)], [(0, 0, 0), (s / 2, s / 2, 0), (s / 2, 0, s / 2), (0, s / 2, s / 2)]
    else:   # two honeycomb layers, the second turned by 5 degrees and 3.35 above
        flat = 1.42 * positions("honeycomb", nx, ny, 1)
        mid = flat.mean(0)
        th = math.radians(5.0)
        rot = np.array([[math.cos(th), -math.sin(th), 0], [math.sin(th), math.cos(th), 0], [0, 0, 1]])
        return np.concatenate([flat, (flat - mid) @ rot.T + mid + [0, 0, 3.35]])
    a = np.array(a, dtype=float)
    return np.array([x * a[0] + y * a[1] + z * a[2] + np.array(b) for z in range(nz) for y in range(ny)
                     for x in range(nx) for b in basis])


def sites(c):
    return c["nx"] * c["ny"] * c["nz"] * {"grid": 1, "honeycomb": 2, "kagome": 3, "fcc": 4, "moire": 4}[c["lattice"]]


def system(c, seed):
    """Hopping, Coulomb and potential matrices, occupations (and eigenvectors) of a case, from the seed."""
    rng = np.random.default_rng(seed)
    pos = positions(c["lattice"], c["nx"], c["ny"], c["nz"])
    n = len(pos)
    D = np.sqrt(((pos[:, None, :] - pos[None, :, :]) ** 2).sum(-1))
    if c["lattice"] == "moire":
        T = np.where((D > 1e-6) & (D <= 4 * 1.42), -np.exp(-(D - 1.42) / 0.45), 0.0)
    else:
        T = np.where(np.abs(D - 1.0) < 1e-2, -1.0, 0.0)
    if c.get("coulomb", "onsite") == "distance":
        U = c["U"] / (1.0 + D)
        V = U - np.diag(np.diag(U))
    else:
        U, V = np.diag(np.full(n, c["U"])), np.zeros((n, n))
    W = c.get("W", 0.0)
    ext = np.diag(rng.uniform(-W / 2, W / 2, n)) if W else None
    state = c.get("state", "random")
    up, dn, rot = np.zeros(n), np.zeros(n), None
    if state == "neel":
        up[::2], dn[1::2] = 1.0, 1.0
    elif state == "wall":
        left = pos[:, 0] < pos[:, 0].mean()
        up[left], dn[left] = 1.0, 1.0
    elif state == "ground":   # half filling of the eigenstates of the hopping in a weak site potential of its own
        _, rot = np.linalg.eigh(T + np.diag(rng.uniform(-0.2, 0.2, n)))
        up[: (n + 1) // 2], dn[: n // 2] = 1.0, 1.0
    else:
        up[rng.permutation(n)[: (n + 1) // 2]], dn[rng.permutation(n)[: n // 2]] = 1.0, 1.0
    return {"n": n, "T": T, "U": U, "V": V, "ext": ext, "up": up, "dn": dn, "rot": rot}


def pulse_of(c, seed):
    """Gaussian-envelope site pulse with one amplitude per time bin, as the adjoint configuration has it."""
    rng = np.random.default_rng(seed + 17)
    pos = positions(c["lattice"], c["nx"], c["ny"], c["nz"])
    t_max = (c["snapshots"] - 1) * c["dt"]
    return {"amp": rng.normal(0.0, 0.5, c["bins"]), "bin_width": t_max / c["bins"], "t0": t_max / 2, "td": t_max / 5,
            "proj": pos[:, 0] - pos[:, 0].mean()}


def members(c, seed):
    out = []
    for k, part in enumerate(c["members"].split(",")):
        lat, nx, ny, nz, traj = part.split(":")
        m = {"lattice": lat, "nx": int(nx), "ny": int(ny), "nz": int(nz), "traj": int(traj), "U": c["U"]}
        s = system(m, seed + 101 * k)
        out.append((m, s, seed * 31 + k))
    return out


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    c = case
    eng = E.Engine()
    st = {"case": c, "eng": eng, "seed": seed}
    if c["kind"] == "batch":
        st["systems"] = [{"tM": s["T"], "U": s["U"], "V": None, "ext": None, "coulomb": E.COUL_ONSITE,
                          "n_traj": m["traj"], "seed": sd, "occ_up": s["up"], "occ_dn": s["dn"]}
                         for m, s, sd in members(c, seed)]
        return st
    s = st["sys"] = system(c, seed)
    distance = c.get("coulomb", "onsite") == "distance"
    eng.set_system(s["T"], s["U"], s["V"] if distance else None, ext=s["ext"],
                   coulomb=E.COUL_DISTANCE if distance else E.COUL_ONSITE)
    if c["kind"] == "grad":
        eng.set_grad_memory(24 << 30)     # so that several programs can share the card
        eng.set_pulse(**pulse_of(c, seed))
    if c["kind"] == "hf":
        st["rho0"] = hf_state(s)
    st["obs"] = E.OBS_DIAG | E.OBS_DIAG2 | E.OBS_DOUBLONS | (E.OBS_ENERGIES if c.get("energies") else 0) | (
        E.OBS_WHOLE if c.get("whole") else 0)
    return st


def hf_state(s):
    out = []
    for occ in (s["up"], s["dn"]):
        N = np.diag(occ).astype(complex) if s["rot"] is None else (s["rot"] * occ) @ s["rot"].T + 0j
        out.append(N)
    return np.stack(out)[None]


def observables(c, r):
    f = np.float64 if c["precision"] == "fp64" else np.float32
    out = {k: getattr(r, k).astype(f) for k in DIAGONALS}
    if c.get("energies", True):
        out["energies"] = r.energies.astype(f)
    if c.get("whole"):
        w = np.stack([r.whole_u, r.whole_d])
        out["whole_re"], out["whole_im"] = w.real.astype(f), w.imag.astype(f)
    return out


def run(state):
    c, eng, seed = state["case"], state["eng"], state["seed"]
    prec = PRECISION[c["precision"]]
    if c["kind"] == "batch":
        rs, _ = eng.run_batch(state["systems"], E.METHOD_FTWA, prec, c["dt"], c["steps"], c["snapshots"])
        return [observables(c, r) for r in rs]
    s = state["sys"]
    if c["kind"] == "hf":
        eng.set_initial_samples(state["rho0"])
        return observables(c, eng.run(E.METHOD_HF, prec, c["dt"], c["steps"], c["snapshots"], state["obs"]))
    eng.sample(c["traj"], seed, s["up"], s["dn"], s["rot"], s["rot"])
    if c["kind"] == "grad":
        g = eng.grad(prec, c["dt"], c["steps"], c["snapshots"], c["checkpoint"])
        f = np.float64 if c["precision"] == "fp64" else np.float32
        return {k: np.asarray(g[k], dtype=f) for k in ("loss", "dU", "dt", "dpulse")}
    return observables(c, eng.run(E.METHOD_FTWA, prec, c["dt"], c["steps"], c["snapshots"], state["obs"]))


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c = case
    if c["kind"] == "batch":
        parts = [dict(zip(("lattice", "nx", "ny", "nz", "traj"), p.split(":"))) for p in c["members"].split(",")]
        tot = {"bytes": 0.0, "flops": 0.0}
        for p in parts:
            p = {k: v if k == "lattice" else int(v) for k, v in p.items()}
            w = work(dict(c, kind="ftwa", state="random", coulomb="onsite", whole=False, **p))
            tot = {k: tot[k] + w[k] for k in tot}
        return tot
    n, B, S, Tp = sites(c), c["traj"], c["steps"], c["snapshots"]
    hf, distance = c["kind"] == "hf", c.get("coulomb", "onsite") == "distance"
    nsteps = (Tp if c["kind"] == "ftwa" else Tp - 1) * S
    if c["lattice"] == "moire" or (hf and distance):
        step = 64.0 * n ** 3                                   # two dense commutators, four stages
    else:
        T = system(dict(c, W=0.0, state="random"), 0)["T"]
        step = 64.0 * n * (np.count_nonzero(T) + n)            # the same with Delta's nonzeros alone
    flops = B * nsteps * step * (2.5 if c["kind"] == "grad" else 1.0)
    if c.get("state") == "ground" and not hf:
        flops += B * 2 * 12.0 * n ** 3                         # rho -> R rho R^H
    state = B * 2 * (n * (n + 1) // 2) * 16.0
    out = 8.0 * Tp * (5 * n + 5 + (4 * n * n if c.get("whole") else 0))
    return {"bytes": 2 * state + out, "flops": float(flops)}


# ------------------------------------------------------------------ the same in 64 bits
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x, dev):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=dev)


def _philox(c, key):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors that hold 32-bit words."""
    M0, M1, m32 = 0xD2511F53, 0xCD9E8D57, 0xFFFFFFFF
    k0, k1 = key
    for _ in range(10):
        a, b = c[0] * M0, c[2] * M1                            # wraps at 64 bits
        c = [((b >> 32) & m32) ^ c[1] ^ k0, b & m32, ((a >> 32) & m32) ^ c[3] ^ k1, a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c


def samples(s, seed, b0, b1, dev):
    """Initial (re, im) of rho = N - 1/2, [b, 2, n, n], of trajectories b0 .. b1-1."""
    n, B = s["n"], b1 - b0
    iu = torch.triu_indices(n, n, 1, device=dev)
    i, j = iu[0], iu[1]
    b = torch.arange(b0, b1, device=dev, dtype=torch.int64)[:, None]
    re, im = (torch.zeros(B, 2, n, n, dtype=torch.float64, device=dev) for _ in range(2))
    for spin, (occ, e) in enumerate(((s["up"], j * n + i), (s["dn"], i * n + j))):
        o = _t(occ, dev)
        z = torch.zeros(B, len(i), dtype=torch.int64, device=dev)
        w = _philox([z + e, z + (b & 0xFFFFFFFF), z + (b >> 32), z + 0x46505347], (seed & 0xFFFFFFFF, seed >> 32))
        # the upper 53 bits of each 64-bit pair
        ua = ((((w[0] << 21) | (w[1] >> 11)).double()) + 0.5) * 2.0 ** -53
        ub = ((((w[2] << 21) | (w[3] >> 11)).double()) + 0.5) * 2.0 ** -53
        r = torch.sqrt(-2.0 * torch.log(ua))
        th = 2 * math.pi * ub
        sg = torch.sqrt((o[i] + o[j] - 2 * o[i] * o[j]) / 2) / math.sqrt(2.0)
        g1, g2 = r * torch.cos(th) * sg, r * torch.sin(th) * sg * (1 if spin == 0 else -1)
        re[:, spin, i, j], re[:, spin, j, i] = g1, g1
        im[:, spin, i, j], im[:, spin, j, i] = g2, -g2
        d = torch.arange(n, device=dev)
        re[:, spin, d, d] = o - 0.5
    if s["rot"] is not None:      # real eigenvectors
        R = _t(s["rot"], dev)
        re, im = R @ re @ R.T, R @ im @ R.T
    return re, im


class Dynamics:
    """d rho/dt = -i [rho, Delta(rho)] of both spins, dense, on (re, im) pairs [b, 2, n, n]."""

    def __init__(self, s, distance, hf, dev, pulse=None, uscale=None, tscale=None, amp=None):
        self.T, self.U, self.V = _t(s["T"], dev), _t(s["U"], dev), _t(s["V"], dev)
        self.Ht = self.T
        self.ext = None if s["ext"] is None else _t(s["ext"], dev)
        self.shift, self.distance, self.fock = (0.0 if hf else 0.5), distance, hf and distance
        self.pulse, self.amp = pulse, amp
        self.proj = None if pulse is None else _t(pulse["proj"], dev)
        self.ud, self.vd = self.U, self.V
        if uscale is not None:
            self.ud, self.vd, self.Ht = self.U * uscale, self.V * uscale, self.T * tscale

    def diag(self, re, t):
        nn = torch.diagonal(re, dim1=-2, dim2=-1) + self.shift
        d = nn.flip(1) @ self.ud
        if self.distance:
            d = d + nn @ self.vd
        if self.ext is not None:
            d = d + torch.diagonal(self.ext)
        if self.pulse is not None:
            p = self.pulse
            k = min(max(int(math.floor(t / p["bin_width"])), 0), len(p["amp"]) - 1)
            d = d + self.amp[k] * math.exp(-0.5 * ((t - p["t0"]) / p["td"]) ** 2) * self.proj
        return d

    def k(self, x, t):
        re, im = x
        d = self.diag(re, t)[:, :, None, :]
        if self.fock:
            D = torch.complex(self.Ht - self.vd * re, -self.vd * im) + torch.diag_embed(d[:, :, 0, :]).to(torch.complex128)
            X = torch.complex(re, im)
            G = X @ D
            gr, gi = G.real, G.imag
        else:
            gr, gi = re @ self.Ht + re * d, im @ self.Ht + im * d
        return gi + gi.transpose(-1, -2), gr.transpose(-1, -2) - gr

    def step(self, x, t, h, dt):
        def add(y, *terms):
            return tuple(sum((c * k[p] for c, k in terms), y[p]) for p in (0, 1))
        k1 = self.k(x, t)
        k2 = self.k(add(x, (h / 3, k1)), t + h / 3)
        k3 = self.k(add(x, (-h / 3, k1), (h, k2)), t + 2 * dt / 3)
        k4 = self.k(add(x, (h, k1), (-h, k2), (h, k3)), t + h)
        return add(x, (h / 8, k1), (3 * h / 8, k2), (3 * h / 8, k3), (h / 8, k4))

    def record(self, x, energies, whole):
        """Ensemble sums of one snapshot."""
        re, im = x
        r = torch.diagonal(re, dim1=-2, dim2=-1)
        u, d = r[:, 0], r[:, 1]
        out = {"d": torch.stack([u.sum(0), d.sum(0), (u * u).sum(0), (d * d).sum(0), (u * d).sum(0)])}
        if energies:
            nn = r + self.shift
            N = re + self.shift * torch.eye(re.shape[-1], dtype=re.dtype, device=re.device)
            e1 = 0.5 * ((nn[:, 0] * (nn[:, 1] @ self.U)).sum() + (nn[:, 1] * (nn[:, 0] @ self.U)).sum())
            e2 = 0.5 * (nn * (nn @ self.V)).sum()
            if self.fock:
                e2 = e2 - 0.5 * (self.V * (re * re + im * im)).sum()
            e3 = (N * self.ext).sum() if self.ext is not None else torch.zeros_like(e1)
            out["e"] = torch.stack([(N * self.T).sum(), e1, e2, e3])
        if whole:
            out["wr"], out["wi"] = re.sum(0), im.sum(0)
        return out


def _simulate(c, s, first, B, hf, seed, dev):
    """The observables of one ensemble, run in pieces of trajectories."""
    n, Tp, S = s["n"], c["snapshots"], c["steps"]
    distance = c.get("coulomb", "onsite") == "distance"
    dyn = Dynamics(s, distance, hf, dev)
    piece = max(1, int(4e8 / (2 * n * n * 8)))
    total = None
    for b0 in range(0, B, piece):
        b1 = min(B, b0 + piece)
        x = first(b0, b1)
        recs = []
        for t in range(Tp):
            recs.append(dyn.record(x, c.get("energies", True), c.get("whole", False)))
            for _ in range(S if t < Tp - 1 else 0):
                x = dyn.step(x, 0.0, c["dt"] / S, c["dt"])     # nothing but a pulse depends on time
        got = {k: torch.stack([r[k] for r in recs]) for k in recs[0]}
        total = got if total is None else {k: total[k] + got[k] for k in got}
    m = {k: v.cpu().numpy() / B for k, v in total.items()}
    u, d, uu, dd, ud = (m["d"][:, k].T for k in range(5))
    h = 0.0 if hf else 0.5
    out = {"niiu": u + h, "niid": d + h, "n2iiu": uu + 2 * h * u + h * h, "n2iid": dd + 2 * h * d + h * h,
           "nund": ud + h * (u + d) + h * h}
    if c.get("energies", True):
        e = m["e"].T
        out["energies"] = np.concatenate([e, e.sum(0, keepdims=True)])
    if c.get("whole"):
        wr = np.moveaxis(m["wr"], 1, 0) + h * np.eye(n)
        out["whole_re"], out["whole_im"] = wr, np.moveaxis(m["wi"], 1, 0)
    return out


def _gradient(c, s, seed, dev):
    p = pulse_of(c, seed)
    h = c["dt"] / c["steps"]
    loss, grads = 0.0, None
    # trajectories whose graph takes about 40 GB
    piece = max(1, int(40e9 / ((c["snapshots"] - 1) * c["steps"] * 4 * 2 * s["n"] ** 2 * 8 * 14)))
    for b0 in range(0, c["traj"], piece):
        b1 = min(c["traj"], b0 + piece)
        x = samples(s, seed, b0, b1, dev)
        us, ts = (torch.ones((), dtype=torch.float64, device=dev, requires_grad=True) for _ in range(2))
        amp = _t(p["amp"], dev).requires_grad_()
        dyn = Dynamics(s, False, False, dev, p, us, ts, amp)
        L, now = 0.0, 0.0
        for t in range(c["snapshots"]):
            r = torch.diagonal(x[0], dim1=-2, dim2=-1) + 0.5
            w = c["dt"] * (0.5 if t in (0, c["snapshots"] - 1) else 1.0)
            L = L + w * (r[:, 0] * r[:, 1]).sum() / (s["n"] * c["traj"])
            for _ in range(c["steps"] if t < c["snapshots"] - 1 else 0):
                x = dyn.step(x, now, h, c["dt"])
                now += h                                       # the pulse's bins follow the accumulated time
        g = [v.detach().cpu().numpy() for v in torch.autograd.grad(L, [us, ts, amp])]
        loss += float(L.detach())
        grads = g if grads is None else [a + b for a, b in zip(grads, g)]
    return {"loss": np.float64(loss), "dU": grads[0], "dt": grads[1], "dpulse": grads[2]}


def exact(case, seed):
    c, dev = case, _dev()
    if dev.type == "cpu" and work(c)["flops"] > 2e10:
        return None
    if c["kind"] == "batch":
        return [_simulate(dict(c, coulomb="onsite"), s, lambda a, b, s=s, sd=sd: samples(s, sd, a, b, dev), m["traj"],
                          False, sd, dev) for m, s, sd in members(c, seed)]
    s = system(c, seed)
    if c["kind"] == "grad":
        return _gradient(c, s, seed, dev)
    if c["kind"] == "hf":
        r0 = hf_state(s)
        return _simulate(c, s, lambda a, b: (_t(r0.real, dev), _t(r0.imag, dev)), 1, True, seed, dev)
    return _simulate(c, s, lambda a, b: samples(s, seed, a, b, dev), c["traj"], False, seed, dev)
