"""The work a user has this framework do, as a list of measured cases.

Every case goes through the package's public entry points (Engine, Surrogate, Mlp, postmc) on a
seeded synthetic system with the sizes of the benchmark configurations and of the two real
complexes of the tests:

  score   energies of given poses (rescoring): from a few poses of a small pocket, where the
          call's own latency counts, to thousands of poses of the largest pocket and ligand
  dock    a replica-exchange Monte Carlo run from the start pose: energies of the start, Monte
          Carlo steps with an exchange every ten, the chains' state read back; a real-size
          pocket (with its records read back), one complex of 128 replicas, one of 6,820
  screen  the same for a ragged batch of ligands docked to several pockets in one context
  da      delayed-acceptance steps with a trained surrogate
  train   loss and gradients of the surrogate network for one batch
  predict the surrogate network's energies of a batch of rows
  cluster the post-Monte-Carlo clustering of a run's records (k-means per replica, pooled)

Distributions: protein points on a jittered lattice (at least 3 A apart, 0.0165 per cubic A)
around a 6 A cavity; bonded-chain ligands with random torsions per conformer, centred on the
cavity; force-field tables in the ranges of the reference's parameters (LJ radii 1.9-4.9 A,
contact distances 2.7-7.4 A, Gaussian contact depths, hydrogen bonds between a third of the
ligand types and a third of the point types); temperatures geometric in kT from 0.3 to 3.
"""
import math

import numpy as np
import torch

from geaxdock_gpu_b200 import abi, engine, postmc

N_PROT_TYPES, N_LIG_TYPES = 24, 12


def listed():
    return [
        # a handful of poses of a small real-size pocket (21 atoms, 410 points): a rescoring
        # service's single request, all latency
        {"name": "score_24_small", "kind": "score", "poses": 24, "lna": 21, "pnp": 410,
         "n_prt": 2, "pnk": 191, "pos": 11},
        # thousands of poses of the 3,000-point, 40-atom system: rescoring a docking run
        {"name": "score_4096", "kind": "score", "poses": 4096, "lna": 40, "pnp": 3000,
         "n_prt": 2, "pnk": 40, "pos": 8},
        # the largest pocket and ligand of the screen
        {"name": "score_16384_large", "kind": "score", "poses": 16384, "lna": 64, "pnp": 6000,
         "n_prt": 1, "pnk": 40, "pos": 8},
        # one real-size complex (34 atoms, 344 points, 252 replicas), a window of 100 steps with
        # its records
        {"name": "dock_real_size", "kind": "dock", "lna": 34, "pnp": 344, "n_prt": 3,
         "n_lig": 21, "n_tmp": 4, "pnk": 454, "pos": 11, "steps": 100, "records": True},
        # one complex of 128 replicas: too few to fill the GPU
        {"name": "dock_128_replicas", "kind": "dock", "lna": 28, "pnp": 1500, "n_prt": 1,
         "n_lig": 8, "n_tmp": 16, "pnk": 40, "pos": 8, "steps": 100, "records": False},
        # the batched benchmark system (6,820 replicas), one exchange interval
        {"name": "dock_6820_replicas", "kind": "dock", "lna": 40, "pnp": 3000, "n_prt": 11,
         "n_lig": 31, "n_tmp": 20, "pnk": 40, "pos": 8, "steps": 10, "records": False},
        # a ragged batch of ligands (10-64 atoms) on pockets of 1,200-6,000 points
        {"name": "screen_16_ligands", "kind": "screen", "ligands": 16, "pockets": 4,
         "n_prt": 4, "n_lig": 8, "n_tmp": 16, "steps": 10},
        # production steps with a trained surrogate, at the move size where about a fifth of
        # the proposals survive
        {"name": "delayed_acceptance", "kind": "da", "lna": 34, "pnp": 410, "n_prt": 11,
         "n_lig": 21, "n_tmp": 20, "pnk": 191, "pos": 11, "steps": 20, "moves": 60.0,
         "train": 100},
        # one training batch of the surrogate
        {"name": "surrogate_gradients_8192", "kind": "train", "rows": 8192, "hidden": 256,
         "n_emb": 341},
        # the surrogate on one row per replica
        {"name": "surrogate_predict_6820", "kind": "predict", "rows": 6820, "hidden": 256,
         "n_emb": 341},
        # the records of a run of 3,410 replicas
        {"name": "cluster_records", "kind": "cluster", "replicas": 3410, "records": 180},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score", "score", "score", "dock", "dock", "dock", "screen", "da", "train",
                       "predict", "cluster"])
    if kind == "score":
        lna, pnp = rng.randint(10, 64), _log(rng, 300, 6000)
        most = max(16, min(16384, 64 * 6000 * 16384 // (lna * pnp)))
        return {"kind": kind, "poses": _log(rng, 16, most), "lna": lna, "pnp": pnp,
                "n_prt": rng.randint(1, 3), "pnk": _log(rng, 20, 450), "pos": rng.randint(3, 12)}
    if kind == "dock":
        n_prt, n_lig, n_tmp = rng.randint(1, 11), rng.randint(4, 31), rng.randint(2, 20)
        n_rep = n_prt * n_lig * n_tmp
        return {"kind": kind, "lna": rng.randint(15, 48), "pnp": _log(rng, 300, 4000),
                "n_prt": n_prt, "n_lig": n_lig, "n_tmp": n_tmp, "pnk": _log(rng, 20, 450),
                "pos": rng.randint(3, 12),
                "steps": 10 * max(1, min(10, 6820 // n_rep, _log(rng, 1, 10))),
                "records": rng.random() < 0.3}
    if kind == "screen":
        return {"kind": kind, "ligands": rng.randint(3, 16), "pockets": rng.randint(1, 4),
                "n_prt": rng.randint(1, 4), "n_lig": rng.randint(3, 8),
                "n_tmp": rng.randint(4, 16), "steps": 10}
    if kind == "da":
        return {"kind": kind, "lna": rng.randint(15, 40), "pnp": rng.randint(300, 420),
                "n_prt": rng.randint(4, 11), "n_lig": rng.randint(8, 21),
                "n_tmp": rng.randint(8, 20), "pnk": _log(rng, 20, 450), "pos": rng.randint(3, 12),
                "steps": 10 * rng.randint(1, 2), "moves": rng.choice([1.0, 20.0, 60.0]),
                "train": rng.randint(60, 120)}
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 200, 8192), "hidden": rng.choice([128, 256]),
                "n_emb": rng.choice([0, 31, 341])}
    if kind == "predict":
        return {"kind": kind, "rows": _log(rng, 100, 20000), "hidden": rng.choice([128, 256]),
                "n_emb": rng.choice([0, 31, 341])}
    return {"kind": kind, "replicas": _log(rng, 50, 3410), "records": rng.randint(40, 180)}


# ---- the synthetic systems ----

def _force_field(rng):
    """Folded tables (abi.EnePara), in the ranges of the reference's parameters."""
    ff = abi.EnePara()
    T2, T1 = abi.MAXTP2, abi.MAXTP1
    sigma = np.clip(rng.normal(3.6, 0.45, (T2, T1)), 1.9, 4.9)
    eps = np.exp(rng.uniform(math.log(0.12), math.log(2.6), (T2, T1)))
    tab = {"p1a": 2.0 * eps * sigma ** 9, "p2a": 3.0 * eps * sigma ** 6,
           "pmf0": np.clip(rng.normal(5.05, 0.6, (T2, T1)), 2.7, 7.38),
           "pmf1": rng.normal(0.0, 1.0, (T2, T1))}
    live = (np.arange(T2)[:, None] % 3 == 0) & (np.arange(T1)[None, :] % 3 == 1)
    tab["hdb0"] = np.where(live, rng.uniform(3.3, 4.5, (T2, T1)), 0.0)
    with np.errstate(divide="ignore"):
        tab["hdb1"] = 1.0 / np.where(live, rng.uniform(0.6, 0.99, (T2, T1)), 0.0)
    for k, v in tab.items():
        np.ctypeslib.as_array(getattr(ff, k))[:] = v.astype(np.float32)
    ff.lj0, ff.lj1 = 0.8814889788627625, 0.7428590059280396
    ff.el0, ff.el1, ff.a1, ff.b1 = 2.0, 0.5, -2.0, 1.0
    ff.ele[:] = rng.normal(0.0, 0.3, abi.MAXTP3).astype(np.float32).tolist()
    ff.hpp[:] = rng.uniform(-1.0, 1.0, abi.MAXTP4).astype(np.float32).tolist()
    hpl1 = rng.uniform(0.35, 0.6, T2).astype(np.float32)
    ff.hpl0[:] = rng.uniform(-0.5, 0.3, T2).astype(np.float32).tolist()
    ff.hpl1[:] = hpl1.tolist()
    ff.hpl2[:] = np.log(1.0 / (hpl1 * math.sqrt(2.0 * math.pi))).astype(np.float32).tolist()
    ff.kde2, ff.kde3 = -2.0, 1.9687012434005737
    ff.w[:] = [1.0, -0.1415438, 0.07523818, 0.18448716, 0.30809662, 0.09295134, -0.38958195,
               0.17181891, 0.01501205, 0.0]
    ff.a_para[:] = [0.77591002, 18.970034, 0.00507, 0.53253597, 2.046236, 0.52519202, 110.81565,
                    0.87786603, 46.40609, 0.0]
    ff.b_para[:] = [1.236367, -0.021163, -0.410825, 0.066766, 1.0, -1.040155, -1.0, -0.167652,
                    -1.0, 0.0]
    return ff


def _protein(rng, ff, pnp, n_prt, center):
    """Points nearest the cavity on a randomly turned, jittered lattice, shared by the
    conformers up to a 0.3 A jitter, and their attributes."""
    step = 0.0165 ** (-1.0 / 3.0)
    n = int(math.ceil((3.0 * (pnp + 40) / (4.0 * math.pi * 0.0165)) ** (1.0 / 3.0) / step)) + 2
    g = (np.stack(np.meshgrid(*[np.arange(-n, n + 1)] * 3, indexing="ij"), -1).reshape(-1, 3) *
         step + rng.uniform(-0.5, 0.5, 3) * step)
    g = g + rng.uniform(-0.3, 0.3, g.shape)
    turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    g = g @ turn
    r = np.linalg.norm(g, axis=1)
    keep = np.argsort(np.where(r < 6.0, np.inf, r))[:pnp]
    base = g[rng.permutation(keep)] + center
    conf = np.stack([base + (rng.normal(0.0, 0.3, base.shape) if n_prt > 1 else 0.0)
                     for _ in range(n_prt)])
    cls = np.arange(pnp) % 4
    res = rng.integers(0, 20, pnp)
    seq = np.arange(pnp) // 3
    psp = np.zeros((abi.MAXTP2, int(seq.max()) + 1), np.float32)
    cols = np.unique(seq[cls == 2])
    psp[:N_LIG_TYPES, cols] = rng.normal(0.0, 0.5, (N_LIG_TYPES, cols.size))
    one = {"prt_t": rng.integers(0, N_PROT_TYPES, pnp), "prt_c": cls,
           "prt_ele": rng.normal(0.0, 0.3, pnp), "prt_seq3r": seq,
           "prt_hflag": ((cls == 0) & (res == 12)) | (cls == 2),
           "prt_hpp": np.array(ff.hpp[:], np.float32)[res]}
    out = {k: np.tile(v, (n_prt, 1)) for k, v in one.items()}
    return dict(out, psp=psp, prt_x=conf[:, :, 0], prt_y=conf[:, :, 1], prt_z=conf[:, :, 2])


def _chain(rng, lna, n_lig):
    """1.5 A bonds, 109.5 degree angles, random torsions; all conformers at once."""
    bond, ang = 1.5, math.radians(109.5)
    x = np.zeros((n_lig, lna, 3))
    x[:, 1:2, 0] = bond
    if lna > 2:
        x[:, 2] = x[:, 1] + bond * np.array([-math.cos(ang), math.sin(ang), 0.0])
    for i in range(3, lna):
        a, b, c = x[:, i - 3], x[:, i - 2], x[:, i - 1]
        bc = (c - b) / bond
        nrm = np.cross(b - a, bc)
        nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
        m = np.cross(nrm, bc)
        tor = rng.uniform(-math.pi, math.pi, (n_lig, 1))
        x[:, i] = c + bond * (-math.cos(ang) * bc + math.sin(ang) * np.cos(tor) * m +
                              math.sin(ang) * np.sin(tor) * nrm)
    return x - x.mean(axis=1, keepdims=True)


def _complex(rng, ff, lna, pnp, n_prt, n_lig, n_tmp, pnk, pos, protein=None, center=None):
    center = np.array([12.5, -3.25, 7.75]) if center is None else center
    protein = _protein(rng, ff, pnp, n_prt, center) if protein is None else protein
    lig = _chain(rng, lna, n_lig)
    q = rng.normal(0.0, 0.3, lna)
    temp = np.zeros(n_tmp, abi.TEMP_DTYPE)
    kt = np.geomspace(0.3, 3.0, n_tmp)
    temp["t"], temp["minus_beta"], temp["order"] = kt, (-1.0 / kt).astype(np.float32), \
        np.arange(n_tmp)
    lig_t = rng.integers(0, N_LIG_TYPES, lna)
    mcs = np.full((3, pos, abi.MAXLIG + 2), abi.MCS_INVALID_COORD, np.float32)
    for m in range(pos):
        valid = np.nonzero(rng.random(lna) < 0.7)[0]
        mcs[:, m, valid + 1] = (lig[0, valid] + center + rng.normal(0.0, 1.0, (valid.size, 3))).T
    kde = center + rng.uniform(-4.0, 4.0, (pnk, 3))
    return abi.ComplexArrays(
        lig_x=lig[:, :, 0], lig_y=lig[:, :, 1], lig_z=lig[:, :, 2],
        lig_center=np.tile(center, (n_lig, 1)), lig_t=np.tile(lig_t, (n_lig, 1)),
        lig_c=np.tile(q - q.mean(), (n_lig, 1)), lig_n=np.tile(np.arange(lna), (n_lig, 1)),
        pocket_center=center, kde_x=kde[:, 0], kde_y=kde[:, 1], kde_z=kde[:, 2],
        kde_t=rng.integers(0, N_LIG_TYPES, pnk), mcs_x=mcs[0], mcs_y=mcs[1], mcs_z=mcs[2],
        mcs_tcc=rng.uniform(0.1, 0.5, pos), temp=temp, **protein)


def _params(seed, record, dump, moves=1.0):
    return abi.mc_params(steps_per_exchange=10, steps_per_dump=dump,
                         move_scale=tuple(moves * v for v in (0.1, 0.1, 0.1, 0.05, 0.05, 0.05)),
                         move_kind=abi.MOVE_GAUSSIAN, record=int(record), seed=seed)


def _score_inputs(case, seed):
    """Force field, complex, and poses spread over the pocket as a docking run leaves them."""
    rng = np.random.default_rng([seed, 1])
    ff = _force_field(rng)
    cx = _complex(rng, ff, case["lna"], case["pnp"], case["n_prt"], 2, 1, case["pnk"],
                  case["pos"])
    mm = np.concatenate([rng.normal(0.0, 1.5, (case["poses"], 3)),
                         rng.uniform(-math.pi, math.pi, (case["poses"], 3))], 1)
    return ff, cx, mm.astype(np.float32)


def _screen_sizes(case):
    """(pnp per pocket, lna per ligand): the same for every seed, so that work() knows them."""
    rng = np.random.default_rng([case["ligands"], case["pockets"], 5])
    return (rng.integers(1200, 6001, case["pockets"]).tolist(),
            rng.integers(10, 65, case["ligands"]).tolist())


def _net_inputs(case, seed):
    """Network parameters, feature rows, conformer ids and targets."""
    rng = np.random.default_rng([seed, 3])
    H, E, n = case["hidden"], case["n_emb"], case["rows"]
    u = lambda *s: rng.uniform(-1.0, 1.0, s) / math.sqrt(s[0])
    parts = [u(64, H), u(H, H)[0], u(H, H), u(H, H)[0], u(H, H), u(H, H)[0], u(H, 1),
             np.zeros(4), rng.uniform(-0.3, 0.3, (E, 32))]
    theta = np.concatenate([p.reshape(-1) for p in parts]).astype(np.float32)
    x = rng.normal(0.0, 0.7, (n, 64)).astype(np.float32)
    conf = rng.integers(0, E, n).astype(np.int32) if E else np.full(n, -1, np.int32)
    t = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 3]).astype(np.float32)
    return theta, x, conf, t


# ---- the cases ----

def prepare(case, seed):
    kind = case["kind"]
    if kind == "score":
        ff, cx, mm = _score_inputs(case, seed)
        return {"kind": kind, "eng": engine.Engine(ff, [cx], _params(seed, 0, 100)), "mm": mm,
                "prt": case["n_prt"] - 1}
    if kind in ("dock", "da"):
        rng = np.random.default_rng([seed, 2])
        ff = _force_field(rng)
        cx = _complex(rng, ff, case["lna"], case["pnp"], case["n_prt"], case["n_lig"],
                      case["n_tmp"], case["pnk"], case["pos"])
        if kind == "dock":
            eng = engine.Engine(ff, [cx], _params(seed, 1, max(100, case["steps"])))
            return {"kind": kind, "eng": eng, "steps": case["steps"], "records": case["records"]}
        eng = engine.Engine(ff, [cx], _params(seed, 1, 100, case["moves"]))
        eng.mc_init()
        sur = engine.Surrogate(eng, embedding=0, sample_cap=1 << 20)
        sur.collect(0, 40)
        sur.train(case["train"])
        sur.run(40, 10)
        return {"kind": kind, "eng": eng, "sur": sur, "steps": case["steps"], "s": 50}
    if kind == "screen":
        rng = np.random.default_rng([seed, 4])
        ff = _force_field(rng)
        pnp, lna = _screen_sizes(case)
        centers = [np.array([100.0 * j, 3.0, -8.0]) for j in range(len(pnp))]
        prots = [_protein(rng, ff, p, case["n_prt"], c) for p, c in zip(pnp, centers)]
        cxs = [_complex(rng, ff, n, 0, case["n_prt"], case["n_lig"], case["n_tmp"], 40, 8,
                        prots[i % len(pnp)], centers[i % len(pnp)]) for i, n in enumerate(lna)]
        return {"kind": "dock", "eng": engine.Engine(ff, cxs, _params(seed, 1, 100)),
                "steps": case["steps"], "records": False}
    if kind in ("train", "predict"):
        theta, x, conf, t = _net_inputs(case, seed)
        net = engine.Mlp(case["hidden"], case["n_emb"], seed=seed)
        net.set_params(theta)
        net.set_params(theta)  # the 16-bit copies are made from parameters that have arrived
        return {"kind": kind, "net": net, "x": x, "conf": conf, "t": t}
    rng = np.random.default_rng([seed, 6])
    counts = rng.integers(case["records"] // 2, case["records"] + 1, case["replicas"])
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    n = int(off[-1])
    # a replica's energies wander slowly about its own level
    w = np.cumsum(rng.normal(0.0, 0.05, (n, abi.MAXWEI)).astype(np.float32), axis=0)
    E = w - np.repeat(w[off[:-1]], counts, axis=0) + np.repeat(
        rng.normal(0.0, 1.0, (case["replicas"], abi.MAXWEI)).astype(np.float32), counts, axis=0)
    return {"kind": kind, "E": E.astype(np.float32), "off": off, "seed": seed}


def _chains(eng):
    """The chains' state as the user reads it back (device errors raised first)."""
    eng.sync()
    st = eng.state()
    return {"move": st["movematrix_old"], "e": st["energy_old"]["e"],
            "cms": st["energy_old"]["cms"], "rmsd": st["energy_old"]["rmsd"],
            "temperature": st["replica"]["idx_tmp"], "accepted": st["n_accept"],
            "exchanged": st["n_exchange"]}


def run(state):
    kind = state["kind"]
    if kind == "score":
        got = state["eng"].eval_energy(0, state["prt"], 1, state["mm"])
        return {"e": got["e"], "cms": got["cms"], "rmsd": got["rmsd"]}
    if kind == "dock":
        eng = state["eng"]
        eng.mc_init()
        eng.run_fused(0, state["steps"])
        out = _chains(eng)
        if state["records"]:
            rows, filled = eng.records()
            out["record_e"], out["filled"] = rows["energy"]["e"], filled
        return out
    if kind == "da":
        eng = state["eng"]
        eng.reset_records()
        state["sur"].run(state["s"], state["steps"])
        state["s"] += state["steps"]
        return _chains(eng)
    if kind == "train":
        loss, grad = state["net"].backward(state["x"], state["t"], state["conf"])
        return {"loss": loss, "grad": grad}
    if kind == "predict":
        return state["net"].forward(state["x"], state["conf"])
    idx, size = postmc.post_mc_indices(state["E"], state["off"], seed=state["seed"] & 0xffff)
    return {"idx": idx, "size": size}


# ---- what a pass cannot do without ----

def _pair_work(n, lna, pnp, pnk, pos):
    """One energy of n poses: 36 operations per ligand-protein pair, 11 per KDE point of the
    atom's type, 9 per atom and restraint position."""
    return n * lna * (36.0 * pnp + 11.0 * pnk / N_LIG_TYPES + 9.0 * 0.7 * pos)


def work(case):
    kind = case["kind"]
    if kind == "score":
        return {"bytes": 72.0 * case["poses"] + case["pnp"] * 32.0,
                "flops": _pair_work(case["poses"], case["lna"], case["pnp"], case["pnk"],
                                    case["pos"])}
    if kind in ("dock", "da"):
        n = case["n_prt"] * case["n_lig"] * case["n_tmp"]
        steps = case["steps"] + (1 if kind == "dock" else 0)
        # delayed acceptance: the network on every proposal, the energy of a fifth of them
        share, net = (1.0, 0.0) if kind == "dock" else (0.2, 2.0 * (64 * 256 + 2 * 256 * 256))
        out = 96.0 * n + (92.0 * n * case["steps"] * 0.8 if case.get("records") else 0.0)
        return {"bytes": out + case["n_prt"] * case["pnp"] * 32.0,
                "flops": steps * (share * _pair_work(n, case["lna"], case["pnp"], case["pnk"],
                                                     case["pos"]) + net * n)}
    if kind == "screen":
        pnp, lna = _screen_sizes(case)
        n = case["n_prt"] * case["n_lig"] * case["n_tmp"]
        return {"bytes": 96.0 * n * len(lna) + sum(pnp) * case["n_prt"] * 32.0,
                "flops": sum((case["steps"] + 1) * _pair_work(n, a, pnp[i % len(pnp)], 40, 8)
                             for i, a in enumerate(lna))}
    if kind in ("train", "predict"):
        H, n = case["hidden"], case["rows"]
        net = 2.0 * n * (64 * H + 2 * H * H + H)
        par = 4.0 * (64 * H + 2 * H * H + 4 * H + 32 * case["n_emb"])
        return {"bytes": n * 4.0 * (66 if kind == "predict" else 67) + par *
                (1 if kind == "predict" else 2), "flops": net * (1 if kind == "predict" else 3)}
    # one assignment of every record to its replica's 50 centres, and of the pooled 50 per
    # replica to 500
    n = 0.75 * case["records"] * case["replicas"]
    return {"bytes": 40.0 * n, "flops": 27.0 * (n * 50 + 50.0 * case["replicas"] * 500)}


# ---- the same values in 64 bits ----

def _exact_score(case, seed):
    ff, cx, mm = _score_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = lambda a: torch.as_tensor(np.array(a, np.float64), device=dev)
    tab = {k: t64(np.ctypeslib.as_array(getattr(ff, k))) for k in
           ("p1a", "p2a", "pmf0", "pmf1", "hdb0", "hdb1", "hpl0", "hpl1", "hpl2")}
    L, P, prt, lig = cx.lna, cx.pnp, case["n_prt"] - 1, 1
    tl = torch.as_tensor(cx.lig_t[lig].astype(np.int64), device=dev)
    tp = torch.as_tensor(cx.prt_t[prt].astype(np.int64), device=dev)
    par = {k: v[tl][:, tp] for k, v in tab.items() if v.dim() == 2}  # [L][P]
    live = par["hdb0"] > float(np.float32(0.1))
    hdb1 = torch.where(live, par["hdb1"], torch.zeros_like(par["hdb1"]))
    q = t64(cx.lig_c[lig])[:, None] * t64(cx.prt_ele[prt])[None, :]
    hpp = t64(cx.prt_hpp[prt] * (cx.prt_hflag[prt] == 1))
    cls2 = torch.as_tensor(cx.prt_c[prt] == 2, device=dev)
    psp = t64(cx.psp)[tl][:, torch.as_tensor(cx.prt_seq3r[prt].astype(np.int64), device=dev)]
    psp = psp * cls2
    orig = torch.stack([t64(a[lig]) for a in (cx.lig_x, cx.lig_y, cx.lig_z)], 1)
    ctr, pocket = t64(cx.lig_center[lig]), t64(cx.pocket_center)
    pts = torch.stack([t64(a[prt]) for a in (cx.prt_x, cx.prt_y, cx.prt_z)], 1)
    # the contacts of the first conformers at the start pose
    ref_lig = torch.stack([t64(a[0]) for a in (cx.lig_x, cx.lig_y, cx.lig_z)], 1) + \
        t64(cx.lig_center[0])
    ref_pts = torch.stack([t64(a[0]) for a in (cx.prt_x, cx.prt_y, cx.prt_z)], 1)
    tl0 = torch.as_tensor(cx.lig_t[0].astype(np.int64), device=dev)
    tp0 = torch.as_tensor(cx.prt_t[0].astype(np.int64), device=dev)
    ref = torch.cdist(ref_lig, ref_pts, compute_mode="donot_use_mm_for_euclid_dist") <= \
        tab["pmf0"][tl0][:, tp0]
    kde = torch.stack([t64(a) for a in (cx.kde_x, cx.kde_y, cx.kde_z)], 1)
    same = (torch.as_tensor(cx.kde_t.astype(np.int64), device=dev)[None, :] == tl[:, None])
    n_same = same.sum(1)
    idx = torch.as_tensor(cx.lig_n[lig].astype(np.int64) + 1, device=dev)
    mcs = torch.stack([t64(a)[:, idx] for a in (cx.mcs_x, cx.mcs_y, cx.mcs_z)], -1)
    valid = mcs[..., 0] != float(np.float32(abi.MCS_INVALID_COORD))
    tcc = t64(cx.mcs_tcc)
    a_para, b_para, w = t64(ff.a_para[:9]), t64(ff.b_para[:9]), t64(ff.w[:9])
    lj0, lj1, el0, el1, a1, b1 = ff.lj0, ff.lj1, ff.el0, ff.el1, ff.a1, ff.b1
    es, cms, rmsd = [], [], []
    poses = t64(mm)
    step = max(1, 12_000_000 // (L * P))
    for i in range(0, poses.shape[0], step):
        m = poses[i:i + step]
        s1, s2, s3 = (torch.sin(m[:, 3 + k]) for k in range(3))
        c1, c2, c3 = (torch.cos(m[:, 3 + k]) for k in range(3))
        rot = torch.stack([c1 * c2, c1 * s2 * s3 - c3 * s1, s1 * s3 + c1 * c3 * s2,
                           c2 * s1, c1 * c3 + s1 * s2 * s3, c3 * s1 * s2 - c1 * s3,
                           -s2, c2 * s3, c2 * c3], 1).reshape(-1, 3, 3)
        at = torch.einsum("nij,lj->nli", rot, orig) + (m[:, :3] + ctr)[:, None, :]
        d2 = sum((at[:, :, None, k] - pts[None, None, :, k]) ** 2 for k in range(3))
        r = d2.sqrt()
        p1, p2 = par["p1a"] / (d2 ** 4 * r), par["p2a"] / d2 ** 3
        vdw = ((p1 - p2) / (p1 * lj0 * (1.0 + lj1 * d2) + 1.0)).sum((1, 2))
        s = el1 * r
        ele = (q * torch.where(s < 1, el0 + a1 * s * s + b1 * s ** 3, 1.0 / s)).sum((1, 2))
        pmf = (par["pmf1"] / (1.0 + torch.exp((6.0 - 0.5 * r) * (r - par["pmf0"])))).sum((1, 2))
        con = r <= par["pmf0"]
        e_psp = (psp * con).sum((1, 2))
        h = (r - par["hdb0"]) * hdb1
        hdb = (-hdb1 / math.sqrt(2.0 * math.pi) * torch.exp(-0.5 * h * h)).sum((1, 2))
        u = d2 / 81.0
        hp = (torch.where(d2 <= 81.0, 1.0 - (3.5 * u - 4.5 * u ** 2 + 2.5 * u ** 3 -
                                             0.5 * u ** 4), torch.zeros_like(u)) * hpp).sum(2)
        h2 = (hp - tab["hpl0"][tl]) / tab["hpl1"][tl]
        hpc = (0.5 * h2 * h2 - tab["hpl2"][tl]).sum(1)
        dk = sum((at[:, :, None, k] - kde[None, None, :, k]) ** 2 for k in range(3))
        ks = (torch.exp(ff.kde2 * dk) * same).sum(2) / n_same.clamp(min=1)
        e_kde = ks.sum(1) / ff.kde3
        dm = ((at[:, None] - mcs[None]) ** 2).sum(-1) * valid
        lhm = (tcc * torch.sqrt(dm.sum(2) / valid.sum(1).clamp(min=1))).sum(1)
        dst = (m[:, :3] + ctr - pocket).norm(dim=1)
        raw = torch.stack([vdw / L, ele / L, pmf / L, e_psp / L, hdb / L, hpc / L, e_kde / L,
                           torch.log(lhm / tcc.numel()), dst], 1)
        e = raw * a_para + b_para
        es.append(torch.cat([e, (e * w).sum(1, keepdim=True)], 1))
        n_c, hit = con.sum((1, 2)).double(), (con & ref).sum((1, 2)).double()
        fp, fn = n_c - hit, ref.sum().double() - hit
        tn = float(L) * P - hit - fp - fn
        den = torch.sqrt((hit + fp) * (hit + fn) * (tn + fp) * (tn + fn))
        cms.append(torch.where(den != 0, (hit * tn - fp * fn) / den.clamp(min=1e-300),
                               torch.zeros_like(den)))
        rmsd.append(((at - orig - ctr) ** 2).sum((1, 2)).div(L).sqrt())
    return {"e": torch.cat(es).cpu(), "cms": torch.cat(cms).cpu(), "rmsd": torch.cat(rmsd).cpu()}


def _exact_net(case, seed):
    theta, x, conf, t = _net_inputs(case, seed)
    H, E = case["hidden"], case["n_emb"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    th = torch.as_tensor(theta.astype(np.float64), device=dev).requires_grad_(True)
    sizes = [64 * H, H, H * H, H, H * H, H, H, 4, 32 * E]
    w1, b1, w2, b2, w3, b3, w4, b4, emb = torch.split(th, sizes)
    X = torch.as_tensor(x.astype(np.float64), device=dev)
    if E:
        c = torch.as_tensor(conf.astype(np.int64), device=dev)
        X = torch.cat([X[:, :7], emb.reshape(E, 32)[c], X[:, 39:]], 1)
    silu = torch.nn.functional.silu
    h = silu(X @ w1.reshape(64, H) + b1)
    h = silu(h @ w2.reshape(H, H) + b2)
    h = silu(h @ w3.reshape(H, H) + b3)
    y = h @ w4 + b4[0]
    if case["kind"] == "predict":
        return y.detach().cpu()
    loss = ((y - torch.as_tensor(t.astype(np.float64), device=dev)) ** 2).mean()
    (g,) = torch.autograd.grad(loss, th)
    return {"loss": float(loss.detach()), "grad": g.cpu()}


def exact(case, seed):
    """Energies and network values in 64 bits. Chains have none: a chain is a sequence of
    accept/reject decisions on rounded energies; a clustering returns whole numbers."""
    if case["kind"] == "score":
        return _exact_score(case, seed)
    if case["kind"] in ("train", "predict"):
        return _exact_net(case, seed)
    return None
