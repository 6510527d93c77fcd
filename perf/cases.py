"""Performance cases: the calls a user of this package makes, over the sizes they make them at.

``listed()`` are the fixed cases, ``draw(rng)`` gives further ones of the same ranges.  A case is
a dict of plain values; ``prepare(case, seed)`` makes its inputs and the objects a program keeps
(model, trainer, pair style), ``run(state)`` is one pass through the public entry points,
``work(case)`` the bytes and operations the pass cannot do without and ``exact(case, seed)`` the
same outputs from plain torch in 64 bits.

Kinds of case:

* ``dp_forward``  neighbor search + ``DP.forward`` on the padded lists, checks on: the model call
                  of the reference's inference and validation loops;
* ``dp_step``     occupied-slot search + ``DP.evaluate``: energy, forces, virial of one MD step;
* ``dp_ops``      ``calculateForce`` / ``calculateVirial`` and their backward, the operators an
                  unmodified reference model calls;
* ``nep_forward`` ``calculate_neighbor`` + ``NEP.forward``, checks on;
* ``nep_step``    ``calculate_neighbor`` + ``NEP.evaluate`` without host reads;
* ``nep_md``      ``SkinNeighbor`` compact lists + ``NEP.evaluate`` along a trajectory;
* ``dp_train``    one graphed force-loss training step of DP on a ragged batch;
* ``nep_ops``     ``calculateNepFeat`` / ``calculateNepMbFeat`` with first and second backward, the
                  descriptor operators of the reference's NEP training step;
* ``lammps``      one ``PairMATPL.compute`` from host arrays to host forces;
* ``replica_md``  ten velocity-Verlet steps of uneven DP replicas.

Boxes are amorphous: distinct sites of a cubic grid, displaced, at the densities of the benchmark
(0.05 - 0.085 atoms / A^3), elements grouped as the reference's images list them.
"""
import math

import numpy as np
import torch

from matpl_gb300 import data, dp, lammps, md, nep, nep_ops, ops, params, structures, train

DEV = "cuda"
RC, RMIN = 6.0, 0.5
STOP_LR = 3.51e-8      # the reference's final learning rate (stop_lr)


# ------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: 108-atom Cu cell in FP64, the reference's plain inference
        {"name": "dp_forward_cu108_f64", "kind": "dp_forward", "batch": 1, "natoms": 108,
         "ntypes": 1, "m": 100, "density": 0.085, "strain": 0.0, "precision": "float64"},
        # a validation pass over small strained two-element cells
        {"name": "dp_forward_16x96_mixed", "kind": "dp_forward", "batch": 16, "natoms": 96,
         "ntypes": 2, "m": 100, "density": 0.07, "strain": 0.03, "precision": "mixed"},
        # the benchmark box: 32,000 atoms, two elements, tensor-core form
        {"name": "dp_step_32k_mixed", "kind": "dp_step", "natoms": 32000, "ntypes": 2, "m": 150,
         "density": 0.05, "precision": "mixed"},
        # the plain FP32 form at an ordinary, odd size
        {"name": "dp_step_7k_f32", "kind": "dp_step", "natoms": 6913, "ntypes": 2, "m": 150,
         "density": 0.05, "precision": "float32"},
        # the force / virial operators of an unmodified model in FP64, forward and backward
        {"name": "dp_ops_2x3000_f64", "kind": "dp_ops", "batch": 2, "natoms": 3000, "ntypes": 2,
         "m": 100, "density": 0.05, "precision": "float64"},
        # a NEP validation batch of small cells (replicated boxes), wide model, FP64
        {"name": "nep_forward_6x72_f64", "kind": "nep_forward", "frames": 6, "natoms": 72,
         "ntypes": 2, "model": "wide", "density": 0.07, "precision": "float64"},
        # the NEP benchmark box: 100,000 atoms of four elements, exact lists every step
        {"name": "nep_step_100k_f32", "kind": "nep_step", "frames": 1, "natoms": 100000,
         "ntypes": 4, "model": "small", "density": 0.06, "precision": "float32"},
        # an MD caller with Verlet-skin lists
        {"name": "nep_md_50k", "kind": "nep_md", "natoms": 49999, "ntypes": 4, "model": "small",
         "density": 0.06},
        # the force-loss training batch: 64 configurations of 32 to 512 atoms
        {"name": "dp_train_64", "kind": "dp_train", "configs": 64, "nmin": 32, "nmax": 512,
         "density": 0.07, "strain": 0.03},
        # the descriptor part of a NEP training step: four frames, 20,000 atoms
        {"name": "nep_ops_20k_f32", "kind": "nep_ops", "frames": 4, "natoms": 5000, "ntypes": 4,
         "model": "small", "density": 0.06, "precision": "float32"},
        # the LAMMPS pair step of one rank: host lists in, host forces out
        {"name": "lammps_8k_mixed", "kind": "lammps", "natoms": 8191, "ntypes": 2, "m": 150,
         "density": 0.05, "precision": "mixed"},
        # many small replicas in one ragged array
        {"name": "replica_md_96", "kind": "replica_md", "replicas": 96, "nmin": 64, "nmax": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dp_forward", "dp_step", "dp_step", "dp_ops", "nep_forward", "nep_step",
                       "nep_step", "nep_md", "dp_train", "nep_ops", "lammps", "replica_md"])
    c = {"kind": kind}
    nt = rng.choice([1, 2, 2, 3])
    if kind == "dp_forward":
        prec = rng.choice(["float64", "float32", "mixed"])
        b = _log(rng, 1, 32)
        c.update(batch=b, natoms=_log(rng, 24, max(25, (1024 if prec == "float64" else 4096) // b)),
                 ntypes=nt, m=100, density=0.07, strain=rng.choice([0.0, 0.03]), precision=prec)
    elif kind == "dp_step":
        prec = rng.choice(["mixed", "mixed", "float32"])
        c.update(natoms=_log(rng, 500, 32000 if prec == "mixed" else 12000), ntypes=nt, m=150,
                 density=0.05, precision=prec)
    elif kind == "dp_ops":
        b = rng.choice([1, 2, 4])
        c.update(batch=b, natoms=_log(rng, 100, 4000 // b), ntypes=nt, m=100, density=0.05,
                 precision=rng.choice(["float64", "float32"]))
    elif kind == "nep_forward":
        f = _log(rng, 1, 16)
        c.update(frames=f, natoms=_log(rng, 16, max(17, 2000 // f)), ntypes=nt,
                 model=rng.choice(["small", "wide"]), density=0.07,
                 precision=rng.choice(["float64", "float32"]))
    elif kind == "nep_step":
        wide = rng.random() < 0.3
        c.update(frames=rng.choice([1, 1, 4]), natoms=_log(rng, 500, 4000 if wide else 25000),
                 ntypes=rng.choice([1, 2, 4]), model="wide" if wide else "small", density=0.06,
                 precision="float32")
    elif kind == "nep_md":
        c.update(natoms=_log(rng, 8000, 60000), ntypes=rng.choice([1, 2, 4]), model="small",
                 density=0.06)
    elif kind == "dp_train":
        c.update(configs=_log(rng, 1, 48), nmin=32, nmax=rng.choice([64, 200, 512]), density=0.07,
                 strain=0.03)
    elif kind == "nep_ops":
        wide, f = rng.random() < 0.3, rng.choice([1, 2, 5])
        prec = rng.choice(["float32", "float32", "float64"])
        most = 600 if prec == "float64" else 5000 if wide else 17500
        c.update(frames=f, natoms=_log(rng, 100, most // f), ntypes=rng.choice([1, 2, 4]),
                 model="wide" if wide else "small", density=0.06, precision=prec)
    elif kind == "lammps":
        c.update(natoms=_log(rng, 1200, 8000), ntypes=rng.choice([1, 2]), m=150, density=0.05,
                 precision=rng.choice(["mixed", "float32"]))
    else:
        c.update(replicas=_log(rng, 4, 90), nmin=64, nmax=rng.choice([256, 1024]))
    return c


# ------------------------------------------------------------------------- inputs, from the seed
def _box(n, density, nt, seed, strain=0.0):
    """(lattice [3,3] rows, frac [n,3], types [n]): n distinct sites of a cubic grid displaced by
    up to 15 % of the spacing, element t in a contiguous run, an optional symmetric strain."""
    rng = np.random.default_rng([seed, n])
    k = int(math.ceil(1.08 * n ** (1.0 / 3.0)))
    site = rng.permutation(k ** 3)[:n]
    g = np.stack([site // (k * k), site // k % k, site % k], 1).astype(np.float64)
    frac = np.mod((g + 0.5 + rng.uniform(-0.15, 0.15, (n, 3))) / k, 1.0)
    lat = np.eye(3) * (n / density) ** (1.0 / 3.0)
    if strain:
        e = rng.normal(0.0, strain, (3, 3))
        lat = lat @ (np.eye(3) + 0.5 * (e + e.T))
    types = np.sort(np.arange(n) % nt).astype(np.int64)
    return lat, frac, types


def _elements(nt):
    return [[29], [3, 14], [3, 14, 8], [3, 14, 8, 72]][nt - 1]


def _t(a, dtype=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dtype, device=DEV)


def _dp_params(nt, seed):
    """Random weights N(0, 1/fan_in) under the reference's names."""
    rng = np.random.default_rng([seed, 77])
    p = {}

    def put(name, v):
        p[name] = torch.tensor(v, dtype=torch.float64)
    for k in range(nt * nt):
        for l, (a, b) in enumerate([(1, 25), (25, 25), (25, 25)]):
            put(f"embedding_net.{k}.layers.{l}.weight", rng.normal(0, a ** -0.5, (a, b)))
            put(f"embedding_net.{k}.layers.{l}.bias", rng.normal(0, 0.1, (1, b)))
    for t in range(nt):
        for l, (a, b) in enumerate([(400, 50), (50, 50), (50, 50), (50, 1)]):
            put(f"fitting_net.{t}.layers.{l}.weight", rng.normal(0, a ** -0.5, (a, b)))
            put(f"fitting_net.{t}.layers.{l}.bias", rng.normal(0, 0.1, (1, b)))
            if l in (1, 2):
                put(f"fitting_net.{t}.layers.{l}.resnet_dt", rng.normal(0.1, 0.001, (1, b)))
    return p


def _dp_stats(nt, m, density):
    """davg, dstd [nt, 4] of the smoothed rows over all slots of a sample box."""
    lat, frac, types = _box(600, density, nt, 4242)
    i, j, v = _pairs(_t(lat), _t(frac), RC)
    rows = _env_rows(v)
    ti = _t(types, torch.int64)[i]
    avg, std = torch.zeros(nt, 4, dtype=torch.float64, device=DEV), None
    sq = torch.zeros_like(avg)
    avg.index_add_(0, ti, rows)
    sq.index_add_(0, ti, rows * rows)
    slots = _t(np.bincount(types, minlength=nt) * m * nt).reshape(-1, 1)
    avg, sq = avg / slots, sq / slots
    avg[:, 1:] = 0.0
    std = (sq - avg * avg).clamp_min(0).sqrt()
    std[:, 1:] = std[:, 1:].mean(1, keepdim=True)
    return avg.cpu(), std.clamp_min(1e-2).cpu()


def _dp_setup(nt, m, density, seed):
    cfg = params.DPConfig(atom_type=_elements(nt), maxNeighborNum=m, Rmax=RC, Rmin=RMIN)
    davg, dstd = _dp_stats(nt, m, density)
    tile = lambda a: a.unsqueeze(1).expand(nt, nt * m, 4).reshape(nt, -1).numpy()  # noqa: E731
    return cfg, _dp_params(nt, seed), tile(davg), tile(dstd)


_NEP_MODELS = {"small": dict(cutoff=(6.0, 4.0), n_max=(4, 4), basis_size=(8, 8), l_max=(4, 2, 1),
                             neuron=30),
               "wide": dict(cutoff=(6.0, 6.0), n_max=(4, 4), basis_size=(12, 12), l_max=(4, 2, 1),
                            neuron=100)}


def _nep_params(model, nt, density, seed):
    """Random parameters of the reference's initial distributions; q_scaler from a sample box."""
    mo = _NEP_MODELS[model]
    rng = np.random.default_rng([seed, 78])
    nr, na, kr, ka = mo["n_max"][0] + 1, mo["n_max"][1] + 1, mo["basis_size"][0] + 1, \
        mo["basis_size"][1] + 1
    F, H = nr + na * 6, mo["neuron"]
    c = lambda *s: torch.tensor(rng.random(s) - 0.5 + 0.1 * rng.normal(size=s))  # noqa: E731
    p = {"c_param_2": c(nt, nt, nr, kr), "c_param_3": c(nt, nt, na, ka)}
    for t in range(nt):
        pre = f"fitting_net.{t}.layers."
        p[pre + "0.weight"] = torch.tensor(rng.normal(size=(F, H)) / math.sqrt(F + H))
        p[pre + "0.bias"] = torch.tensor(rng.normal(size=(1, H)))
        p[pre + "1.weight"] = torch.tensor(rng.normal(size=(H, 1)) / math.sqrt(H + 1))
        p[pre + "1.bias"] = torch.tensor(-3.0 + rng.normal(size=(1, 1)))
    lat, frac, types = _box(500, density, nt, 4243)
    lists = [_with_r(*_pairs(_t(lat), _t(frac), rc)) for rc in mo["cutoff"]]
    q = _nep_features(mo, {k: v.to(DEV) for k, v in p.items()}, _t(types, torch.int64), lists)
    lo, hi = q.min(0).values, q.max(0).values
    for b in range(0, F, 5):
        lo[b:b + 5], hi[b:b + 5] = lo[b:b + 5].min(), hi[b:b + 5].max()
    p["q_scaler"] = (1.0 / (hi - lo)).cpu()
    return p


def _nep_config(model, nt):
    return nep.NepConfig(atom_type=_elements(nt), **_NEP_MODELS[model])


def _nep_boxes(case, seed):
    nf = case.get("frames", 1)
    return [_box(case["natoms"], case["density"], case["ntypes"], seed + 1000 * f)
            for f in range(nf)]


def _nep_inputs(case, seed):
    """The concatenated frames as the reference's loader hands them over, and the list sizes."""
    boxes = _nep_boxes(case, seed)
    mo = _NEP_MODELS[case["model"]]
    ex = [nep.expand_box(b[0], mo["cutoff"][0]) for b in boxes]
    s = {"num": _t([[len(b[1])] for b in boxes], torch.int64),
         "tm": _t(np.concatenate([b[2] for b in boxes]), torch.int64),
         "box": _t([e[0] for e in ex]), "orig": _t([e[1] for e in ex]),
         "cell": _t([e[2] for e in ex], torch.int64),
         "pos": _t(np.concatenate([b[1] @ b[0] for b in boxes])),
         "types": torch.arange(case["ntypes"], device=DEV), "rc": mo["cutoff"]}
    # list widths as a trainer fixes them for a data set: above the fullest atom of any frame
    s["max"] = tuple(8 * math.ceil((1.25 * _sphere(case["density"], rc) + 8) / 8)
                     for rc in s["rc"])
    return s


def _nep_lists(s, check=True):
    return ops.calculate_neighbor(s["num"], s["tm"], s["types"], s["box"], s["orig"], s["cell"],
                                  s["pos"], *s["rc"], *s["max"], True, check_overflow=check)


def _train_configs(case, seed):
    counts = np.random.default_rng([79, case["configs"]]).integers(
        case["nmin"], case["nmax"] + 1, case["configs"])
    out = []
    for k, n in enumerate(counts):
        lat, frac, _ = _box(int(n), case["density"], 1, seed + 1000 * k, case["strain"])
        types = (np.arange(n) >= n // 3).astype(np.int64)      # Hf:O 1:2
        out.append((lat, frac, types))
    return out


def _nmax(case):
    """Rows of LAMMPS' per-atom arrays: room above the local and ghost atoms."""
    n, d = case["natoms"], case["density"]
    return int(1.1 * n * (1 + 2 * (RC + 1.0) / (n / d) ** (1 / 3.0)) ** 3) + 256


def _ghost_system(case, seed):
    """One LAMMPS rank: local atoms, the periodic images within the neighbor cutoff (6 A + 1 A
    skin) as ghosts, and a full list per local atom in random order."""
    lat, frac, types = _box(case["natoms"], case["density"], case["ntypes"], seed)
    cut, n, L = RC + 1.0, case["natoms"], lat[0, 0]
    xs, own = [frac * L], [np.arange(n)]
    for a in range(-1, 2):
        for b in range(-1, 2):
            for c in range(-1, 2):
                if (a, b, c) != (0, 0, 0):
                    f = frac + np.array([a, b, c], dtype=np.float64)
                    keep = np.nonzero(((f >= -cut / L) & (f < 1.0 + cut / L)).all(1))[0]
                    xs.append(f[keep] * L)
                    own.append(keep)
    x, own = np.concatenate(xs), np.concatenate(own)
    xd = _t(x)
    rows, cols = [], []
    for a in range(0, n, 512):
        d = xd.unsqueeze(0) - xd[a:min(n, a + 512)].unsqueeze(1)
        i, j = torch.nonzero((d * d).sum(-1) < cut * cut, as_tuple=True)
        rows.append((i + a).cpu())
        cols.append(j.cpu())
    rows, cols = torch.cat(rows).numpy(), torch.cat(cols).numpy()
    rows, cols = rows[rows != cols], cols[rows != cols]
    order = np.random.default_rng([seed, 80]).permutation(len(rows))
    order = order[np.argsort(rows[order], kind="stable")]
    jflat = cols[order].astype(np.int32)
    numneigh = np.bincount(rows, minlength=n).astype(np.int32)
    start = np.concatenate([[0], np.cumsum(numneigh)[:-1]]).astype(np.uint64)
    return {"x": np.ascontiguousarray(x), "type": (types[own] + 1).astype(np.int32), "nlocal": n,
            "nghost": len(x) - n, "ilist": np.arange(n, dtype=np.int32), "numneigh": numneigh,
            "jflat": jflat, "rows": rows[order],
            "first": (np.uint64(jflat.ctypes.data) + np.uint64(4) * start).astype(np.uint64)}


def _replicas(case, seed):
    """FCC Cu replicas of 4 nx nx nz atoms, counts log-uniform, with 300 K velocities (A / fs)."""
    rng, sizes = np.random.default_rng([seed, 81]), np.random.default_rng([81, case["replicas"]])
    out, vel = [], []
    for _ in range(case["replicas"]):
        cells = math.exp(sizes.uniform(math.log(case["nmin"]), math.log(case["nmax"]))) / 4.0
        nx = max(2, int(round(cells ** (1.0 / 3.0))))
        nz = max(2, int(round(cells / (nx * nx))))
        base = np.array([[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]])
        cell = np.stack(np.meshgrid(np.arange(nx), np.arange(nx), np.arange(nz),
                                    indexing="ij"), -1).reshape(-1, 1, 3)
        lat = np.diag([3.615 * nx, 3.615 * nx, 3.615 * nz])
        cart = (cell + base).reshape(-1, 3) * 3.615
        frac = np.mod((cart + rng.normal(0, 0.05, cart.shape)) / np.diag(lat), 1.0)
        out.append((lat, frac))
        v = rng.normal(0, math.sqrt(0.025852 / (63.546 * md.AMU_A2_FS2_EV)), cart.shape)
        vel.append(v - v.mean(0))
    return out, np.concatenate(vel)


def _ops_inputs(case, seed):
    """Padded 0-based lists with random dE, Ri_d (zero in empty slots) and incoming gradients."""
    dt = getattr(torch, case["precision"])
    B, N, S, m = case["batch"], case["natoms"], case["ntypes"] * case["m"], case["m"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    nl = torch.full((B, N, S), -1, dtype=torch.int32, device=DEV)
    rij = torch.zeros(B, N, S, 3, dtype=dt, device=DEV)
    for b in range(B):
        lat, frac, types = _box(N, case["density"], case["ntypes"], seed + 1000 * b)
        i, j, v = _pairs(_t(lat), _t(frac), RC)
        tj = _t(types, torch.int64)[j]
        order = torch.argsort((i * case["ntypes"] + tj) * N + j, stable=True)
        i, j, v, tj = i[order], j[order], v[order], tj[order]
        key = i * case["ntypes"] + tj
        first = torch.searchsorted(key, torch.arange(N * case["ntypes"], device=DEV))
        slot = tj * m + torch.arange(len(key), device=DEV) - first[key]
        nl[b, i, slot] = j.to(torch.int32)
        rij[b, i, slot] = v.to(dt)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=dt)  # noqa: E731
    has = (nl >= 0).unsqueeze(-1)
    rid = (rn(B, N, S, 12) * has).reshape(B, N, 4 * S, 3)
    return {"nl": nl.unsqueeze(2), "rij": rij, "rid": rid, "dE": rn(B, N, S, 4).reshape(B, N, 1, 4 * S),
            "Fc": rn(B, N, 3), "gF": rn(B, N, 3), "gV": rn(B, 9)}


def _nep_ops_inputs(case, seed):
    """Padded lists (-1 empty) with rows (r, x, y, z), G = dE/dq, and the gradients that a loss
    sends to q (U) and to dE/d(r, x, y, z) (H, zero in empty slots)."""
    dt, mo = getattr(torch, case["precision"]), _NEP_MODELS[case["model"]]
    boxes = _nep_boxes(case, seed)
    n = sum(len(b[1]) for b in boxes)
    g = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    prm = _nep_params(case["model"], case["ntypes"], case["density"], seed)
    F = prm["q_scaler"].numel()
    qs = prm["q_scaler"].to(DEV)
    s = {"tm": _t(np.concatenate([b[2] for b in boxes]), torch.int64), "mo": mo,
         "c2": prm["c_param_2"].to(DEV, dt), "c3": prm["c_param_3"].to(DEV, dt),
         "G": (qs * rn(n, F)).to(dt), "U": (qs * rn(n, F)).to(dt), "NL": [], "d": [], "H": []}
    for rc in mo["cutoff"]:
        i, j, v = _frames_pairs(boxes, rc)
        order = torch.argsort(i, stable=True)
        i, j, v = i[order], j[order], v[order]
        slot = torch.arange(len(i), device=DEV) - torch.searchsorted(
            i, torch.arange(n, device=DEV))[i]
        width = 8 * math.ceil((1.25 * _sphere(case["density"], rc) + 8) / 8)
        nl = torch.full((n, width), -1, dtype=torch.int64, device=DEV)
        nl[i, slot] = j
        d = torch.zeros(n, width, 4, dtype=torch.float64, device=DEV)
        d[i, slot] = torch.cat([v.norm(dim=1, keepdim=True), v], 1)
        s["NL"].append(nl)
        s["d"].append(d.to(dt))
        s["H"].append((rn(n, width, 4) * (nl >= 0).unsqueeze(2)).to(dt))
    return s


def _trajectory(case, seed):
    """64 positions along a closed path: every atom swings by up to 0.9 A about its site."""
    lat, frac, types = _box(case["natoms"], case["density"], case["ntypes"], seed)
    rng = np.random.default_rng([seed, 82])
    amp = rng.normal(0, 0.2, frac.shape)
    amp *= np.minimum(1.0, 0.9 / np.linalg.norm(amp, axis=1, keepdims=True))
    return lat, types, frac @ lat, amp


# ---------------------------------------------------------------------------------- preparation
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("dp_forward", "dp_step"):
        B = case.get("batch", 1)
        boxes = [_box(case["natoms"], case["density"], case["ntypes"], seed + 1000 * b,
                      case.get("strain", 0.0)) for b in range(B)]
        cfg, prm, davg, dstd = _dp_setup(case["ntypes"], case["m"], case["density"], seed)
        model = dp.DP(cfg, prm, davg, dstd, precision=case["precision"], device=DEV,
                      check_errors=kind == "dp_forward")
        return {"kind": kind, "cfg": cfg, "model": model,
                "types": _t(boxes[0][2], torch.int32), "frac": _t([b[1] for b in boxes]),
                "lat": _t([b[0] for b in boxes]), "present": model.present_types(cfg.atom_type),
                "list_dtype": torch.float64 if kind == "dp_forward" else model.dtype}
    if kind == "dp_ops":
        s = _ops_inputs(case, seed)
        s["dE"].requires_grad_()
        return {"kind": kind, **s}
    if kind in ("nep_forward", "nep_step"):
        s = _nep_inputs(case, seed)
        prm = _nep_params(case["model"], case["ntypes"], case["density"], seed)
        s["model"] = nep.NEP(_nep_config(case["model"], case["ntypes"]), prm, case["precision"],
                             device=DEV, check_errors=kind == "nep_forward")
        return {"kind": kind, **s}
    if kind == "nep_md":
        s = _nep_inputs(case, seed)
        _, _, x0, amp = _trajectory(case, seed)
        x0, amp = _t(x0), _t(amp)
        s["path"] = [(x0 + amp * math.sin(2 * math.pi * k / 64)).contiguous() for k in range(64)]
        s["at"] = 0
        mr, ma = s["max"]
        s["lists"] = ops.SkinNeighbor(s["num"], s["box"], s["orig"], s["cell"], s["path"][0],
                                      *s["rc"], mr + 24, ma + 16, skin=1.0, compact=True)
        prm = _nep_params(case["model"], case["ntypes"], case["density"], seed)
        s["model"] = nep.NEP(_nep_config(case["model"], case["ntypes"]), prm, "float32",
                             device=DEV, check_errors=False)
        return {"kind": kind, **s}
    if kind == "dp_train":
        boxes = _train_configs(case, seed)
        cfg, prm, davg, dstd = _dp_setup(2, 100, case["density"], seed)
        cfg.atom_type = [72, 8]
        E, F = _train_labels(case, seed, boxes, davg, dstd)
        images = [structures.Structure(b[0], b[1], b[2].astype(np.int32), [72, 8]) for b in boxes]
        batch = data.ragged_batch(cfg, images, device=DEV, energies=E, forces=F,
                                  out_dtype=torch.float32)
        model = train.DPTrainModel(cfg, prm, davg, dstd, dtype=torch.float32, device=DEV)
        opt = torch.optim.Adam(model.parameters(), lr=STOP_LR, capturable=True, fused=True)
        tr = train.GraphedTrainer(train.FusedTrainer(model, "mixed"), opt)
        tr.step(batch)                 # captures the graph, once per batch shape
        return {"kind": kind, "trainer": tr, "batch": batch, "model": model}
    if kind == "nep_ops":
        s = _nep_ops_inputs(case, seed)
        for x in (s["c2"], s["c3"], s["G"], *s["d"]):
            x.requires_grad_()
        nep_ops.set_check_errors(False)        # as a training loop does
        return {"kind": kind, **s}
    if kind == "lammps":
        s = _ghost_system(case, seed)
        cfg, prm, davg, dstd = _dp_setup(case["ntypes"], case["m"], case["density"], seed)
        model = dp.DP(cfg, prm, davg, dstd, precision=case["precision"], device=DEV)
        pair = lammps.PairMATPL(model, cfg.atom_type)
        s["f"] = np.zeros((_nmax(case), 3))
        return {"kind": kind, "pair": pair, **s}
    reps, vel = _replicas(case, seed)
    cfg, prm, davg, dstd = _dp_setup(1, 100, 0.085, seed)
    sts = [structures.Structure(lat, frac, np.zeros(len(frac), dtype=np.int32), [29])
           for lat, frac in reps]
    sim = md.ReplicaMD(cfg, prm, davg, dstd, sts, [63.546], dt_fs=1.0, precision="mixed",
                       device=DEV, skin=1.0, steps_per_graph=10)
    sim.v.copy_(_t(vel))
    sim.capture()
    return {"kind": kind, "sim": sim}


# ---------------------------------------------------------------------------------- one pass
def run(s):
    kind = s["kind"]
    if kind == "dp_forward":
        ln, idr = ops.find_neighbore(s["types"], s["frac"], s["lat"], s["cfg"].ntypes,
                                     s["cfg"].maxNeighborNum, RC, RC, out_dtype=s["list_dtype"])
        E, Ei, F, _, V = s["model"](ln, s["types"], s["cfg"].atom_type, idr, 0)
        return {"list": ln, "dr": idr, "E": E, "Ei": Ei, "F": F, "V": V}
    if kind == "dp_step":
        ln, idr, nn = ops.find_neighbore(s["types"], s["frac"], s["lat"], s["cfg"].ntypes,
                                         s["cfg"].maxNeighborNum, RC, RC,
                                         out_dtype=s["list_dtype"], check_overflow=False,
                                         occupied_only=True)
        r = s["model"].evaluate(ln, s["types"], s["present"], idr, 0, num_neigh=nn)
        return {"num": nn, "E": r["Etot"], "Ei": r["Ei_atom"], "F": r["Force"], "V": r["Virial"]}
    if kind == "dp_ops":
        F = ops.calculateForce(s["nl"], s["dE"], s["rid"], s["Fc"], 0)[0]
        V, av = ops.calculateVirial(s["nl"], s["dE"], s["rij"], s["rid"], 0)
        g, = torch.autograd.grad([F, V], [s["dE"]], [s["gF"], s["gV"]])
        return {"F": F, "V": V, "atom_virial": av, "grad": g}
    if kind == "nep_forward":
        a, b, la, lb, ra, rb = _nep_lists(s)
        E, Ei, F, _, V = s["model"](a, la, ra, b, lb, rb, s["num"], s["tm"])
        return {"lists": [a, b, la, lb, ra, rb], "E": E, "Ei": Ei, "F": F, "V": V}
    if kind == "nep_step":
        a, b, la, lb, ra, rb = _nep_lists(s, check=False)
        r = s["model"].evaluate(a, la, ra, b, lb, rb, s["num"], s["tm"])
        return {"lists": [a, b, la, lb, ra, rb], "E": r["Etot"], "Ei": r["Ei"], "F": r["Force"],
                "V": r["Virial"]}
    if kind == "nep_md":
        s["at"] = (s["at"] + 1) % len(s["path"])
        a, b, la, lb, ra, rb = s["lists"].lists(s["path"][s["at"]])
        r = s["model"].evaluate(a, la, ra, b, lb, rb, s["num"], s["tm"])
        return {"num": [a, b], "E": r["Etot"], "Ei": r["Ei"], "F": r["Force"], "V": r["Virial"]}
    if kind == "dp_train":
        loss = s["trainer"].step(s["batch"])
        return {"loss": loss, "grad": {n: s["model"].param(n).grad for n in s["model"].names}}
    if kind == "nep_ops":
        (nr, na), (dr, da), mo = s["NL"], s["d"], s["mo"]
        q = torch.cat([
            ops.calculateNepFeat(s["c2"], dr, nr, s["tm"], s["G"], mo["cutoff"][0], 30)[0],
            ops.calculateNepMbFeat(s["c3"], da, na, s["tm"], s["G"], 5, *mo["l_max"],
                                   mo["cutoff"][1])[0]], 1)
        dE = torch.autograd.grad(q, [dr, da], s["G"], create_graph=True)
        grads = torch.autograd.grad([q, *dE], [s["c2"], s["c3"], s["G"]], [s["U"], *s["H"]])
        return {"q": q, "dE": list(dE), "grad": list(grads)}
    if kind == "lammps":
        r = s["pair"].compute(s["x"], s["type"], s["nlocal"], s["nghost"], s["ilist"],
                              s["numneigh"], s["first"], eflag_atom=True, f_out=s["f"])
        return {"f": r["f"], "eng": r["eng"], "virial": r["virial"], "eatom": r["eatom"],
                "min_rsq": r["min_rsq"]}
    s["sim"].step(10)
    return {"x": s["sim"].x, "v": s["sim"].v, "F": s["sim"].out["Force"]}


# ---------------------------------------------------------------------------------- least work
def _sphere(density, rc):
    return density * 4.0 / 3.0 * math.pi * rc ** 3


# per pair / atom of DP: embedding forward + adjoint, fitting forward + adjoint
_DP_PAIR, _DP_ATOM = 5742, 109800


def _nep_flops(mo, density):
    n, na, k, ka = (mo["n_max"][0] + 1, mo["n_max"][1] + 1, mo["basis_size"][0] + 1,
                    mo["basis_size"][1] + 1)
    F, H = n + 6 * na, mo["neuron"]
    return _sphere(density, mo["cutoff"][0]) * (6 * k + 4 * n * k + 2 * n + 24) + \
        _sphere(density, mo["cutoff"][1]) * (6 * ka + 4 * na * ka + 144 * na + 302) + \
        318 * na + 4 * F * H + 6 * H + F


def work(case):
    kind, d = case["kind"], case.get("density", 0.085)
    if kind == "dp_forward":
        n, size = case["batch"] * case["natoms"], 8 if case["precision"] == "float64" else 4
        S = case["ntypes"] * case["m"]
        return {"bytes": n * (24 + 4 + S * 36 + 4 * size),
                "flops": n * (_sphere(d, RC) * _DP_PAIR + _DP_ATOM)}
    if kind == "dp_step":
        n = case["natoms"]
        return {"bytes": n * (24 + 4 + 4 * case["ntypes"] + 16),
                "flops": n * (_sphere(d, RC) * _DP_PAIR + _DP_ATOM)}
    if kind == "dp_ops":
        n, e, p = case["batch"] * case["natoms"], 8 if case["precision"] == "float64" else 4, \
            _sphere(d, RC)
        S = case["ntypes"] * case["m"]
        return {"bytes": n * (S * (4 + 4 * e) + p * (4 + 12 + 3) * e + (3 * 3 + 9) * e),
                "flops": n * p * 120.0}
    if kind in ("nep_forward", "nep_step"):
        mo, n = _NEP_MODELS[case["model"]], case.get("frames", 1) * case["natoms"]
        e = 8 if case["precision"] == "float64" else 4
        p = sum(_sphere(d, rc) for rc in mo["cutoff"])
        return {"bytes": n * (24 + 8 + 16 + 40 * p + 4 * e), "flops": n * _nep_flops(mo, d)}
    if kind == "nep_md":
        mo, n = _NEP_MODELS[case["model"]], case["natoms"]
        return {"bytes": n * (24 + 8 + 8 + 16), "flops": n * _nep_flops(mo, d)}
    if kind == "dp_train":
        n, p = case["configs"] * (case["nmin"] + case["nmax"]) / 2, _sphere(d, RC)
        return {"bytes": n * (200 * 4 + p * 16 + 16) + 4e5,
                "flops": n * (p * (_DP_PAIR + 6 * 2750) + 3 * _DP_ATOM)}
    if kind == "nep_ops":
        mo, n = _NEP_MODELS[case["model"]], case["frames"] * case["natoms"]
        e, F = 8 if case["precision"] == "float64" else 4, 35
        p = sum(_sphere(d, rc) for rc in mo["cutoff"])
        w = sum(8 * math.ceil((1.25 * _sphere(d, rc) + 8) / 8) for rc in mo["cutoff"])
        return {"bytes": n * (p * (8 + 8 * e) + w * 4 * e + 4 * F * e + 8),
                "flops": 3.0 * n * _nep_flops(mo, d)}
    if kind == "lammps":
        n = case["natoms"]
        nall = n * (1 + 14 / (n / d) ** (1 / 3.0)) ** 3
        return {"bytes": nall * (24 + 4 + 24) + n * (4 * _sphere(d, RC + 1) + 24),
                "flops": n * (_sphere(d, RC) * _DP_PAIR + _DP_ATOM)}
    n = 10 * case["replicas"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    return {"bytes": n * (3 * 24 * 2 + 16), "flops": n * (_sphere(d, RC) * _DP_PAIR + _DP_ATOM)}


# ---------------------------------------------------------------- 64-bit values, plain torch
def _pairs(lat, frac, rc):
    """(i, j, r_j - r_i) of every pair within rc: nearest images where every cell vector is at
    least 2 rc long, else every periodic image."""
    n = frac.shape[0]
    if bool((lat.norm(dim=1) >= 2 * rc).all()):
        shifts = torch.zeros(1, 3, dtype=frac.dtype, device=frac.device)
    else:
        inv = torch.linalg.inv(lat)
        k = [int(math.ceil(rc * float(inv[:, a].norm()) + 0.5)) for a in range(3)]
        shifts = torch.cartesian_prod(*(torch.arange(-q, q + 1, device=frac.device) for q in k))
        shifts = shifts.to(frac.dtype)
    I, J, V = [], [], []
    step = max(1, int(2.5e7) // (n * len(shifts)))
    for a in range(0, n, step):
        f = frac.unsqueeze(0) - frac[a:a + step].unsqueeze(1)
        f = (f - torch.round(f)).unsqueeze(2) + shifts
        v = f @ lat
        r2 = (v * v).sum(-1)
        i, j, k = torch.nonzero((r2 < rc * rc) & (r2 > 1e-8), as_tuple=True)
        I.append(i + a)
        J.append(j)
        V.append(v[i, j, k])
    return torch.cat(I), torch.cat(J), torch.cat(V)


def _env_rows(v):
    """(s, s x / r, s y / r, s z / r) of each pair vector."""
    r = v.norm(dim=1, keepdim=True)
    u = (r - RMIN) / (RC - RMIN)
    poly = u ** 3 * (-6 * u ** 2 + 15 * u - 10) + 1
    s = torch.where(r < RMIN, 1 / r, torch.where(r < RC, poly / r, torch.zeros_like(r)))
    return torch.cat([s, s * v / r], 1)


def _layer_net(p, pre, x, nlayers):
    for l in range(nlayers):
        w = p[f"{pre}{l}.weight"]
        h = torch.tanh(x @ w + p[f"{pre}{l}.bias"])
        dt = p.get(f"{pre}{l}.resnet_dt")
        x = (h if dt is None else h * dt) + (x if w.shape[0] == w.shape[1] else 0.0)
    return x


def _dp_energies(p, davg, dstd, types, m, i, j, v):
    """Ei [N] of the DP model from pairs (i, j, v), differentiable in v and the parameters.
    davg, dstd [nt, 4]; every type block of an atom has m slots, the empty ones hold the
    normalised zero row."""
    nt, n = davg.shape[0], types.shape[0]
    ti, tj = types[i], types[j]
    R = (_env_rows(v) - davg[ti]) / dstd[ti]
    A = torch.zeros(n, 100, dtype=v.dtype, device=v.device)
    count = torch.zeros(n, nt, dtype=v.dtype, device=v.device)
    count.index_put_((i, tj), torch.ones(len(i), dtype=v.dtype, device=v.device), accumulate=True)
    for a in range(nt):
        mine = types == a
        pad = -davg[a] / dstd[a]
        for b in range(nt):
            pre = f"embedding_net.{a * nt + b}.layers."
            k = torch.nonzero((ti == a) & (tj == b)).flatten()
            G = _layer_net(p, pre, R[k, :1], 3)
            A = A.index_add(0, i[k], (R[k].unsqueeze(2) * G.unsqueeze(1)).reshape(-1, 100))
            row = (pad.reshape(4, 1) * _layer_net(p, pre, pad[:1].reshape(1, 1), 3)).reshape(1, 100)
            A = A + ((m - count[:, b]) * mine).unsqueeze(1) * row
    A = A.reshape(n, 4, 25) / (m * nt)
    D = (A.transpose(1, 2) @ A[:, :, :16]).reshape(n, 400)
    E = torch.zeros(n, dtype=v.dtype, device=v.device)
    for a in range(nt):
        k = torch.nonzero(types == a).flatten()
        pre = f"fitting_net.{a}.layers."
        x = _layer_net(p, pre, D[k], 3)
        E = E.index_add(0, k, (x @ p[pre + "3.weight"] + p[pre + "3.bias"]).flatten())
    return E


def _forces(E, i, j, v, n, create_graph=False):
    """(forces [n,3], -dE/dv) of the total energy."""
    f = -torch.autograd.grad(E.sum(), v, create_graph=create_graph)[0]
    F = torch.zeros(n, 3, dtype=v.dtype, device=v.device).index_add(0, j, f).index_add(0, i, -f)
    return F, f


def _dev(p):
    return {k: x.to(DEV, torch.float64) for k, x in p.items()}


def _stat4(a, nt):
    return torch.as_tensor(a).reshape(nt, -1, 4)[:, 0].to(DEV, torch.float64)


def _frames_pairs(boxes, rc):
    """Pairs of every box in one numbering of all atoms."""
    I, J, V, off = [], [], [], 0
    for lat, frac, _ in boxes:
        i, j, v = _pairs(_t(lat), _t(frac), rc)
        I.append(i + off)
        J.append(j + off)
        V.append(v)
        off += len(frac)
    return torch.cat(I), torch.cat(J), torch.cat(V)


def _frame_sum(x, boxes):
    which = _t(np.repeat(np.arange(len(boxes)), [len(b[1]) for b in boxes]), torch.int64)
    out = torch.zeros((len(boxes),) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    return out.index_add(0, which, x)


def _virial(f, v, i, n, boxes):
    per_atom = torch.zeros(n, 9, dtype=f.dtype, device=f.device)
    per_atom = per_atom.index_add(0, i, (f.unsqueeze(2) * v.unsqueeze(1)).reshape(-1, 9))
    return _frame_sum(per_atom, boxes)


def _dp_boxes(p, davg, dstd, m, boxes, create_graph=False):
    types = _t(np.concatenate([b[2] for b in boxes]), torch.int64)
    i, j, v = _frames_pairs(boxes, RC)
    v = v.requires_grad_()
    Ei = _dp_energies(p, davg, dstd, types, m, i, j, v)
    F, f = _forces(Ei, i, j, v, len(types), create_graph)
    return Ei, F, f, v, i


def _train_labels(case, seed, boxes, davg, dstd):
    """Energies and forces of a teacher net plus N(0, 0.01) noise."""
    p = _dev(_dp_params(2, seed + 500))
    Ei, F, _, _, _ = _dp_boxes(p, _stat4(davg, 2), _stat4(dstd, 2), 100, boxes)
    rng = np.random.default_rng([seed, 83])
    E = _frame_sum(Ei.detach(), boxes).cpu().numpy()
    F = F.detach().cpu().numpy()
    cut = np.cumsum([len(b[1]) for b in boxes])[:-1]
    return E + rng.normal(0, 0.01, E.shape), np.split(F + rng.normal(0, 0.01, F.shape), cut)


# NEP descriptor constants: 3-body weights of the 24 harmonics (m > 0 doubled), 4- and 5-body
_C3B = [0.238732414637843, 0.238732414637843, 0.238732414637843, 0.099471839432435,
        1.1936620731892151, 1.1936620731892151, 0.2984155182973038, 0.2984155182973038,
        0.139260575205408, 0.20889086280811264, 0.20889086280811264, 2.088908628081126,
        2.088908628081126, 0.34815143801352105, 0.34815143801352105, 0.01119058193614889,
        0.44762327744595565, 0.44762327744595565, 0.22381163872297782, 0.22381163872297782,
        3.1333629421216895, 3.1333629421216895, 0.3916703677652112, 0.3916703677652112]
_C4B = [-0.007499480826664, -0.134990654879954, 0.067495327439977, 0.404971964639861,
        -0.809943929279723]
_C5B = [0.026596810706114, 0.053193621412227, 0.026596810706114]


def _chebyshev(r, nk, rc):
    x = 2.0 * (r / rc - 1.0) ** 2 - 1.0
    fc = 0.5 + 0.5 * torch.cos(math.pi * r / rc)
    t = [torch.ones_like(r), x]
    for _ in range(2, nk):
        t.append(2.0 * x * t[-1] - t[-2])
    return torch.stack([0.5 * (a + 1.0) * fc for a in t[:nk]], 1)


def _harmonics(u):
    x, y, z = u.unbind(1)
    z2, d = z * z, x * x - y * y
    return torch.stack([
        z, x, y, 3 * z2 - 1, x * z, y * z, d, 2 * x * y,
        (5 * z2 - 3) * z, (5 * z2 - 1) * x, (5 * z2 - 1) * y, d * z, 2 * x * y * z,
        (x * x - 3 * y * y) * x, (3 * x * x - y * y) * y,
        (35 * z2 - 30) * z2 + 3, (7 * z2 - 3) * x * z, (7 * z2 - 3) * y * z, (7 * z2 - 1) * d,
        (7 * z2 - 1) * 2 * x * y, (x * x - 3 * y * y) * x * z, (3 * x * x - y * y) * y * z,
        d * d - 4 * x * x * y * y, 4 * x * y * d], 1)


def _with_r(i, j, v):
    return i, j, v.norm(dim=1), v


def _nep_features(mo, p, types, lists):
    """[N, F] descriptor from the radial and the angular pairs (i, j, r, xyz)."""
    n, out = types.shape[0], []
    for (i, j, r, v), c, nk, rc, angular in zip(
            lists, (p["c_param_2"], p["c_param_3"]), [b + 1 for b in mo["basis_size"]],
            mo["cutoff"], (False, True)):
        g = (c[types[i], types[j]] @ _chebyshev(r, nk, rc).unsqueeze(2)).squeeze(2)   # [P, n]
        if not angular:
            out.append(torch.zeros(n, g.shape[1], dtype=g.dtype, device=g.device).index_add(0, i, g))
            continue
        na = g.shape[1]
        b = _harmonics(v / r.unsqueeze(1))
        s = torch.zeros(n, na * 24, dtype=g.dtype, device=g.device)
        s = s.index_add(0, i, (g.unsqueeze(2) * b.unsqueeze(1)).reshape(-1, na * 24))
        s = s.reshape(n, na, 24)
        sq = s * s
        w = sq * torch.tensor(_C3B, dtype=s.dtype, device=s.device)
        out += [w[..., a:e].sum(-1) for a, e in ((0, 3), (3, 8), (8, 15), (15, 24))]
        s3, s4, s5, s6, s7 = (s[..., k] for k in range(3, 8))
        out.append(_C4B[0] * s3 ** 3 + _C4B[1] * s3 * (s4 * s4 + s5 * s5)
                   + _C4B[2] * s3 * (s6 * s6 + s7 * s7) + _C4B[3] * s6 * (s5 * s5 - s4 * s4)
                   + _C4B[4] * s4 * s5 * s7)
        a0, a12 = sq[..., 0], sq[..., 1] + sq[..., 2]
        out.append(_C5B[0] * a0 * a0 + _C5B[1] * a0 * a12 + _C5B[2] * a12 * a12)
    return torch.cat(out, 1)


def _nep_boxes_eval(mo, p, boxes, create_graph=False):
    """(E [B], Ei, F, V [B, 9]) of the NEP model over the frames."""
    types = _t(np.concatenate([b[2] for b in boxes]), torch.int64)
    n = len(types)
    lists = [_frames_pairs(boxes, rc) for rc in mo["cutoff"]]
    lists = [(i, j, v.requires_grad_()) for i, j, v in lists]
    q = _nep_features(mo, p, types, [_with_r(*a) for a in lists]) * p["q_scaler"]
    E = torch.zeros(n, dtype=q.dtype, device=q.device)
    for t in range(p["c_param_2"].shape[0]):
        k = torch.nonzero(types == t).flatten()
        pre = f"fitting_net.{t}.layers."
        h = torch.tanh(q[k] @ p[pre + "0.weight"] + p[pre + "0.bias"])
        E = E.index_add(0, k, (h @ p[pre + "1.weight"] + p[pre + "1.bias"]).flatten())
    F, V = 0.0, 0.0
    grads = torch.autograd.grad(E.sum(), [v for _, _, v in lists], create_graph=create_graph)
    for (i, j, v), g in zip(lists, grads):
        F = F + torch.zeros(n, 3, dtype=q.dtype, device=q.device).index_add(0, i, g).index_add(
            0, j, -g)
        V = V + _virial(-g, v, i, n, boxes)
    return _frame_sum(E, boxes), E, F, V


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dp_forward", "dp_step"):
        boxes = [_box(case["natoms"], case["density"], case["ntypes"], seed + 1000 * b,
                      case.get("strain", 0.0)) for b in range(case.get("batch", 1))]
        B, N, nt = len(boxes), case["natoms"], case["ntypes"]
        davg, dstd = (x.to(DEV) for x in _dp_stats(nt, case["m"], case["density"]))
        Ei, F, f, v, i = _dp_boxes(_dev(_dp_params(nt, seed)), davg, dstd, case["m"], boxes)
        E, V = _frame_sum(Ei.detach(), boxes), _virial(f, v.detach(), i, B * N, boxes)
        Ei, F = Ei.detach().reshape(B, N), F.reshape(B, N, 3)
        if kind == "dp_forward":
            return {"list": None, "dr": None, "E": E.reshape(B, 1), "Ei": Ei, "F": F, "V": V}
        return {"num": None, "E": E, "Ei": Ei, "F": F, "V": V}
    if kind == "dp_ops":
        s = {k: x.double() if x.is_floating_point() else x for k, x in _ops_inputs(case, seed).items()}
        B, N, S = case["batch"], case["natoms"], s["rij"].shape[2]
        rid, nl = s["rid"].reshape(B, N, S, 4, 3), s["nl"].reshape(B, N, S).long()
        f = (s["dE"].reshape(B, N, S, 4, 1) * rid).sum(3)
        b, i, k = torch.nonzero(nl >= 0, as_tuple=True)
        at = b * N + nl[b, i, k]
        F = s["Fc"].reshape(-1, 3).index_add(0, at, f[b, i, k])
        av = (f[b, i, k].unsqueeze(2) * s["rij"][b, i, k].unsqueeze(1)).reshape(-1, 9)
        av = torch.zeros(B * N, 9, dtype=torch.float64, device=DEV).index_add(0, at, av)
        g = torch.zeros(B, N, S, 4, dtype=torch.float64, device=DEV)
        w = s["gF"].reshape(-1, 3)[at] - s["gF"][b, i]
        w = w + (s["gV"].reshape(B, 3, 3)[b] @ s["rij"][b, i, k].unsqueeze(2)).squeeze(2)
        g[b, i, k] = (rid[b, i, k] @ w.unsqueeze(2)).squeeze(2)
        av = av.reshape(B, N, 9)
        return {"F": F.reshape(B, N, 3), "V": av.sum(1), "atom_virial": av,
                "grad": g.reshape(B, N, 1, 4 * S)}
    if kind in ("nep_forward", "nep_step"):
        p = _dev(_nep_params(case["model"], case["ntypes"], case["density"], seed))
        E, Ei, F, V = _nep_boxes_eval(_NEP_MODELS[case["model"]], p, _nep_boxes(case, seed))
        E = E.reshape(-1, 1) if kind == "nep_forward" else E
        return {"lists": [None] * 6, "E": E.detach(), "Ei": Ei.detach(), "F": F, "V": V.detach()}
    if kind == "nep_md":
        lat, types, x0, amp = _trajectory(case, seed)
        x = x0 + amp * math.sin(2 * math.pi / 64)
        p = _dev(_nep_params(case["model"], case["ntypes"], case["density"], seed))
        E, Ei, F, V = _nep_boxes_eval(_NEP_MODELS[case["model"]], p,
                                      [(lat, x @ np.linalg.inv(lat), types)])
        return {"num": [None, None], "E": E.detach(), "Ei": Ei.detach(), "F": F, "V": V.detach()}
    if kind == "dp_train":
        boxes = _train_configs(case, seed)
        davg, dstd = (x.to(DEV) for x in _dp_stats(2, 100, case["density"]))
        E_l, F_l = _train_labels(case, seed, boxes, davg.cpu(), dstd.cpu())
        p = {k: x.requires_grad_() for k, x in _dev(_dp_params(2, seed)).items()}
        Ei, F, _, _, _ = _dp_boxes(p, davg, dstd, 100, boxes, create_graph=True)
        loss = (_frame_sum(Ei, boxes) - _t(E_l)).square().mean() + \
            (F - _t(np.concatenate(F_l))).square().mean()
        loss.backward()
        return {"loss": loss.detach(), "grad": {k: x.grad for k, x in p.items()}}
    if kind == "nep_ops":
        s = _nep_ops_inputs(case, seed)
        c2, c3, G = (s[k].double().requires_grad_() for k in ("c2", "c3", "G"))
        ds, lists = [x.double().requires_grad_() for x in s["d"]], []
        for nl, d in zip(s["NL"], ds):
            i, k = torch.nonzero(nl >= 0, as_tuple=True)
            rows = d[i, k]
            lists.append((i, nl[i, k], rows[:, 0], rows[:, 1:]))
        q = _nep_features(s["mo"], {"c_param_2": c2, "c_param_3": c3}, s["tm"], lists)
        dE = torch.autograd.grad(q, ds, G, create_graph=True)
        grads = torch.autograd.grad([q, *dE], [c2, c3, G],
                                    [s["U"].double(), *(x.double() for x in s["H"])])
        return {"q": q.detach(), "dE": [x.detach() for x in dE], "grad": list(grads)}
    if kind == "lammps":
        s = _ghost_system(case, seed)
        nt, n = case["ntypes"], s["nlocal"]
        x, types = _t(s["x"]), _t(s["type"], torch.int64) - 1
        i, j = _t(s["rows"], torch.int64), _t(s["jflat"], torch.int64)
        v = x[j] - x[i]
        r2 = (v * v).sum(1)
        keep = r2 <= RC * RC
        i, j, v = i[keep], j[keep], v[keep].requires_grad_()
        davg, dstd = (a.to(DEV) for a in _dp_stats(nt, case["m"], case["density"]))
        Ei = _dp_energies(_dev(_dp_params(nt, seed)), davg, dstd, types, case["m"], i, j, v)[:n]
        F, f = _forces(Ei, i, j, v, len(types))
        W = (f.unsqueeze(2) * v.detach().unsqueeze(1)).sum(0)
        virial = torch.stack([W[0, 0], W[1, 1], W[2, 2], W[0, 1], W[0, 2], W[1, 2]])
        f = torch.zeros(_nmax(case), 3, dtype=F.dtype, device=DEV)
        f[:len(F)] = F
        return {"f": f, "eng": Ei.detach().sum(), "virial": virial, "eatom": Ei.detach(),
                "min_rsq": r2.min()}
    reps, vel = _replicas(case, seed)
    davg, dstd = (a.to(DEV) for a in _dp_stats(1, 100, 0.085))
    p = _dev(_dp_params(1, seed))
    lats, lens = [lat for lat, _ in reps], [len(f) for _, f in reps]
    x, vel = np.concatenate([f @ lat for lat, f in reps]), _t(vel)
    inv_mass = 1.0 / (63.546 * md.AMU_A2_FS2_EV)

    def forces(x):
        parts = np.split(x, np.cumsum(lens)[:-1])
        boxes = [(lat, q @ np.linalg.inv(lat), np.zeros(len(q), dtype=np.int64))
                 for lat, q in zip(lats, parts)]
        return _dp_boxes(p, davg, dstd, 100, boxes)[1]
    F = forces(x)
    x = _t(x)
    for _ in range(10):
        x = x + vel + 0.5 * inv_mass * F
        new = forces(x.cpu().numpy())
        vel, F = vel + 0.5 * inv_mass * (F + new), new
    return {"x": x, "v": vel, "F": F.unsqueeze(0)}
