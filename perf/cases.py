"""What this framework's users have it do, as measurable cases.

Each case is a dict of plain values; `prepare` makes what a user's program
holds before the call (a context with its receptor, maps and ligands, and the
inputs), `run` is one pass through the public entry points of `vdock`, and
`exact` restates in 64 bits, in plain torch and numpy, what a pass returns
where that is a computed number (energies, gradients, maps, scores, RMSD
bounds).  What a stochastic search or an iterated optimisation ends with has
no such value.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vina-cuda_b200"))
import vdock  # noqa: E402
from vdock import synth  # noqa: E402

TYPES17 = list(range(17))


def listed():
    return [
        # One step of a minimiser or sampler written in torch: a few poses of
        # a drug-sized ligand on the caller's stream.  Latency and launches.
        dict(name="minimiser_step", kind="pose", call="energy_grad_device", poses=64, atoms=24, tors=5,
             rec_atoms=2000, rec_radius=40.0, box=20.0),
        # Scoring and differentiating a large pose set resident on the device
        # (the adjoint configuration of synth.CONFIGS).
        dict(name="adjoint_65536", kind="pose", call="energy_grad_device", poses=65536, atoms=40, tors=10,
             rec_atoms=2000, rec_radius=40.0, box=40.0),
        # Rescoring poses that another program wrote, from host arrays.
        dict(name="energy_host_10007", kind="pose", call="energy", poses=10007, atoms=33, tors=9,
             rec_atoms=4000, rec_radius=50.0, box=30.0),
        # Peptide-sized ligands: many intra pairs, deep torsion trees.
        dict(name="adjoint_peptide", kind="pose", call="energy_grad_device", poses=3001, atoms=90, tors=32,
             rec_atoms=4000, rec_radius=50.0, box=45.0),
        # Local optimisation of poses from another search, from host arrays.
        dict(name="local_opt_2000", kind="local_opt", poses=2000, atoms=28, tors=7, steps=20,
             rec_atoms=4000, rec_radius=50.0, box=30.0),
        # Grid maps of a pocket box, read back: what the reference's
        # kernel_grid call returns to its host program.
        dict(name="maps_pocket", kind="maps", types=7, box_x=22.5, box_y=18.4, box_z=26.1,
             rec_atoms=2500, rec_radius=40.0, poses=0, atoms=24, tors=5, weights=0),
        # A new receptor in the wide-box configuration: maps, then the poses
        # of a known ligand scored in it.
        dict(name="receptor_wide_box", kind="maps", types=8, box_x=70.0, box_y=70.0, box_z=70.0,
             rec_atoms=8000, rec_radius=60.0, poses=4096, atoms=40, tors=10, weights=0),
        # One ligand docked with a long search (the plain configuration).
        dict(name="dock_plain_1024x1000", kind="dock", form="plain", ligands=1, atoms_lo=24, atoms_hi=24, tors_lo=5,
             tors_hi=5, chains=1024, depth=1000, dense=0, rec_atoms=2000, rec_radius=40.0, box=20.0),
        # One ligand docked with the default chains and heuristic depth: what
        # a command-line user runs.
        dict(name="dock_plain_default", kind="dock", form="plain", ligands=1, atoms_lo=31, atoms_hi=31, tors_lo=8,
             tors_hi=8, chains=6500, depth=0, dense=0, rec_atoms=4000, rec_radius=50.0, box=30.0),
        # One batch of the virtual screen (the benchmark's workload): new
        # ligands handed over and docked in the wide box.
        dict(name="screen_batch_64", kind="dock", form="batched", ligands=64, atoms_lo=15, atoms_hi=45, tors_lo=2,
             tors_hi=12, chains=6500, depth=0, dense=0, rec_atoms=8000, rec_radius=60.0, box=70.0),
        # Ligands of very different sizes, few long chains each (the batched
        # configuration's 8,192 chains): the tail counts.
        dict(name="uneven_batch_256", kind="dock", form="batched", ligands=256, atoms_lo=10, atoms_hi=60, tors_lo=0,
             tors_hi=15, chains=32, depth=500, dense=0, rec_atoms=4000, rec_radius=50.0, box=30.0),
        # The docked modes of one ligand refined, scored and compared.
        dict(name="rescore_20", kind="rescore", poses=20, atoms=45, tors=12, rec_atoms=8000, rec_radius=60.0,
             box=30.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pose", "pose", "local_opt", "maps", "maps", "plain", "batched", "rescore"])
    atoms = rng.randint(10, 60)
    tors = rng.randint(0, min(15, atoms - 6))
    rec = rng.choice([(2000, 40.0), (4000, 50.0), (8000, 60.0)])
    box = round(rng.uniform(18.0, 45.0), 1)
    c = dict(rec_atoms=rec[0], rec_radius=rec[1])
    if kind == "pose":
        if rng.random() < 0.25:
            atoms, tors = rng.randint(61, 90), rng.randint(16, 40)
        top = 65536 if atoms <= 40 else 16384
        return dict(c, kind="pose", call=rng.choice(["energy_grad_device", "energy_device", "energy_grad", "energy",
                                                     "pose_coords"]),
                    poses=_log(rng, 16, top), atoms=atoms, tors=tors, box=box)
    if kind == "local_opt":
        return dict(c, kind="local_opt", poses=_log(rng, 16, 8192), atoms=atoms, tors=tors, steps=rng.randint(5, 30),
                    box=box)
    if kind == "maps":
        sides = [round(rng.uniform(14.0, 30.0), 1) for _ in range(3)]
        poses, weights = 0, 0
        if rng.random() < 0.6:  # score in new maps; some of these are a sweep over scoring weights
            sides = [round(math.exp(rng.uniform(math.log(18.0), math.log(70.0))), 1) for _ in range(3)]
            poses, weights = _log(rng, 64, 8192), rng.choice([0, 0, 2, 4])
        return dict(c, kind="maps", types=rng.randint(3, 8) if poses == 0 else rng.choice([8, 17]), box_x=sides[0],
                    box_y=sides[1], box_z=sides[2], poses=poses, atoms=min(atoms, 45), tors=min(tors, 12),
                    weights=weights)
    if kind == "plain":
        deep = rng.random() < 0.5
        atoms = min(atoms, 45)
        return dict(c, kind="dock", form="plain", ligands=1, atoms_lo=atoms, atoms_hi=atoms, tors_lo=min(tors, 12),
                    tors_hi=min(tors, 12), chains=_log(rng, 64, 1024) if deep else _log(rng, 1024, 8192),
                    depth=_log(rng, 50, 400) if deep else 0, dense=int(rng.random() < 0.25), box=box)
    if kind == "batched":
        n = _log(rng, 4, 128)
        return dict(c, kind="dock", form="batched", ligands=n, atoms_lo=rng.randint(10, 20),
                    atoms_hi=rng.randint(30, 50), tors_lo=rng.randint(0, 2), tors_hi=rng.randint(6, 12),
                    chains=_log(rng, 16, max(32, min(6500, 131072 // n))), depth=0, dense=int(rng.random() < 0.2),
                    box=box)
    return dict(c, kind="rescore", poses=rng.randint(2, 20), atoms=atoms, tors=tors, box=box)


# ------------------------------------------------------------------ inputs
def _box(case):
    return [case["box"]] * 3 if "box" in case else [case["box_x"], case["box_y"], case["box_z"]]


def _receptor(case, seed):
    return synth.receptor(case["rec_atoms"], case["rec_radius"], 1000 + seed)


def _ligand(case, seed):
    return synth.ligand(case["atoms"], case["tors"], 2000 + seed)


def _poses(case, lig, n, seed):
    """Positions at least 9 A inside the box where it is that large, uniform rotations and torsions."""
    half = np.array([max(1.0, b / 2 - 9.0) for b in _box(case)])
    return synth.random_poses(n, len(lig["node_parent"]) - 1, -half, half, 3000 + seed)


def _map_types(case, lig, seed):
    """The ligand's own types and others up to the number asked for."""
    if case["types"] >= 17:
        return TYPES17
    own = sorted(set(int(t) for t in lig["xs"]))
    rest = [t for t in synth.TYPES8 if t not in own]
    np.random.default_rng(4000 + seed).shuffle(rest)
    return sorted(own + rest[:max(0, case["types"] - len(own))]) if case["poses"] else (own + rest)[:case["types"]]


def _weights(case, seed):
    """Weight sets around the default ones, as a calibration tries them."""
    r = np.random.default_rng(5000 + seed)
    w = np.array(vdock.DEFAULT_WEIGHTS)
    return [w * (1 + 0.1 * r.uniform(-1, 1, 6)) for _ in range(case["weights"])]


def _context(case, seed, types):
    ctx = vdock.Context()
    ctx.set_receptor(*_receptor(case, seed))
    ctx.set_box([0.0, 0.0, 0.0], _box(case))
    if types is not None:
        ctx.build_grids(types)
    return ctx


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "pose":
        lig = _ligand(case, seed)
        s["ctx"] = ctx = _context(case, seed, sorted(set(int(t) for t in lig["xs"])))
        s["lig"] = ctx.add_ligand(lig)
        p = _poses(case, lig, case["poses"], seed)
        if case["call"].endswith("_device"):
            s["poses"] = torch.from_numpy(p).cuda()
            s["e"] = torch.empty(len(p), device="cuda")
            s["g"] = torch.empty(len(p), p.shape[1] - 1, device="cuda")
        else:
            s["poses"] = p
    elif kind == "local_opt":
        lig = _ligand(case, seed)
        s["ctx"] = ctx = _context(case, seed, sorted(set(int(t) for t in lig["xs"])))
        s["lig"] = ctx.add_ligand(lig)
        s["poses"] = _poses(case, lig, case["poses"], seed)
    elif kind == "maps":
        lig = _ligand(case, seed)
        s["ctx"] = ctx = vdock.Context()
        s["receptor"] = _receptor(case, seed)
        s["types"] = _map_types(case, lig, seed)
        s["weights"] = _weights(case, seed)
        s["lig"] = ctx.add_ligand(lig)
        if case["poses"]:
            s["poses"] = _poses(case, lig, case["poses"], seed)
    elif kind == "dock":
        # the receptor is the target of many calls: one for all seeds; its
        # ligands are what changes
        s["ctx"] = ctx = _context(case, 0, synth.TYPES8)
        s["descs"] = synth.ligand_set(case["ligands"], (case["atoms_lo"], case["atoms_hi"]),
                                      (case["tors_lo"], case["tors_hi"]), 6000 + seed)
        s["sp"] = vdock.search_params(seed=seed & 0x7FFFFFFF, n_chains=case["chains"], search_depth=case["depth"],
                                      refine=1, dense_bfgs=case["dense"])
        if case["form"] == "plain":
            s["lig"] = ctx.add_ligand(s["descs"][0])
    else:
        lig = _ligand(case, seed)
        s["ctx"] = ctx = _context(case, seed, None)
        s["lig"] = ctx.add_ligand(lig)
        s["poses"] = _poses(case, lig, case["poses"], seed)
    return s


# -------------------------------------------------------------------- passes
def _table(results, tors):
    """Docking results as whole arrays, [ligand][mode] and poses [ligand][mode][7 + tors], zeros past a ligand's own."""
    n, m = len(results), vdock.MAX_MODES
    out = {k: np.zeros((n, m), np.float32) for k in ("energy", "rmsd_lb", "rmsd_ub")}
    modes, evals = np.zeros(n, np.int32), np.zeros(n, np.int64)
    pose = np.zeros((n, m, 7 + tors), np.float32)
    for i, r in enumerate(results):
        k = len(r["energy"])
        modes[i], evals[i] = k, r["bfgs_evals"]
        for name, a in out.items():
            a[i, :k] = r[name]
        if k:
            pose[i, :k, :r["pose"].shape[1]] = r["pose"]
    return dict(out, pose=pose, modes=modes, bfgs_evals=evals)


def run(s):
    ctx, case, kind = s["ctx"], s["case"], s["kind"]
    if kind == "pose":
        call = case["call"]
        if call == "energy_grad_device":
            ctx.energy_grad_device(s["lig"], len(s["poses"]), s["poses"].data_ptr(), s["e"].data_ptr(),
                                   s["g"].data_ptr(), torch.cuda.current_stream().cuda_stream)
            return {"e": s["e"], "g": s["g"]}
        if call == "energy_device":
            ctx.energy_device(s["lig"], len(s["poses"]), s["poses"].data_ptr(), s["e"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
            return {"e": s["e"]}
        if call == "energy_grad":
            e, g = ctx.energy_grad(s["lig"], s["poses"])
            return {"e": e, "g": g}
        if call == "pose_coords":
            return {"xyz": ctx.pose_coords(s["lig"], s["poses"])}
        return {"e": ctx.energy(s["lig"], s["poses"])}
    if kind == "local_opt":
        e, p, evals = ctx.local_opt(s["lig"], s["poses"], case["steps"])
        return {"e": e, "poses": p, "evals": evals}
    if kind == "maps":
        ctx.set_receptor(*s["receptor"])
        ctx.set_box([0.0, 0.0, 0.0], _box(case))
        out = {}
        for i, w in enumerate(s["weights"] or [None]):
            if w is not None:
                ctx.set_scoring(w, device=True)
            ctx.build_grids(s["types"])
            if case["poses"]:
                out["e%d" % i], out["g%d" % i] = ctx.energy_grad(s["lig"], s["poses"])
            else:
                out["maps"] = [ctx.grid(t) for t in s["types"]]
        return out
    if kind == "dock":
        if case["form"] == "plain":
            return _table([ctx.dock_plain(s["lig"], s["sp"])], case["tors_hi"])
        ctx.clear_ligands()
        return _table(ctx.dock_batched(ctx.add_ligands(s["descs"]), s["sp"]), case["tors_hi"])
    e, p = ctx.refine(s["lig"], s["poses"])
    score, intra = ctx.score(s["lig"], s["poses"])
    lb, ub = ctx.rmsd_bounds(s["lig"], s["poses"])
    return {"refined_e": e, "refined": p, "score": score, "intra": intra, "lb": lb, "ub": ub}


def work(case):
    """Inputs read and results written once, and ~115 FP32 operations per
    heavy atom and ~25 per intra pair of an evaluation (a grid point: ~12 per
    receptor atom in reach and map); searches by their usual number of
    evaluations per Monte-Carlo step."""
    kind = case["kind"]
    table = 36 * 2049 * 16
    if kind == "dock":
        a, t = (case["atoms_lo"] + case["atoms_hi"]) / 2, (case["tors_lo"] + case["tors_hi"]) / 2
        depth = case["depth"] or max(1, int((0.24 * a + 0.29 * t - 3.41) * (2.4 if case["dense"] else 2.0)))
        evals = case["ligands"] * case["chains"] * depth * 25.0
        pairs = 0.33 * a * a
        return {"bytes": 8 * 4 * (case["box"] / 0.375 + 1) ** 3 + table + case["ligands"] * case["chains"] * 4 * (8 + t),
                "flops": evals * (115 * a + 25 * pairs)}
    a, t, n = case["atoms"], case["tors"], case["poses"]
    per = 115 * a + 25 * 0.37 * a * a
    if kind == "maps":
        pts = np.prod([b / 0.375 + 1 for b in _box(case)])
        near = case["rec_atoms"] * (8.0 / case["rec_radius"]) ** 3
        k = max(1, case["weights"])
        return {"bytes": k * (case["types"] * 4 * pts + 4.0 * n * (2 * t + 14)) + 32 * case["rec_atoms"],
                "flops": k * (pts * near * (8 + case["types"]) + n * per)}
    if kind == "rescore":
        near = case["rec_atoms"] * (8.0 / case["rec_radius"]) ** 3
        return {"bytes": 4.0 * n * (3 * t + 24) + 32 * case["rec_atoms"] + table,
                "flops": n * 5 * case["atoms"] * (per + 25 * near * a)}
    cells = min(32.0 * n * a, 32 * 8 * (case["box"] / 0.375) ** 3)
    if kind == "local_opt":
        return {"bytes": cells + table + 4.0 * n * (2 * t + 15), "flops": n * case["steps"] * 1.5 * per}
    out = {"pose_coords": 3 * a, "energy": 1, "energy_device": 1}.get(case["call"], 7 + t)
    if case["call"] == "pose_coords":
        return {"bytes": 4.0 * n * (7 + t + out), "flops": 30.0 * n * a}
    return {"bytes": cells + table + 4.0 * n * (7 + t + out), "flops": n * per}


# --------------------------------------------------------------- 64-bit values
_RADIUS = [1.9] * 2 + [1.8] * 4 + [1.7] * 4 + [2.0, 2.1, 1.5, 1.8, 2.0, 2.2, 1.2]
_HYDROPHOBIC, _ACCEPTOR, _DONOR = {0, 12, 13, 14, 15}, {4, 5, 8, 9}, {3, 5, 7, 9, 16}
_N = 2051


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _tables(w):
    """[17][17][2051] smooth energies, their derivative over r and the bin means."""
    r = np.sqrt(np.arange(_N) / 32.0)
    se, sd = np.zeros((17, 17, _N)), np.zeros((17, 17, _N))
    for a in range(17):
        for b in range(17):
            d = r - (_RADIUS[a] + _RADIUS[b])
            e = w[0] * np.exp(-(d / 0.5) ** 2) + w[1] * np.exp(-((d - 3.0) / 2.0) ** 2)
            e += w[2] * np.where(d < 0, d * d, 0.0)
            if a in _HYDROPHOBIC and b in _HYDROPHOBIC:
                e += w[3] * np.clip(1.5 - d, 0.0, 1.0)
            if (a in _DONOR and b in _ACCEPTOR) or (b in _DONOR and a in _ACCEPTOR):
                e += w[4] * np.clip(-d / 0.7, 0.0, 1.0)
            se[a, b] = e
            sd[a, b, 1:-1] = (e[2:] - e[:-2]) / ((r[2:] - r[:-2]) * r[1:-1])
    fast = (np.concatenate([se[:, :, 1:], np.zeros((17, 17, 1))], 2) + se) / 2
    return [torch.from_numpy(x).to(_dev()) for x in (se, sd, fast)]


def _geometry(case):
    n = [int(math.ceil(b / 0.375)) for b in _box(case)]
    begin = np.array([-0.375 * k / 2 for k in n])
    end = begin + 0.375 * np.array(n)
    finv = 1 / (np.array(n, float) / (end - begin))
    return [k + 1 for k in n], begin, end, finv


def _maps(case, rec, types, fast):
    """Grid maps [type][z][y][x]: sums over receptor atoms within 8 A of the bin's mean energy."""
    d = _dev()
    n, begin, end, finv = _geometry(case)
    xyz, xs = torch.from_numpy(rec[0]).to(d), torch.from_numpy(np.asarray(rec[1], np.int64)).to(d)
    # atoms within 8 A of the box
    q = torch.maximum(torch.from_numpy(begin).to(d) - xyz, xyz - torch.from_numpy(end).to(d)).clamp(min=0)
    near = (q * q).sum(1) < 64.0
    xyz, xs = xyz[near], xs[near]
    ax = [torch.from_numpy(begin[k] + finv[k] * np.arange(n[k])).to(d) for k in range(3)]
    out = torch.zeros(len(types), n[2], n[1], n[0], dtype=torch.float64, device=d)
    for z0 in range(0, n[2], 4):
        for y0 in range(0, n[1], 16):
            z, y = ax[2][z0:z0 + 4], ax[1][y0:y0 + 16]
            m = (xyz[:, 2] > z[0] - 8.1) & (xyz[:, 2] < z[-1] + 8.1) & (xyz[:, 1] > y[0] - 8.1) & (xyz[:, 1] < y[-1] + 8.1)
            a, t = xyz[m], xs[m]
            if not len(a):
                continue
            dx, dy, dz = (a[:, 0][:, None] - ax[0]), (a[:, 1][:, None] - y), (a[:, 2][:, None] - z)
            r2 = ((dx * dx)[:, None, None, :] + (dy * dy)[:, None, :, None]) + (dz * dz)[:, :, None, None]
            i, p = torch.nonzero((r2 <= 64.0).reshape(len(a), -1), as_tuple=True)
            b = (32.0 * r2.reshape(len(a), -1)[i, p]).long()
            plane = len(z) * len(y) * n[0]
            for j, tj in enumerate(types):
                acc = torch.zeros(plane, dtype=torch.float64, device=d)
                acc.index_add_(0, p, fast[tj][t[i], b])
                out[j, z0:z0 + 4, y0:y0 + 16] = acc.reshape(len(z), len(y), n[0])
    return out


def _qrot(q, v):
    w, u = q[..., :1], q[..., 1:]
    t = 2 * torch.linalg.cross(u, v.expand(q.shape[:-1] + (3,)))
    return v + w * t + torch.linalg.cross(u, t)


def _qmul(a, b):
    aw, av, bw, bv = a[..., :1], a[..., 1:], b[..., :1], b[..., 1:]
    return torch.cat([aw * bw - (av * bv).sum(-1, keepdim=True), aw * bv + bw * av + torch.linalg.cross(av, bv)], -1)


def _coords(lig, poses):
    """Atom positions [pose][atom][3], body origins and torsion axes [pose][body][3] in space."""
    d = _dev()
    p = torch.from_numpy(np.asarray(poses, np.float64)).to(d)
    xyz = torch.from_numpy(np.asarray(lig["xyz"], np.float64)).to(d)
    q = [p[:, 3:7] / p[:, 3:7].norm(dim=1, keepdim=True)]
    o, ax = [p[:, :3]], [torch.zeros_like(p[:, :3])]
    org = lig["node_origin_atom"]
    for k in range(1, len(lig["node_parent"])):
        pa = int(lig["node_parent"][k])
        u = xyz[int(org[k])] - xyz[int(lig["node_axis_atom"][k])]
        u = u / u.norm()
        o.append(o[pa] + _qrot(q[pa], xyz[int(org[k])] - xyz[int(org[pa])]))
        ax.append(_qrot(q[pa], u))
        h = 0.5 * p[:, 7 + k - 1:7 + k]
        q.append(_qmul(q[pa], torch.cat([torch.cos(h), torch.sin(h) * u], 1)))
    x = [o[int(b)] + _qrot(q[int(b)], xyz[i] - xyz[int(org[int(b)])]) for i, b in enumerate(lig["atom_node"])]
    return torch.stack(x, 1), torch.stack(o, 1), torch.stack(ax, 1)


def _grid_term(case, maps, slot, x, xs):
    """Trilinear energy [pose][atom] and force gradient [pose][atom][3], curl cap 10, slope 1e6 outside."""
    n, begin, end, finv = _geometry(case)
    d = x.device
    b, top = torch.from_numpy(begin).to(d), torch.tensor([k - 1.0 for k in n], dtype=torch.float64, device=d)
    factor = top / torch.from_numpy(end - begin).to(d)
    s = (x - b) * factor
    miss = ((torch.clamp(-s, min=0) + torch.clamp(s - top, min=0)) / factor).sum(-1)
    region = torch.where(s < 0, -1.0, torch.where(s >= top, 1.0, 0.0)).double()
    c = torch.minimum(torch.clamp(s, min=0), top)
    a = torch.minimum(c.long(), (top - 1).long())
    f = torch.where(s >= top, torch.ones_like(s), c - a)
    t = torch.tensor([slot[int(k)] for k in xs], device=d)[None, :].expand(x.shape[:2])
    g = 1 - f
    val, grad = 0.0, [0.0, 0.0, 0.0]
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                v = maps[t, a[..., 2] + k, a[..., 1] + j, a[..., 0] + i]
                wx, wy, wz = ((f if on else g)[..., q] for q, on in enumerate((i, j, k)))
                val = val + v * wx * wy * wz
                grad[0] = grad[0] + (2 * i - 1) * v * wy * wz
                grad[1] = grad[1] + (2 * j - 1) * v * wx * wz
                grad[2] = grad[2] + (2 * k - 1) * v * wx * wy
    cap = torch.where(val > 0, 10.0 / (10.0 + val), torch.ones_like(val))
    gr = torch.stack(grad, -1) * factor * (cap * cap)[..., None]
    return val * cap + 1e6 * miss, torch.where(region == 0, gr, 1e6 * region)


def _intra_term(lig, x, xs, se, sd):
    """Intra-ligand energy [pose] and its gradient on the atoms, interpolated tables, curl cap 10."""
    e = torch.zeros(len(x), dtype=torch.float64, device=x.device)
    f = torch.zeros_like(x)
    for lo in range(0, len(lig["pairs"]), 256):
        pr = torch.from_numpy(np.asarray(lig["pairs"][lo:lo + 256], np.int64)).to(x.device)
        ta, tb = xs[pr[:, 0]], xs[pr[:, 1]]
        r = x[:, pr[:, 1]] - x[:, pr[:, 0]]
        r2 = (r * r).sum(-1)
        inside = r2 < 64.0
        s = torch.clamp(32.0 * r2, max=2047.5)
        i = s.long()
        w = s - i
        v = se[ta, tb, i] * (1 - w) + se[ta, tb, i + 1] * w
        dv = sd[ta, tb, i] * (1 - w) + sd[ta, tb, i + 1] * w
        cap = torch.where(v > 0, 10.0 / (10.0 + v), torch.ones_like(v))
        e += torch.where(inside, v * cap, torch.zeros_like(v)).sum(1)
        pull = torch.where(inside, dv * cap * cap, torch.zeros_like(v))[..., None] * r
        f.index_add_(1, pr[:, 1], pull)
        f.index_add_(1, pr[:, 0], -pull)
    return e, f


def _energy_grad(case, lig, poses, maps, slot, tables):
    xs = torch.from_numpy(np.asarray(lig["xs"], np.int64)).to(_dev())
    e_all, g_all = [], []
    parent = [int(k) for k in lig["node_parent"]]
    for lo in range(0, len(poses), 4096):
        x, o, ax = _coords(lig, poses[lo:lo + 4096])
        e, f = _grid_term(case, maps, slot, x, lig["xs"])
        ei, fi = _intra_term(lig, x, xs, tables[0], tables[1])
        f = f + fi
        e_all.append(e.sum(1) + ei)
        F = [torch.zeros_like(o[:, 0]) for _ in parent]
        T = [torch.zeros_like(o[:, 0]) for _ in parent]
        for i, b in enumerate(lig["atom_node"]):
            F[int(b)] = F[int(b)] + f[:, i]
            T[int(b)] = T[int(b)] + torch.linalg.cross(x[:, i] - o[:, int(b)], f[:, i])
        g = [None] * len(parent)
        for k in range(len(parent) - 1, 0, -1):
            g[k] = (T[k] * ax[:, k]).sum(1)
            pa = parent[k]
            F[pa] = F[pa] + F[k]
            T[pa] = T[pa] + T[k] + torch.linalg.cross(o[:, k] - o[:, pa], F[k])
        g_all.append(torch.cat([F[0], T[0]] + [v[:, None] for v in g[1:]], 1))
    return torch.cat(e_all), torch.cat(g_all)


def _scores(case, lig, poses, rec, fast):
    """Adjusted score and intramolecular energy of poses on the direct-sum score, relative to pose 0."""
    d = _dev()
    x, _, _ = _coords(lig, poses)
    _, begin, end, _ = _geometry(case)
    b, e = torch.from_numpy(begin).to(d), torch.from_numpy(end).to(d)
    xyz, rx = torch.from_numpy(rec[0]).to(d), torch.from_numpy(np.asarray(rec[1], np.int64)).to(d)
    q = torch.maximum(b - xyz, xyz - e).clamp(min=0)
    near = (q * q).sum(1) < 64.0
    xyz, rx = xyz[near], rx[near]
    xs = torch.from_numpy(np.asarray(lig["xs"], np.int64)).to(d)
    c = torch.minimum(torch.maximum(x, b), e)
    inter = 1e6 * (x - c).abs().sum((1, 2))
    for i in range(x.shape[1]):
        r2 = ((c[:, i, None, :] - xyz) ** 2).sum(-1)
        v = torch.where(r2 < 64.0, fast[xs[i]][rx[None, :], (32.0 * r2).clamp(max=2050).long()], 0.0).sum(1)
        inter += torch.where(v > 0, v * 1000.0 / (1000.0 + v), v)
    pr = torch.from_numpy(np.asarray(lig["pairs"], np.int64).reshape(-1, 2)).to(d)
    r2 = ((x[:, pr[:, 0]] - x[:, pr[:, 1]]) ** 2).sum(-1)
    v = fast[xs[pr[:, 0]], xs[pr[:, 1]], (32.0 * r2).clamp(max=2050).long()]
    v = torch.where(v > 0, v * 1000.0 / (1000.0 + v), v)
    intra = torch.where(r2 < 64.0, v, torch.zeros_like(v)).sum(1)
    rotor = 0.1 * (vdock.DEFAULT_WEIGHTS[5] + 1)
    return (inter + intra - intra[0]) / (1 + rotor * float(lig["num_tors"]) / 5.0), intra


def _rmsd(lig, poses):
    x, _, _ = _coords(lig, poses)
    el = torch.from_numpy(np.asarray(lig["el"], np.int64)).to(_dev())
    other = (el[:, None] != el[None, :]).double() * 1e30
    ub = ((x - x[0]) ** 2).sum((1, 2)).div(x.shape[1]).sqrt()
    d2 = ((x[:, :, None, :] - x[0][None, None, :, :]) ** 2).sum(-1) + other
    one, two = d2.min(2).values.mean(1).sqrt(), d2.min(1).values.mean(1).sqrt()
    return torch.maximum(one, two), ub


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dock", "local_opt"):
        return None  # a search: no value of its own
    lig = _ligand(case, seed)
    rec = _receptor(case, seed)
    if kind == "rescore":
        poses = _poses(case, lig, case["poses"], seed)
        score, intra = _scores(case, lig, poses, rec, _tables(vdock.DEFAULT_WEIGHTS)[2])
        lb, ub = _rmsd(lig, poses)
        return {"refined_e": None, "refined": None, "score": score, "intra": intra, "lb": lb, "ub": ub}
    if kind == "maps":
        types = _map_types(case, lig, seed)
        out = {}
        for i, w in enumerate(_weights(case, seed) or [vdock.DEFAULT_WEIGHTS]):
            tables = _tables(w)
            maps = _maps(case, rec, types, tables[2])
            if not case["poses"]:
                return {"maps": [m for m in maps]}
            out["e%d" % i], out["g%d" % i] = _energy_grad(case, lig, _poses(case, lig, case["poses"], seed), maps,
                                                          {t: j for j, t in enumerate(types)}, tables)
        return out
    poses = _poses(case, lig, case["poses"], seed)
    if case["call"] == "pose_coords":
        return {"xyz": _coords(lig, poses)[0]}
    types = sorted(set(int(t) for t in lig["xs"]))
    tables = _tables(vdock.DEFAULT_WEIGHTS)
    maps = _maps(case, rec, types, tables[2])
    e, g = _energy_grad(case, lig, poses, maps, {t: j for j, t in enumerate(types)}, tables)
    return {"e": e, "g": g} if case["call"].startswith("energy_grad") else {"e": e}
