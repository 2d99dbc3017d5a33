"""Performance cases of the docking engine: calls that a user's program makes through the public
entry points (``ud2b200.Engine``, ``ud2b200.ligset``, ``DockingPipeline``), on seeded
synthetic receptors and ligands of the shapes of the configurations in ``ud2b200/synth.py``.

``listed()`` are the cases, ``draw(rng)`` gives another of the same ranges, ``prepare`` makes what
the program holds before the call, ``run`` is one pass, ``work`` the bytes and operations it cannot
do without, ``tolerance`` and ``exact`` say how its outputs compare.
"""
import json
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "uni-dock2_b200"), ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from ud2b200.engine import GRID_F16, GRID_F32, MODE_DIRECT, MODE_GRID, Engine  # noqa: E402
from ud2b200.ligset import parse_ligands_bulk  # noqa: E402
from ud2b200.model import Box, VDW_RADII  # noqa: E402

# ---------------------------------------------------------------------- synthetic inputs
# XS types of the generated atoms, as in ud2b200/synth.py
C_H, C_P, N_P, N_D, N_A, O_A, O_DA, S_P = 2, 3, 4, 5, 6, 10, 11, 15
MAP_TYPES = [C_H, C_P, N_D, N_A, O_A]


def make_receptor(natom, cube, rng, pocket=8.0, gap=2.5):
    """natom heavy atoms, uniform in a cube, at least ``gap`` apart, with an empty sphere in the
    middle (the pocket): (xyz, types)."""
    edge = gap / math.sqrt(3.0)                        # a cell holds at most one atom
    m = int(cube / edge) + 1
    held = np.full((m + 4,) * 3, -1, np.int64)         # two empty cells around
    near = np.array([(a, b, c) for a in range(-2, 3) for b in range(-2, 3) for c in range(-2, 3)])
    pts = np.zeros((0, 3))
    while len(pts) < natom:
        cand = rng.uniform(0.0, cube, (4 * natom, 3))
        cand = cand[np.sum((cand - cube / 2) ** 2, 1) >= pocket * pocket]
        cell = (cand / edge).astype(np.int64) + 2
        # the first candidate of every cell, away from the atoms placed so far
        _, first = np.unique((cell[:, 0] * (m + 4) + cell[:, 1]) * (m + 4) + cell[:, 2], return_index=True)
        first.sort()
        cand, cell = cand[first], cell[first]

        def close(c, q, below=None):
            bad = np.zeros(len(c), bool)
            for d in near:
                j = held[q[:, 0] + d[0], q[:, 1] + d[1], q[:, 2] + d[2]]
                ok = j >= 0 if below is None else (j >= 0) & (j < below)
                if ok.any():
                    r = np.sum((c[ok] - pts[j[ok]]) ** 2, 1)
                    bad[np.nonzero(ok)[0][r < gap * gap]] = True
            return bad

        keep = ~close(cand, cell)
        cand, cell = cand[keep], cell[keep]
        base = len(pts)
        pts = np.concatenate([pts, cand])
        idx = np.arange(base, base + len(cand))
        held[cell[:, 0], cell[:, 1], cell[:, 2]] = idx
        # among the new ones, an atom stays if no earlier new one is close
        drop = close(cand, cell, below=idx)
        held[cell[drop, 0], cell[drop, 1], cell[drop, 2]] = -1
        ok = np.concatenate([np.ones(base, bool), ~drop])
        new = np.cumsum(ok) - 1
        pts = pts[ok]
        held = np.where(held >= 0, new[held], -1)
        if len(pts) > natom:
            cut = held >= natom
            held[cut] = -1
            pts = pts[:natom]
    u, v = rng.random(natom), rng.random(natom)
    types = np.where(u < 0.62, np.where(v < 0.5, C_H, C_P),
                     np.where(u < 0.79, np.where(v < 0.95, N_D, np.where(v < 0.99, N_P, N_A)),
                              np.where(u < 0.98, np.where(v < 0.86, O_A, O_DA), S_P)))
    return pts.astype(np.float32), types.astype(np.int32)


def make_ligand(natom, ntors, rng, center):
    """One ligand of the input schema: a random-walk tree of heavy atoms (1.5 A bonds, 109.5
    degree angles, 1-4 atoms at least 2.5 A apart and others 3.2 A), ntors of its inner bonds
    rotatable (fewer than half of the bonds)."""
    ang = math.radians(109.5)
    while True:
        x = np.zeros((natom, 3))
        par = np.full(natom, -1)
        deg = np.zeros(natom, int)
        dist = np.zeros((natom, natom), int)           # bonds between two atoms
        i, tries = 1, 0
        while i < natom and tries < 60 * natom:
            tries += 1
            p = max(0, i - 1 - int(rng.exponential(2.5)))
            if deg[p] >= 3:
                continue
            if par[p] >= 0 or deg[p]:
                g = par[p] if par[p] >= 0 else int(np.nonzero(par[:i] == p)[0][0])
                u = (x[p] - x[g]) / 1.5
                a = np.cross(u, [1.0, 0, 0] if abs(u[0]) < 0.9 else [0, 1.0, 0])
                a /= math.sqrt(a @ a)
                b = np.cross(u, a)
                phi = rng.uniform(0, 2 * math.pi)
                d = -math.cos(ang) * u + math.sin(ang) * (math.cos(phi) * a + math.sin(phi) * b)
            else:
                d = rng.normal(size=3)
                d /= math.sqrt(d @ d)
            q = x[p] + 1.5 * d
            r = np.sum((x[:i] - q) ** 2, 1)
            r[p] = 99.0
            r[par[:i] == p] = 99.0
            if par[p] >= 0:
                r[par[p]] = 99.0
            far = dist[p, :i] >= 3
            if r.min() < 2.5 ** 2 or r[far].min(initial=99.0) < 3.2 ** 2:
                continue
            x[i], par[i] = q, p
            dist[i, :i] = dist[:i, i] = dist[p, :i] + 1
            deg[p] += 1
            deg[i] += 1
            i += 1
        cand = [j for j in range(1, natom) if deg[j] > 1 and deg[par[j]] > 1]
        if i == natom and len(cand) >= ntors:
            break
    u = rng.random(natom)
    adj = np.zeros((natom, natom), bool)
    adj[np.arange(1, natom), par[1:]] = True
    adj |= adj.T
    polar = u >= 0.7
    nd = rng.random(natom) < 0.3
    types = np.where(u < 0.7, np.where((adj & polar[None, :]).any(1), C_P, C_H),
                     np.where(u < 0.85, np.where(nd, N_D, N_A), O_A))
    # subtree of every atom (the tree's parents come first)
    sub = np.eye(natom, dtype=bool)
    for j in range(natom - 1, 0, -1):
        sub[par[j]] |= sub[j]
    rot = sorted(cand[k] for k in rng.choice(len(cand), ntors, replace=False)) if ntors else []
    frag = np.zeros(natom, int)                        # rigid fragments
    for j in range(1, natom):
        frag[j] = j if j in rot else frag[par[j]]
    ids, size = np.unique(frag, return_counts=True)
    root = ids[np.argmax(size)]
    r0 = int(np.nonzero(frag == root)[0][0])
    tors = []
    for j in rot:
        side = sub[j].copy()
        frm, to = int(par[j]), j
        if side[r0]:
            side, frm, to = ~side, j, int(par[j])
        i0 = [int(k) for k in np.nonzero(adj[frm])[0] if k != to][0]
        i3 = [int(k) for k in np.nonzero(adj[to])[0] if k != frm][0]
        b0, b1, b2 = x[i0] - x[frm], x[to] - x[frm], x[i3] - x[to]
        b1 = b1 / math.sqrt(b1 @ b1)
        v, w = b0 - (b0 @ b1) * b1, b2 - (b2 @ b1) * b1
        val = math.degrees(math.atan2(np.cross(b1, v) @ w, v @ w))
        tors.append([[i0, frm, to, i3], val, [[-180.0, 180.0]], np.nonzero(side)[0].tolist(), []])
    n12, n13 = (dist > 0) & (dist <= 2), dist == 3
    x = x - x.mean(0) + np.asarray(center)
    atoms = [[float(x[i, 0]), float(x[i, 1]), float(x[i, 2]), int(types[i]), 0, 0.0, np.nonzero(n12[i])[0].tolist(),
              np.nonzero(n13[i])[0].tolist()] for i in range(natom)]
    return {"atoms": atoms, "torsions": tors, "root_atoms": np.nonzero(frag == root)[0].tolist()}


CUBE, CENTER = 40.0 * 2.0 ** (1.0 / 3.0), 20.0 * 2.0 ** (1.0 / 3.0)
BOX = 30.0


def sizes(kind, count):
    """(heavy atoms, rotatable bonds) of ``count`` ligands: the size mixes of ud2b200/synth.py, with
    no more than about half of the bonds rotatable.  The same for every seed."""
    rng = np.random.default_rng([count, 0x5172E])
    out = []
    for _ in range(count):
        if kind == "small":                            # one drug-like size
            out.append((24, 5))
        elif kind == "lead":                           # lead-like library
            out.append((int(rng.integers(12, 29)), int(min(4, rng.poisson(3)))))
        elif kind == "screen":                         # plain virtual screen
            out.append((int(rng.integers(12, 49)), int(min(12, rng.poisson(5)))))
        elif kind == "template":                       # congeners that share a core
            out.append((int(rng.integers(15, 41)), int(rng.integers(1, 9))))
        else:                                          # "uneven": everything up to 80 atoms, 20 bonds
            out.append((int(np.clip(round(math.exp(rng.normal(math.log(28), 0.45))), 8, 80)), int(rng.integers(0, 21))))
    return [(n, min(t, max(0, n // 2 - 3))) for n, t in out]


def make_ligands(kind, count, rng):
    """``count`` ligands of the input schema by name; above 148 the 148 distinct ones repeat under
    other names (a chain's random stream depends on the ligand's place in the batch)."""
    base = [make_ligand(n, t, rng, [CENTER] * 3) for n, t in sizes(kind, min(count, 148))]
    return {"lig%05d" % i: base[i % len(base)] for i in range(count)}


def make_engine(case, rng, ligands):
    """An engine that holds the receptor, its grid maps and the ligands."""
    eng = Engine(Box.from_center_size([CENTER] * 3, [BOX] * 3))
    eng.set_flags(constraint=bool(case.get("constraint", False)))
    xyz, types = make_receptor(case["receptor"], CUBE, rng)
    eng.set_receptor(xyz, types)
    eng.build_grid(0.375, MAP_TYPES, GRID_F16 if case.get("f16") else GRID_F32)
    ls = parse_ligands_bulk(ligands)
    eng.add_ligands(ls)
    return eng, ls, (xyz, types)


def place(ls, pose_lig, rng, spread):
    """A rigid pose of every ligand in ``pose_lig``: turned at random, its centre within ``spread``
    of the pocket's, moved into the box where it sticks out."""
    lo, hi = CENTER - BOX / 2 + 0.1, CENTER + BOX / 2 - 0.1
    coords = [None] * len(pose_lig)
    pose_lig = np.asarray(pose_lig)
    for l in np.unique(pose_lig):
        at = np.nonzero(pose_lig == l)[0]
        a0, a1 = ls.a["atom_off"][l], ls.a["atom_off"][l + 1]
        x = ls.a["xyz"][3 * a0:3 * a1].reshape(-1, 3).astype(np.float64)
        q = rng.normal(size=(len(at), 4))
        w, i, j, k = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
        R = np.stack([1 - 2 * (j * j + k * k), 2 * (i * j - k * w), 2 * (i * k + j * w),
                      2 * (i * j + k * w), 1 - 2 * (i * i + k * k), 2 * (j * k - i * w),
                      2 * (i * k - j * w), 2 * (j * k + i * w), 1 - 2 * (i * i + j * j)], 1).reshape(-1, 3, 3)
        p = np.einsum("pij,aj->pai", R, x - x.mean(0)) + (CENTER + rng.uniform(-spread, spread, (len(at), 1, 3)))
        p += np.maximum(0.0, lo - p.min(1, keepdims=True)) - np.maximum(0.0, p.max(1, keepdims=True) - hi)
        for r, c in zip(at, p.astype(np.float32)):
            coords[r] = c
    return coords


# ---------------------------------------------------------------------- the cases
def listed():
    return [
        # one ligand's few poses scored in a loop of the caller's own: latency of a call
        dict(name="score_few", do="score", poses=8, ligands=1, kind="small", receptor=4000, f16=False, direct=False),
        # rescoring of a pose collection of uneven ligands on half-precision maps
        dict(name="score_many", do="score", poses=16384, ligands=64, kind="uneven", receptor=4000, f16=True,
             direct=False),
        # exact energies and their decomposition per atom: the final scores of a screen's poses
        dict(name="terms_decomp", do="terms", poses=4099, ligands=64, kind="screen", receptor=4000, decomp=True),
        # a new receptor: its maps, the ligands loaded again, and the first scores on them
        dict(name="receptor", do="receptor", poses=512, ligands=8, kind="screen", receptor=4000, f16=False),
        # one round of refinement of pose candidates on exact sums (refine_steps=1)
        dict(name="refine", do="refine", poses=2048, ligands=64, kind="screen", receptor=4000, rounds=1),
        # a single congener docked thoroughly by few chains, its core held: a chain's latency
        dict(name="dock_one", do="dock", ligands=1, kind="template", receptor=4000, chains=64, mc_steps=200,
             constraint=True),
        # a batch of the plain virtual screen
        dict(name="dock_screen", do="dock", ligands=148, kind="screen", receptor=4000, chains=128, mc_steps=100),
        # uneven ligands up to 80 atoms by plain Metropolis moves (task "mc"), half-precision maps
        dict(name="mc_uneven", do="dock", ligands=256, kind="uneven", receptor=4000, chains=128, mc_steps=100, f16=True,
             plain=True),
        # congeners with their core held, the last four poses of every chain clustered at 2 A
        dict(name="template", do="dock", ligands=37, kind="template", receptor=4000, chains=256, mc_steps=20,
             constraint=True, retain=4, rmsd=2.0),
        # the same with the search on exact pair sums (scoring="direct")
        dict(name="template_direct", do="dock", ligands=8, kind="template", receptor=4000, chains=64, mc_steps=3,
             constraint=True, direct=True),
        # training of the proposal network
        dict(name="mlp_train", do="train", samples=16384, batch=1024, epochs=2),
        # a user's program: receptor rows and a ligand dict in, JSON files out, preset "fast"
        dict(name="pipeline_fast", do="pipeline", ligands=256, kind="lead", receptor=2000, mode="fast"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    rec = log(1500, 4000)
    do = rng.choice(["score", "score", "score", "terms", "receptor", "refine", "dock", "learned", "mc", "template",
                     "template", "train"])
    if do == "score":
        return dict(do="score", poses=log(1, 16384), ligands=log(1, 64), kind=rng.choice(["small", "screen", "uneven"]),
                    receptor=rec, f16=rng.random() < 0.5, direct=rng.random() < 0.3)
    if do == "terms":
        return dict(do="terms", poses=log(1, 4099), ligands=log(1, 64), kind=rng.choice(["small", "screen", "uneven"]),
                    receptor=rec, decomp=rng.random() < 0.5)
    if do == "receptor":
        return dict(do="receptor", poses=log(32, 512), ligands=8, kind="screen", receptor=rec, f16=rng.random() < 0.5)
    if do == "refine":
        return dict(do="refine", poses=log(64, 2048), ligands=64, kind=rng.choice(["lead", "screen"]), receptor=rec,
                    rounds=1)
    if do in ("dock", "learned"):
        case = dict(do="dock", ligands=rng.randint(200, 296), kind="lead", receptor=rec, chains=128,
                    mc_steps=rng.randint(40, 60))
        if do == "learned":                            # the proposal network's moves among the random ones
            case.update(p_learned=rng.choice([0.125, 0.25]))
        return case
    if do == "mc":
        return dict(do="dock", ligands=log(16, 256), kind="uneven", receptor=rec, chains=log(32, 128),
                    mc_steps=log(20, 100), f16=rng.random() < 0.5, plain=True)
    if do == "template":
        return dict(do="dock", ligands=log(8, 37), kind="template", receptor=rec, chains=log(64, 256),
                    mc_steps=log(10, 20), constraint=True, retain=rng.randint(1, 4), rmsd=2.0)
    return dict(do="train", samples=log(2048, 16384), batch=rng.choice([256, 512, 1024]), epochs=rng.randint(1, 2))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 0xD0C])
    do = case["do"]
    if do == "train":
        n = case["samples"]
        x = rng.standard_normal((n, Engine.MLP_IN), np.float32)
        y = x[:, :Engine.MLP_NDIM] * np.float32(0.5) + rng.standard_normal((n, Engine.MLP_NDIM), np.float32) * np.float32(0.3)
        m = (rng.random((n, Engine.MLP_NDIM)) < 0.6).astype(np.float32)
        eng = Engine(Box.from_center_size([0.0] * 3, [BOX] * 3))
        eng.mlp_init(seed & 0xFFFF)
        return dict(case=case, eng=eng, x=x, y=y, m=m, params=eng.mlp_get_params(), seed=seed)
    ligands = make_ligands(case["kind"], case["ligands"], rng)
    if do == "pipeline":
        edge = CUBE / 2.0 ** (1.0 / 3.0)
        xyz, types = make_receptor(case["receptor"], edge, rng)
        xyz = xyz + np.float32(CENTER - edge / 2)      # the smaller cube around the same centre
        rows = [[float(a), float(b), float(c), int(t), 0, 0.0] for (a, b, c), t in zip(xyz, types)]
        return dict(case=case, rows=rows, ligands=ligands, dir=tempfile.TemporaryDirectory(), seed=seed)
    if do == "receptor":
        ls = parse_ligands_bulk(ligands)
        rec = make_receptor(case["receptor"], CUBE, rng)
        eng = Engine(Box.from_center_size([CENTER] * 3, [BOX] * 3))
    else:
        eng, ls, rec = make_engine(case, rng, ligands)
        if case.get("retain"):
            eng.set_retain(case["retain"])
        if case.get("p_learned"):
            eng.mlp_init(seed & 0xFFFF)
    st = dict(case=case, eng=eng, ls=ls, rec=rec, seed=seed)
    if "poses" in case:
        n = case["poses"]
        st["lig"] = (np.arange(n) % len(ls)).astype(np.int32)
        st["coords"] = place(ls, st["lig"], rng, 2.0 if do == "refine" else 3.0)
        st["centers"] = np.array([c.mean(0) for c in st["coords"]], np.float32)
        rv = rng.normal(size=(n, 3))
        rv *= rng.uniform(0.05, 3.0, (n, 1)) / np.linalg.norm(rv, axis=1, keepdims=True)
        st["rotvecs"] = rv.astype(np.float32)
    if do == "refine":
        a = ls.a
        st["records"] = [np.concatenate([[999.0], c, np.zeros(4), x.reshape(-1),
                                         a["dihedrals"][a["tors_off"][l]:a["tors_off"][l + 1]]]).astype(np.float32)
                         for l, c, x in zip(st["lig"], st["centers"], st["coords"])]
    st["opt_steps"] = 0 if case.get("plain") else (25 + int(ls.natoms.max())) // 3
    return st


def run(st):
    case, do = st["case"], st["case"]["do"]
    if do == "score":
        e, g = st["eng"].score_batch(st["lig"], st["coords"], st["centers"], st["rotvecs"],
                                     mode=MODE_DIRECT if case["direct"] else MODE_GRID, vcap=10.0)
        return {"energy": e, "gradient": np.concatenate(g)}
    if do == "terms":
        t, d = st["eng"].score_terms(st["lig"], st["coords"], decomp=case["decomp"])
        return {"terms": t, "decomp": d}
    if do == "receptor":
        eng = st["eng"]
        eng.set_receptor(*st["rec"])
        eng.build_grid(0.375, MAP_TYPES, GRID_F16 if case["f16"] else GRID_F32)
        eng.clear_ligands()
        eng.add_ligands(st["ls"])
        e, g = eng.score_batch(st["lig"], st["coords"], st["centers"], st["rotvecs"], vcap=10.0)
        return {"energy": e, "gradient": np.concatenate(g)}
    if do == "refine":
        out, _ = st["eng"].bfgs_batch(st["lig"], st["records"], 2, case["rounds"], vcap=1000.0, slope0=100.0, ramp=True,
                                      mode=MODE_DIRECT)
        return {"energy": np.array([r[0] for r in out]), "pose": np.concatenate([r[8:] for r in out])}
    if do == "dock":
        res, _ = st["eng"].dock(st["seed"], case["chains"], case["mc_steps"], st["opt_steps"],
                                0 if case.get("plain") else 5, 1, case.get("rmsd", 1.0), 10.0,
                                mode=MODE_DIRECT if case.get("direct") else MODE_GRID, p_learned=case.get("p_learned"))
        score = np.array([r.terms[0].sum() for r in res])
        if not (case.get("plain") or case.get("constraint")):
            return {"ranked": np.sort(score)}
        out = {"score": score, "energy": np.array([r.records[0][0] for r in res])}
        if case.get("plain"):
            out["pose"] = np.concatenate([r.records[0][8:] for r in res])
        return out
    if do == "train":
        eng = st["eng"]
        eng.mlp_set_params(st["params"])
        loss = eng.mlp_train(st["x"], st["y"], st["m"], case["epochs"], case["batch"], 1e-3, seed=st["seed"])
        return {"loss": loss, "params": eng.mlp_get_params()}
    from unidock_engine.api.python.pipeline import DockingPipeline
    p = DockingPipeline(output_dir=st["dir"].name, center_x=CENTER, center_y=CENTER, center_z=CENTER, size_x=22.5,
                        size_y=22.5, size_z=22.5, search_mode=case["mode"], num_pose=1, seed=st["seed"], name_json="out")
    p.set_receptor(st["rows"])
    p.add_ligands(st["ligands"])
    p.run()
    affinity = []
    for f in sorted(os.listdir(st["dir"].name)):
        with open(os.path.join(st["dir"].name, f)) as h:
            affinity += [poses[0]["energy"][0] for poses in json.load(h).values()]
    return {"ranked": np.sort(affinity)}


# mean heavy atoms, torsions and scored intra pairs of a ligand of each kind
MEAN = {"small": (24, 5, 200), "lead": (20, 3, 80), "screen": (29, 5, 260), "uneven": (29, 9, 350), "template": (28, 5, 235)}


def work(case):
    """Bytes: inputs and outputs once, and the map values (or receptor atoms) at hand once.
    Operations: per evaluation about 40 a scored pair, 80 an atom on the maps (or 25 for each of
    the ~190 receptor atoms within 8 A) and 40 an atom and torsion level moved."""
    do = case["do"]
    if do == "train":
        n, w = case["samples"], 672 * 256 + 2 * 256 * 256 + 256 * 64
        steps = case["epochs"] * (n // case["batch"])
        return {"bytes": 4.0 * n * (672 + 52) + 4.0 * 2 * w + steps * (case["batch"] * 672 * 2.0 + 28.0 * w),
                "flops": 6.0 * w * steps * case["batch"]}
    atoms, tors, pairs = MEAN[case["kind"]]
    maps = 5 * 81 ** 3 * (2.0 if case.get("f16") else 4.0)
    direct = do in ("terms", "refine") or case.get("direct")
    near = 16.0 * case["receptor"]
    ev = 40.0 * pairs + (190 * 25.0 if direct else 80.0) * atoms
    if do in ("score", "receptor", "terms"):
        n = case["poses"]
        io = n * (12.0 * atoms + 28.0 + 4.0 * (7 + tors)) if do != "terms" else n * (12.0 * atoms + 20.0)
        if do == "terms" and case["decomp"]:
            io += n * 20.0 * atoms
        touched = near if direct else min(maps, n * atoms * 32.0)
        flops = n * ev
        if do == "receptor":                           # every map value: ~190 atoms near it
            touched = maps + near
            flops += 81.0 ** 3 * 190 * 5 * 15
        return {"bytes": io + touched, "flops": flops}
    ev += 40.0 * atoms * (1 + 0.5 * tors)
    rec = 4.0 * (8 + 3 * atoms + tors)
    if do == "refine":
        return {"bytes": case["poses"] * 2 * rec + near, "flops": case["poses"] * case["rounds"] * 3 * ev}
    chains = case["ligands"] * (128 if do == "pipeline" else case["chains"])
    steps = 20 if do == "pipeline" else case["mc_steps"]
    each = 1 if case.get("plain") else 1 + (25 + atoms) // 3
    return {"bytes": maps + case["ligands"] * (16.0 * pairs + rec) + case["ligands"] * rec,
            "flops": float(chains) * steps * each * ev}


def tolerance(case):
    """About four times what the same code differs by without fused multiply-adds.

    A BFGS search amplifies rounding until its chains part (over 98 % of them end elsewhere after
    20 steps), so of a free docking only the ranked best scores of the batch compare: 0.5-1.8 % in
    2-norm, the noise of two searches.  With the core held most chains stay together (best
    scores within 1.3 %); plain Metropolis chains and one round of refinement stay together but for
    single ones."""
    do = case["do"]
    if do == "terms":
        return {"rel": 2e-6, "max": 1e-4}
    if do in ("score", "receptor"):                    # the gradient jumps at the faces of the map's cells
        return {"rel": 2e-4, "max": 0.05} if case["f16"] else {"rel": 1e-4, "max": 0.02}
    if do == "train":                                  # BF16 activations, Adam steps
        return {"rel": 0.02, "max": 0.5}
    if do == "dock" and case.get("plain"):
        return {"rel": 5e-3, "max": 0.5}
    return {"rel": 0.03}


# ---------------------------------------------------------------------- 64-bit reference
HYD, ACC, DON = (2, 12, 16, 17, 18), (6, 7, 10, 11), (5, 7, 9, 11, 20)


def _flags(dev):
    t = torch.zeros(3, 32, dtype=torch.bool, device=dev)
    for row, ids in enumerate((HYD, ACC, DON)):
        t[row, list(ids)] = True
    return t


def _vina(d, hyd, hb):
    e = -0.035579 * torch.exp(-(2.0 * d) ** 2) - 0.005156 * torch.exp(-((d - 3.0) / 2.0) ** 2)
    e = e + 0.840245 * torch.clamp(d, max=0.0) ** 2
    e = e - 0.035069 * torch.clamp(1.5 - d, 0.0, 1.0) * hyd
    return e - 0.587439 * torch.clamp(-d / 0.7, 0.0, 1.0) * hb


def _near_sum(x, types, rec, rtypes, flags, radii, chunk=1 << 24):
    """Sum of the pair terms of points x (n, 3) of the given types with the receptor atoms within
    8 A."""
    parts = []
    step = max(1, chunk // len(rec))
    for s in range(0, len(x), step):
        p, t = x[s:s + step], types[s:s + step]
        r2 = ((p[:, None, :] - rec[None]) ** 2).sum(2)
        i, j = torch.nonzero(r2.detach() < 64.0, as_tuple=True)
        ti, tj = t[i], rtypes[j]
        d = torch.sqrt(r2[i, j]) - radii[ti] - radii[tj]
        hb = (flags[1][ti] & flags[2][tj]) | (flags[2][ti] & flags[1][tj])
        parts.append(torch.zeros(len(p), dtype=x.dtype, device=x.device).index_add(0, i, _vina(d, flags[0][ti] & flags[0][tj], hb)))
    return torch.cat(parts)


def _rotation(v):
    a = v.norm(dim=1)[:, None, None]
    z = torch.zeros_like(v[:, 0])
    K = torch.stack([z, -v[:, 2], v[:, 1], v[:, 2], z, -v[:, 0], -v[:, 1], v[:, 0], z], 1).reshape(-1, 3, 3)
    return torch.eye(3, dtype=v.dtype, device=v.device) + torch.sin(a) / a * K + (1 - torch.cos(a)) / a ** 2 * (K @ K)


def exact(case, seed):
    """Energies, gradients and score terms in 64 bits.  A search, a refinement and a training run
    have no such value: rounding decides which way they go."""
    do = case["do"]
    if do not in ("score", "receptor", "terms"):
        return None
    st = prepare(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    flags, radii = _flags(dev), torch.tensor(VDW_RADII, **f64)
    lo, hi = (torch.tensor(b, **f64) for b in (st["eng"].box.lo, st["eng"].box.hi))
    inside = np.all((st["rec"][0] >= st["eng"].box.lo - np.float32(8)) & (st["rec"][0] <= st["eng"].box.hi + np.float32(8)), 1)
    rec = torch.tensor(st["rec"][0][inside], **f64)
    rtypes = torch.tensor(st["rec"][1][inside], dtype=torch.long, device=dev)
    a, lig = st["ls"].a, st["lig"]
    grid = do != "terms" and not case.get("direct")
    n = len(lig)
    energy, grad, terms = [None] * n, [None] * n, [None] * n
    for l in np.unique(lig):
        at = np.nonzero(lig == l)[0]
        a0, a1, t0, t1 = (int(a[k][l + q]) for k in ("atom_off", "tors_off") for q in (0, 1))
        types = torch.tensor(a["types"][a0:a1], dtype=torch.long, device=dev)
        po = a["pair_off"][a0:a1 + 1]
        pi = np.repeat(np.arange(a1 - a0), np.diff(po))
        pj = a["pairs"][po[0]:po[-1]]
        pi, pj = (torch.tensor(v[pi < pj], dtype=torch.long, device=dev) for v in (pi, pj))
        x = torch.tensor(np.stack([st["coords"][k] for k in at]), **f64).requires_grad_(do != "terms")
        P, N = x.shape[:2]
        tt = types.repeat(P)
        # intra
        r2 = ((x[:, pj] - x[:, pi]) ** 2).sum(2)
        hb = (flags[1][types[pi]] & flags[2][types[pj]]) | (flags[2][types[pi]] & flags[1][types[pj]])
        ep = _vina(torch.sqrt(r2) - radii[types[pi]] - radii[types[pj]], flags[0][types[pi]] & flags[0][types[pj]], hb)
        ep = torch.where(r2 < 64.0, ep, torch.zeros_like(ep))
        out = (torch.clamp(lo - x, min=0.0) + torch.clamp(x - hi, min=0.0)).sum((1, 2)) * 1e6
        # inter
        if grid:
            h = 0.375
            top = math.ceil(BOX / h - 1e-4)
            u = torch.clamp((x - lo) / h, 0.0, float(top))
            i0 = torch.clamp(u.detach().floor(), 0, top - 1)
            f = u - i0
            ea = torch.zeros(P, N, **f64)
            for c in range(8):
                b = torch.tensor([c & 1, c >> 1 & 1, c >> 2], **f64)
                pt = ((i0 + b) * h + lo).to(torch.float32).to(torch.float64).reshape(-1, 3)
                w = torch.where(b > 0, f, 1 - f).prod(2)
                ea = ea + w * _near_sum(pt, tt, rec, rtypes, flags, radii).reshape(P, N)
        else:
            ea = _near_sum(x.reshape(-1, 3), tt, rec, rtypes, flags, radii).reshape(P, N)
        if do == "terms":
            T = torch.stack([ep.sum(1), ea.sum(1), out, torch.zeros_like(out)], 1).cpu().numpy()
            for k, r in zip(at, T):
                terms[k] = r
            continue
        cap = lambda e: torch.where(e > 0, e * 10.0 / (10.0 + torch.clamp(e, min=0.0)), e)  # noqa: E731
        E = cap(ep).sum(1) + cap(ea).sum(1) + out
        F = torch.autograd.grad(E.sum(), x)[0]
        x = x.detach()
        v = torch.tensor(st["rotvecs"][at], **f64)
        local = (x - torch.tensor(st["centers"][at], **f64)[:, None]) @ _rotation(v)
        v.requires_grad_(True)
        gv = torch.autograd.grad((F * (local @ _rotation(v).transpose(1, 2))).sum(), v)[0]
        g = [F.sum(1), gv]
        for k in range(t0, t1):
            frm, to = int(a["axis"][2 * k]), int(a["axis"][2 * k + 1])
            rot = torch.tensor(a["rot"][a["rot_off"][k]:a["rot_off"][k + 1]], dtype=torch.long, device=dev)
            ax = x[:, to] - x[:, frm]
            m = torch.linalg.cross(x[:, rot] - x[:, to][:, None], F[:, rot]).sum(1)
            g.append(((m * ax).sum(1) / ax.norm(dim=1))[:, None])
        E, g = E.detach().cpu().numpy(), torch.cat(g, 1).cpu().numpy()
        for q, k in enumerate(at):
            energy[k], grad[k] = E[q], g[q]
    if do == "terms":
        return {"terms": np.stack(terms), "decomp": None}
    return {"energy": np.array(energy), "gradient": np.concatenate(grad)}
