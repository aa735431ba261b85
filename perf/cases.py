"""The calls that users of this engine spend their time in, as cases to time.

A docking program keeps an engine with its pair tables and receptor, and
calls it through the Python binding (``smina_b200.py`` over the C ABI):

  eval      model::eval_deriv of a batch of conformations (rescoring, local
            analysis); FP32, FP16 maps, FP64; with and without charges
  bfgs      the search's local optimisation of a batch of conformations
  receptor  a new receptor: cell lists, the grid maps of every ligand type,
            then a pose library evaluated on them
  minimize  --minimize: FP64 local optimisation of docked poses
  score     final rescoring of refined poses on the direct receptor sum
  dock64    the plain FP64 search (smina's trajectories)
  dock      the batched mixed-precision search with its FP64 refinement: a
            lone ligand, a screen, flexible residues with FP16 maps

Receptors, ligands and boxes are the synthetic ones of the benchmark: 2,000 to
5,000 receptor atoms, 22 to 30 A boxes, ligands of 10 to 60 heavy atoms and 0
to 15 rotors.  Searches run a part of smina's step count (its chains are some
thousand times the same step), so that a pass stays within a second.

Local optimisations and searches are chaotic: a changed last bit in one
evaluation moves a line search's accept, and after a few iterations a part of
the chains is in other minima (between 32 and 64 threads per chain, which only
order FP32 additions differently, up to half of the optimised conformations
end elsewhere).  Outputs of such calls can be compared as equal bits or not at
all, so their tolerance is "exact"; single evaluations have a relative one.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gpu-smina_b200"))

import smina_b200 as sb  # noqa: E402

CENTER = (0.5, 0.25, -0.3)
PREC = {"fp64": sb.PREC_FP64, "fp32": sb.PREC_FP32, "fp16maps": sb.PREC_FP32_H16}
# the user-weighted scoring of the flexible-residue configuration
CUSTOM = """-0.0400 gauss(o=0,_w=0.5,_c=8)
-0.0060 gauss(o=3,_w=2,_c=8)
0.8000 repulsion(o=0,_c=8)
-0.0300 hydrophobic(g=0.5,_b=1.5,_c=8)
-0.5500 non_dir_h_bond(g=-0.7,_b=0,_c=8)
1.923 num_tors_div
"""

_tables = {}


def _tables_for(scoring):
    """Pair tables depend on the scoring function only; a program builds them once."""
    if scoring not in _tables:
        _tables[scoring] = sb.Tables("vina", custom_text=CUSTOM) if scoring == "custom" else sb.Tables(scoring)
    return _tables[scoring]


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one pose of a 24-atom, 5-rotor ligand scored on resident maps
        {"name": "eval_one_pose", "kind": "eval", "prec": "fp32", "scoring": "vina", "heavy": 24, "rotors": 5,
         "poses": 1, "box": 22.0, "atoms": 3000},
        # a pose library of one ligand rescored
        {"name": "eval_library", "kind": "eval", "prec": "fp32", "scoring": "vina", "heavy": 31, "rotors": 7,
         "poses": 20000, "box": 25.0, "atoms": 3000},
        # charge-dependent scoring on the FP64 path (four table components, charge maps)
        {"name": "eval_charged_fp64", "kind": "eval", "prec": "fp64", "scoring": "ad4_scoring", "heavy": 37,
         "rotors": 9, "poses": 1500, "box": 25.0, "atoms": 3000},
        # the search's local optimisation on its own, a large flexible ligand
        {"name": "bfgs_large_ligand", "kind": "bfgs", "prec": "fp32", "scoring": "vina", "heavy": 50, "rotors": 12,
         "poses": 1536, "box": 30.0, "atoms": 3000},
        # a new receptor (the largest of the serving configuration) and its maps
        {"name": "new_receptor", "kind": "receptor", "prec": "fp32", "scoring": "vina", "heavy": 27, "rotors": 4,
         "poses": 4000, "box": 26.0, "atoms": 5000},
        # --minimize of one ligand's nine modes
        {"name": "minimize_nine", "kind": "minimize", "prec": "fp64", "scoring": "vina", "ligands": 1, "hmin": 24,
         "hmax": 24, "rmin": 5, "rmax": 5, "poses": 9, "box": 22.0, "atoms": 3000},
        # --minimize of 210 ligands x 9 docked poses (the published minimisation benchmark's size)
        {"name": "minimize_1890", "kind": "minimize", "prec": "fp64", "scoring": "vina", "ligands": 210, "hmin": 10,
         "hmax": 50, "rmin": 0, "rmax": 12, "poses": 9, "box": 22.0, "atoms": 3000},
        # final rescoring of a screen's refined poses
        {"name": "score_screen", "kind": "score", "prec": "fp32", "scoring": "vina", "ligands": 100, "hmin": 10,
         "hmax": 50, "rmin": 0, "rmax": 12, "poses": 20, "box": 22.0, "atoms": 3000},
        # plain FP64 redock, exhaustiveness 8
        {"name": "redock_fp64", "kind": "dock64", "prec": "fp64", "scoring": "vina", "heavy": 24, "rotors": 5,
         "chains": 8, "steps": 40, "box": 22.0, "atoms": 3000},
        # the redock ligand alone in the batched search: latency of its chains
        {"name": "dock_lone", "kind": "dock", "prec": "fp32", "scoring": "vina", "ligands": 1, "hmin": 24, "hmax": 24,
         "rmin": 5, "rmax": 5, "chains": 8, "steps": 400, "flex": 0, "box": 22.0, "atoms": 3000},
        # the screen: the device full of chains of ligands of all sizes
        {"name": "dock_screen", "kind": "dock", "prec": "fp32", "scoring": "vina", "ligands": 400, "hmin": 10,
         "hmax": 50, "rmin": 0, "rmax": 12, "chains": 8, "steps": 120, "flex": 0, "box": 22.0, "atoms": 3000},
        # flexible residues, custom scoring and FP16 maps
        {"name": "dock_flexible", "kind": "dock", "prec": "fp16maps", "scoring": "custom", "ligands": 24, "hmin": 10,
         "hmax": 50, "rmin": 0, "rmax": 12, "chains": 8, "steps": 30, "flex": 4, "box": 22.0, "atoms": 3000},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "bfgs", "receptor", "minimize", "score", "dock64", "dock", "dock", "dock"])
    heavy = rng.randint(10, 50)
    rotors = rng.randint(0, min(12, heavy // 3))
    atoms = rng.choice([2000, 3000, 5000])
    box = rng.choice([22.0, 23.5, 26.0, 30.0])
    size = (15 + heavy) * (15 + heavy) / 2500.0  # a pose's work relative to a 35-atom ligand's
    if kind == "eval":
        prec = rng.choice(["fp32", "fp32", "fp16maps", "fp64"])
        return {"kind": kind, "prec": prec, "scoring": rng.choice(["vina", "vina", "vinardo", "ad4_scoring"]),
                "heavy": heavy, "rotors": rotors, "poses": _log(rng, 1, 20000 / size if prec != "fp64" else 1500),
                "box": box, "atoms": atoms}
    if kind == "bfgs":
        return {"kind": kind, "prec": rng.choice(["fp32", "fp32", "fp16maps"]), "scoring": "vina", "heavy": heavy,
                "rotors": rotors, "poses": _log(rng, 1, 2500 / size), "box": box, "atoms": atoms}
    if kind == "receptor":
        return {"kind": kind, "prec": rng.choice(["fp32", "fp32", "fp16maps", "fp64"]),
                "scoring": rng.choice(["vina", "vina", "vinardo", "ad4_scoring"]), "heavy": rng.randint(10, 30),
                "rotors": rng.randint(0, 3), "poses": _log(rng, 16, 2000), "box": rng.choice([22.0, 23.5, 26.0]),
                "atoms": atoms}
    lo = rng.randint(10, 24)
    hi = rng.randint(lo, 50)
    if kind in ("minimize", "score"):
        return {"kind": kind, "prec": rng.choice(["fp64", "fp32"]), "scoring": rng.choice(["vina", "vina", "vinardo"]),
                "ligands": _log(rng, 1, 200), "hmin": lo, "hmax": hi, "rmin": 0, "rmax": min(12, lo // 2),
                "poses": rng.choice([1, 3, 9]), "box": box, "atoms": atoms}
    if kind == "dock64":
        return {"kind": kind, "prec": "fp64", "scoring": rng.choice(["vina", "vinardo"]), "heavy": rng.randint(10, 28),
                "rotors": rng.randint(0, 5), "chains": _log(rng, 1, 64), "steps": rng.randint(4, 30), "box": box,
                "atoms": atoms}
    ligands = _log(rng, 1, 300)
    chains = rng.choice([8, 8, 8, 16, 32, 128])
    ligands = max(1, min(ligands, 2400 // chains))
    return {"kind": kind, "prec": rng.choice(["fp32", "fp32", "fp16maps"]), "scoring": rng.choice(["vina", "vina", "custom"]),
            "ligands": ligands, "hmin": lo, "hmax": hi, "rmin": 0, "rmax": min(12, lo // 2), "chains": chains,
            "steps": _log(rng, 10, 100), "flex": 0, "box": box, "atoms": atoms}


# ---- inputs ---------------------------------------------------------------------------------
def _poses(m, n, rng, box, near, reach=0.2):
    """n conformations: near the pocket's centre as the ligand was built there
    (docked poses, ``near``), or anywhere within ``reach`` box sizes of the
    centre, as a search visits them."""
    init = np.array([m.desc.frame_init_origin[i] for i in range(3)])
    out = np.zeros((n, m.conf_size))
    if near:
        out[:, :3] = init + rng.normal(scale=0.4, size=(n, 3))
        ax = rng.normal(size=(n, 3))
        ax /= np.linalg.norm(ax, axis=1, keepdims=True)
        ang = rng.normal(scale=0.3, size=(n, 1))
        out[:, 3:7] = np.concatenate([np.cos(ang / 2), np.sin(ang / 2) * ax], axis=1)
        out[:, 7:] = rng.normal(scale=0.4, size=(n, m.conf_size - 7))
    else:
        out[:, :3] = np.array(CENTER) + rng.uniform(-reach, reach, size=(n, 3)) * box
        q = rng.normal(size=(n, 4))
        out[:, 3:7] = q / np.linalg.norm(q, axis=1, keepdims=True)
        out[:, 7:] = rng.uniform(-np.pi, np.pi, size=(n, m.conf_size - 7))
    return out


def _charged(pdbqt, rng):
    """The PDBQT with partial charges in its charge columns (the generator writes zeros)."""
    out = []
    for line in pdbqt.splitlines():
        if line.startswith(("ATOM", "HETATM")):
            line = line[:66] + "    " + f"{float(np.clip(rng.normal(scale=0.25), -0.9, 0.9)):+6.3f}" + line[76:]
        out.append(line)
    return "\n".join(out) + "\n"


class _ChargedReceptor:
    def __init__(self, base, rng):
        d = base.desc
        self.base = base
        self.q = np.clip(rng.normal(scale=0.3, size=d.num_atoms), -0.9, 0.9)
        self.desc = sb.ReceptorDesc(d.num_atoms, d.coords, d.type, sb.dptr(self.q))


_receptors = {}


def _receptor(atoms, seed):
    if (atoms, seed) not in _receptors:
        if len(_receptors) > 8:
            _receptors.clear()
        _receptors[(atoms, seed)] = sb.Receptor(atoms, seed, CENTER)
    return _receptors[(atoms, seed)]


def _inputs(case, seed):
    """Everything on the host: models, receptor, box, conformations, jobs."""
    rng = np.random.default_rng(seed)
    s = {"case": case, "tables": _tables_for(case["scoring"])}
    charged = case["scoring"] == "ad4_scoring"
    s["receptor"] = _receptor(case["atoms"], 7 if case["kind"] != "receptor" else 100 + seed % 5)
    if charged:
        s["receptor"] = _ChargedReceptor(s["receptor"], rng)
    s["box"] = sb.make_box(CENTER, (case["box"],) * 3)
    kind = case["kind"]

    def model(h, r, flex=None):
        text = sb.make_ligand_pdbqt(h, r, int(rng.integers(1, 1 << 40)), CENTER)
        return sb.Model(_charged(text, rng) if charged else text, flex)

    if "ligands" in case:
        flex = sb.make_flex_pdbqt(case["flex"], 42, CENTER) if case.get("flex") else None
        sizes = np.random.default_rng(case["ligands"])  # a case's ligand sizes; the seed makes other ligands of them
        s["models"] = [model(int(sizes.integers(case["hmin"], case["hmax"] + 1)),
                             int(sizes.integers(case["rmin"], case["rmax"] + 1)), flex) for _ in range(case["ligands"])]
    else:
        s["models"] = [model(case["heavy"], case["rotors"])]
    if kind in ("minimize", "score"):
        n, cs = case["poses"], max(m.conf_size for m in s["models"])
        s["pose_model"] = np.repeat(np.arange(len(s["models"]), dtype=np.int32), n)
        s["confs"] = np.zeros((len(s["pose_model"]), cs))
        for k, m in enumerate(s["models"]):
            s["confs"][k * n:(k + 1) * n, :m.conf_size] = _poses(m, n, rng, case["box"], True)
        p = [m.search_params() for m in s["models"]]
        s["maxiters"] = np.array([p[k].maxiters for k in s["pose_model"]], dtype=np.int32)
    elif kind in ("eval", "bfgs", "receptor"):
        s["confs"] = _poses(s["models"][0], case["poses"], rng, case["box"], kind == "bfgs",
                            0.5 if kind == "receptor" else 0.2)
        s["params"] = s["models"][0].search_params()
    elif kind == "dock64":
        m = s["models"][0]
        s["params"] = m.search_params()
        s["confs"], s["mt"] = m.seed_chains(int(rng.integers(1, 1 << 30)), case["chains"], s["box"])
    elif kind == "dock":
        s["params"] = s["models"][0].search_params()
        s["jobs"] = [sb.LigandJob(model=k, num_chains=case["chains"], num_steps=case["steps"],
                                  maxiters=m.search_params().maxiters, seed=seed, ligand_key=k)
                     for k, m in enumerate(s["models"])]
    return s


def _map_types(models):
    return sorted({t for m in models for t in m.types() if 2 <= t < sb.NUM_TYPES})


def prepare(case, seed):
    s = _inputs(case, seed)
    e = s["engine"] = sb.Engine(0, PREC[case["prec"]])
    e.set_tables(s["tables"])
    if case["kind"] != "receptor":
        e.set_receptor(0, s["receptor"], s["box"])
        if case["kind"] not in ("minimize", "score"):  # those use the direct receptor sum, no maps
            e.build_grids(0, _map_types(s["models"]))
    return s


# ---- a pass ---------------------------------------------------------------------------------
# the ligand types a receptor's maps are built for ahead of a screen
SCREEN_TYPES = list(range(2, 18))


def run(s):
    e, kind, ms = s["engine"], s["case"]["kind"], s["models"]
    if kind == "eval":
        return e.eval(0, ms[0], s["confs"])
    if kind == "bfgs":
        return e.bfgs(0, ms[0], s["confs"], maxiters=s["params"].maxiters)
    if kind == "receptor":
        e.set_receptor(0, s["receptor"], s["box"])
        e.build_grids(0, SCREEN_TYPES)
        return e.eval(0, ms[0], s["confs"])
    if kind == "minimize":
        return e.minimize(0, ms, s["pose_model"], s["confs"], maxiters=s["maxiters"])
    if kind == "score":
        return e.score(0, ms, s["pose_model"], s["confs"])
    if kind == "dock64":
        b = e.dock(0, ms, [0] * s["case"]["chains"], s["confs"], s["mt"], s["params"], steps=s["case"]["steps"])
        return {"e": b.e, "conf": b.conf, "coords": b.coords, "count": b.count, "evals": b.evals.astype(np.int64)}
    res = e.dock_batch(0, ms, s["jobs"], s["params"])
    # one table of poses, as a program keeps a screen's results (unused rows 0)
    n, c = s["params"].num_saved_mins, max(m.conf_size for m in ms)
    out = {"count": np.zeros(len(res), np.int64), "evals": np.zeros(len(res), np.int64), "e": np.zeros((len(res), n)),
           "conf": np.zeros((len(res), n, c)), "coords": np.zeros((len(res), n, max(m.heavy for m in ms), 3))}
    for k, r in enumerate(res):
        q = out["count"][k] = len(r["e"])
        out["evals"][k] = r["evals"]
        out["e"][k, :q] = r["e"]
        out["conf"][k, :q, :r["conf"].shape[1]] = r["conf"]
        out["coords"][k, :q, :r["coords"].shape[1]] = r["coords"]
    return out


def tolerance(case):
    if case["kind"] in ("eval", "receptor") and case["prec"] != "fp64":
        # one evaluation in FP32: up to 4e-6 from the 64-bit result was seen over
        # the ranges above
        return {"rel": 1.6e-5, "max": 2e-3}
    # FP64 paths round as the CPU algorithm does, bit for bit; optimisations
    # and searches are chaotic (above)
    return "exact"


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Bytes: inputs read and outputs written once.  Operations: per evaluation
    about 60 per grid lookup, 35 per pair and 150 per frame; a local
    optimisation evaluates at least once per iteration and updates its inverse
    Hessian."""
    kind, atoms = case["kind"], case["atoms"]

    def shape(h, r):
        n = h * 1.15  # with polar hydrogens
        return h, 0.4 * n * n * r / (r + 4), r + 1, 6 + r  # pairs: as counted on the generator's ligands

    h, r = (case["heavy"], case["rotors"]) if "heavy" in case else ((case["hmin"] + case["hmax"]) / 2,
                                                                    (case["rmin"] + case["rmax"]) / 2)
    if case.get("flex"):
        h, r = h + 30, r + 12
    grid, pairs, frames, dof = shape(h, r)
    ev = 60 * grid + 35 * pairs + 150 * frames
    direct = 60.0  # receptor atoms within the cutoff of an atom in the pocket's wall
    evd = 35 * direct * grid + 35 * pairs + 150 * frames
    iters = (25 + h * 1.15) / 3
    upd = 8 * dof * dof
    points = (case["box"] / 0.375 + 1) ** 3
    pose = 8 * (dof + 1)
    if kind == "eval":
        n = case["poses"]
        return {"bytes": n * (pose + 8 + 8 * dof), "flops": n * ev}
    if kind == "bfgs":
        n = case["poses"]
        return {"bytes": n * (2 * pose + 8), "flops": n * (iters + 1) * (ev + upd)}
    if kind == "receptor":
        n = case["poses"]
        per = {"fp64": 8, "fp32": 40, "fp16maps": 56}[case["prec"]] * (2 if case["scoring"] == "ad4_scoring" else 1)
        return {"bytes": 40 * atoms + len(SCREEN_TYPES) * points * per + n * (pose + 8 + 8 * dof),
                "flops": points * 60 * (10 + 2 * len(SCREEN_TYPES)) + n * ev}
    if kind == "minimize":
        n = case["ligands"] * case["poses"]
        return {"bytes": 40 * atoms + n * (2 * pose + 8 + 24 * h), "flops": n * (iters + 1) * (evd + upd)}
    if kind == "score":
        n = case["ligands"] * case["poses"]
        return {"bytes": 40 * atoms + n * (pose + 16 + 24 * h), "flops": n * evd}
    n = case.get("ligands", 1) * case["chains"]
    poses = 20 * case.get("ligands", case["chains"])
    return {"bytes": poses * (pose + 8 + 24 * h) + 2500 * (n if kind == "dock64" else 0),
            "flops": n * case["steps"] * (iters + 1) * (ev + upd) + (poses * (iters + 1) * (evd + upd) if kind == "dock" else 0)}


# ---- the same in plain torch, 64 bits -----------------------------------------------------------
class _Plain:
    """One model on one receptor: energies straight from the pair tables."""

    def __init__(self, s):
        dev = self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        f64 = dict(dtype=torch.float64, device=dev)
        td, rd, self.gd = s["tables"].desc, s["receptor"].desc, s["box"]
        n, nc, np_ = td.n, td.num_components, 27 * 28 // 2
        arr = np.ctypeslib.as_array
        self.nc, self.n, self.factor, self.cut = nc, n, td.factor, td.cutoff_sqr
        self.smooth = torch.tensor(arr(td.smooth, (np_, n, nc, 2)), **f64)
        self.fast = torch.tensor(arr(td.fast, (np_, n, nc)), **f64)
        t = arr(rd.type, (rd.num_atoms,)).copy()
        ok = (t >= 2) & (t < 27)
        self.rx = torch.tensor(arr(rd.coords, (rd.num_atoms, 3))[ok], **f64)
        self.rt = torch.tensor(t[ok], dtype=torch.int64, device=dev)
        self.rq = torch.tensor(arr(rd.charge, (rd.num_atoms,))[ok], **f64)
        self.f64 = f64

    def model(self, m):
        d, arr = m.desc, np.ctypeslib.as_array
        N, F, P = d.num_atoms, d.num_frames, d.num_pairs
        g = lambda p, shape: arr(p, shape).copy()  # noqa: E731
        self.M, self.F, self.dof = d.num_movable, F, d.dof
        self.type = torch.tensor(g(d.atom_type, (N,)), dtype=torch.int64, device=self.dev)
        self.q = torch.tensor(g(d.atom_charge, (N,)), **self.f64)
        self.local = torch.tensor(g(d.atom_local, (N, 3)), **self.f64)
        self.lab = torch.tensor(g(d.atom_lab, (N, 3)), **self.f64)
        self.kind, self.parent = g(d.frame_kind, (F,)), g(d.frame_parent, (F,))
        self.begin, self.end = g(d.frame_begin, (F,)), g(d.frame_end, (F,))
        self.fconf, self.fdof = g(d.frame_conf, (F,)), g(d.frame_dof, (F,))
        self.fo = torch.tensor(g(d.frame_origin, (F, 3)), **self.f64)
        self.fa = torch.tensor(g(d.frame_axis, (F, 3)), **self.f64)
        pr = g(d.pairs, (P, 2)) if P else np.zeros((0, 2), np.int32)
        self.pa, self.pb = (torch.tensor(pr[:, k], dtype=torch.int64, device=self.dev) for k in (0, 1))
        self.nother = d.num_other_pairs
        self.heavy = torch.tensor([i for i in range(self.M) if 2 <= int(self.type[i]) < 27], dtype=torch.int64, device=self.dev)
        return self

    @staticmethod
    def _qmul(a, b):
        aw, ax, ay, az = a.unbind(-1)
        bw, bx, by, bz = b.unbind(-1)
        return torch.stack([aw * bw - ax * bx - ay * by - az * bz, aw * bx + ax * bw + ay * bz - az * by,
                            aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw], -1)

    @staticmethod
    def _rows(q):
        a, b, c, d = q.unbind(-1)
        return torch.stack([a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (a * c + b * d),
                            2 * (a * d + b * c), a * a - b * b + c * c - d * d, 2 * (c * d - a * b),
                            2 * (b * d - a * c), 2 * (a * b + c * d), a * a - b * b - c * c + d * d], -1).reshape(-1, 3, 3)

    def set(self, conf):
        B = len(conf)
        self.O, self.A, Q, R = {}, {}, {}, {}
        X = self.lab.expand(B, -1, -1).clone()
        for f in range(self.F):
            c, p = int(self.fconf[f]), int(self.parent[f])
            if self.kind[f] == 0:
                self.O[f], Q[f], self.A[f] = conf[:, c:c + 3], conf[:, c + 3:c + 7], None
            else:
                if p >= 0:
                    self.O[f] = self.O[p] + (R[p] @ self.fo[f])
                    self.A[f] = R[p] @ self.fa[f]
                else:
                    self.O[f], self.A[f] = self.fo[f].expand(B, 3), self.fa[f].expand(B, 3)
                h = 0.5 * conf[:, c:c + 1]
                q = torch.cat([torch.cos(h), torch.sin(h) * self.A[f]], 1)
                Q[f] = self._qmul(q, Q[p]) if p >= 0 else q
            Q[f] = Q[f] / Q[f].norm(dim=1, keepdim=True)
            R[f] = self._rows(Q[f])
            b, e = int(self.begin[f]), int(self.end[f])
            X[:, b:e] = self.O[f][:, None] + torch.einsum("bij,aj->bai", R[f], self.local[b:e])
        return X

    def _pair(self, ta, tb):
        lo, hi = torch.minimum(ta, tb), torch.maximum(ta, tb)
        return lo + hi * (hi + 1) // 2, ta > tb

    def _weights(self, ta, qa, tb, qb):
        _, sw = self._pair(ta, tb)
        a, b = torch.where(sw, qb, qa), torch.where(sw, qa, qb)
        return torch.stack([torch.ones_like(a), a.abs(), b.abs(), a * b], -1)[..., :self.nc]

    @staticmethod
    def _curl(e, v):
        t = torch.where(e > 0, v / (v + e), torch.ones_like(e))
        return e * t, t * t

    def _map_value(self, t, pts):
        """(energy, energy per unit charge) of type t at points [K, 3]: the grid maps' values."""
        out = torch.zeros(len(pts), 2, **self.f64)
        p, sw = self._pair(self.rt, torch.full_like(self.rt, t))
        for k in range(0, len(pts), 8192):
            r2 = ((pts[k:k + 8192, None] - self.rx) ** 2).sum(-1)
            inn = r2 <= self.cut
            i = torch.where(inn, self.factor * r2, torch.zeros_like(r2)).long()
            f = self.fast[p.expand_as(i), i] * inn[..., None]
            a = f[..., 0]
            if self.nc > 1:
                c1, c2 = torch.where(sw, f[..., 2], f[..., 1]), torch.where(sw, f[..., 1], f[..., 2])
                out[k:k + 8192, 1] = (c2 + f[..., 3] * self.rq).sum(1)
                a = a + c1 * self.rq.abs()
            out[k:k + 8192, 0] = a.sum(1)
        return out

    def grid(self, X, v, slope):
        """Grid energies and their derivatives per movable atom."""
        B = len(X)
        lo = torch.tensor(list(self.gd.begin), **self.f64)
        hi = torch.tensor(list(self.gd.end), **self.f64)
        n = torch.tensor(list(self.gd.n), **self.f64)
        fac = n / (hi - lo)
        E, D = torch.zeros(B, **self.f64), torch.zeros(B, self.type.numel(), 3, **self.f64)
        for t in sorted(set(self.type[self.heavy].tolist())):
            at = self.heavy[self.type[self.heavy] == t]
            s = ((X[:, at] - lo) * fac).reshape(-1, 3)
            under, over = s < 0, s >= n
            miss = torch.where(under, -s, torch.where(over, s - n, torch.zeros_like(s)))
            region = over.double() - under.double()
            cell = torch.where(under, torch.zeros_like(s), torch.where(over, n - 1, s.floor()))
            cell = torch.minimum(cell, n - 1)
            fr = torch.where(under, torch.zeros_like(s), torch.where(over, torch.ones_like(s), s - cell))
            corner = torch.tensor([[i & 1, i >> 1 & 1, i >> 2] for i in range(8)], **self.f64)
            idx = (cell[:, None] + corner).long()
            dim = (n + 1).long()
            key = idx[..., 0] + dim[0] * (idx[..., 1] + dim[1] * idx[..., 2])
            uniq, inv = key.unique(return_inverse=True)
            pts = lo + torch.stack([uniq % dim[0], uniq // dim[0] % dim[1], uniq // (dim[0] * dim[1])], -1) / fac
            val = self._map_value(t, pts)[inv]
            w = corner * fr[:, None] + (1 - corner) * (1 - fr[:, None])
            sg = 2 * corner - 1
            for c in range(2 if self.nc > 1 else 1):
                q = self.q[at].repeat(B) if c else torch.ones(len(s), **self.f64)
                f = (val[..., c] * w.prod(-1)).sum(1)
                gr = torch.stack([(val[..., c] * sg[:, 0] * w[..., 1] * w[..., 2]).sum(1),
                                  (val[..., c] * w[..., 0] * sg[:, 1] * w[..., 2]).sum(1),
                                  (val[..., c] * w[..., 0] * w[..., 1] * sg[:, 2]).sum(1)], -1)
                f, k2 = self._curl(f, v)
                f = f + slope * (miss / fac).sum(-1)
                gr = fac * torch.where(region == 0, k2[:, None] * gr, torch.zeros_like(gr)) + slope * region
                if c:
                    f, gr = torch.where(q != 0, q * f, torch.zeros_like(f)), torch.where(q[:, None] != 0, q[:, None] * gr, torch.zeros_like(gr))
                E += f.reshape(B, -1).sum(1)
                D[:, at] += gr.reshape(B, -1, 3)
        return E, D

    def eval(self, conf, v=10.0, slope=1e6):
        X = self.set(conf)
        E, D = self.grid(X, v, slope)
        if len(self.pa):
            r = X[:, self.pb] - X[:, self.pa]
            r2 = (r * r).sum(-1)
            inn = r2 < self.cut
            p, _ = self._pair(self.type[self.pa], self.type[self.pb])
            w = self._weights(self.type[self.pa], self.q[self.pa], self.type[self.pb], self.q[self.pb])
            rf = torch.where(inn, self.factor * r2, torch.zeros_like(r2))
            i = rf.long()
            rem = rf - i
            lo = (self.smooth[p.expand_as(i), i] * w[:, :, None]).sum(-2)
            hi = (self.smooth[p.expand_as(i), i + 1] * w[:, :, None]).sum(-2)
            ed = lo + rem[..., None] * (hi - lo)
            e, k2 = self._curl(ed[..., 0], v)
            E = E + (e * inn).sum(1)
            f = r * (ed[..., 1] * k2 * inn)[..., None]
            D.index_add_(1, self.pa, -f)
            D.index_add_(1, self.pb, f)
        G = torch.zeros(len(conf), self.dof, **self.f64)
        Fs, Ts = {}, {}
        for f in range(self.F - 1, -1, -1):
            b, e = int(self.begin[f]), int(self.end[f])
            Fs[f] = D[:, b:e].sum(1) + Fs.get(f, 0)
            o = self.O[f]
            Ts[f] = torch.linalg.cross(X[:, b:e] - o[:, None], D[:, b:e]).sum(1) + Ts.get(f, 0)
            p, d0 = int(self.parent[f]), int(self.fdof[f])
            if p >= 0:
                Fs[p] = Fs.get(p, 0) + Fs[f]
                Ts[p] = Ts.get(p, 0) + Ts[f] + torch.linalg.cross(o - self.O[p], Fs[f])
            if self.kind[f] == 0:
                G[:, d0:d0 + 3], G[:, d0 + 3:d0 + 6] = Fs[f], Ts[f]
            else:
                G[:, d0] = (Ts[f] * self.A[f]).sum(-1)
        return E, G

    def score(self, conf, v=1000.0, slope=1e6):
        X = self.set(conf)
        lo = torch.tensor(list(self.gd.begin), **self.f64)
        hi = torch.tensor(list(self.gd.end), **self.f64)
        x = X[:, self.heavy]
        adj = torch.minimum(torch.maximum(x, lo), hi)
        r2 = ((adj[:, :, None] - self.rx) ** 2).sum(-1)
        inn = r2 < self.cut
        i = torch.where(inn, self.factor * r2, torch.zeros_like(r2)).long()
        ta, tb = self.type[self.heavy][:, None], self.rt[None, :]
        p, _ = self._pair(ta, tb)
        w = self._weights(ta, self.q[self.heavy][:, None], tb, self.rq[None, :])
        e = ((self.fast[p.expand_as(i), i] * w).sum(-1) * inn).sum(-1)
        e = (self._curl(e, v)[0] + slope * (x - adj).abs().sum(-1)).sum(1)
        intra = torch.zeros_like(e)
        if len(self.pa):
            r2 = ((X[:, self.pa] - X[:, self.pb]) ** 2).sum(-1)
            inn = r2 < self.cut
            i = torch.where(inn, self.factor * r2, torch.zeros_like(r2)).long()
            p, _ = self._pair(self.type[self.pa], self.type[self.pb])
            w = self._weights(self.type[self.pa], self.q[self.pa], self.type[self.pb], self.q[self.pb])
            intra = (self._curl((self.fast[p.expand_as(i), i] * w).sum(-1), v)[0] * inn).sum(1)
        return e + intra, intra, x


def exact(case, seed):
    if case["kind"] not in ("eval", "receptor", "score"):
        return None  # where an optimisation or a search ends depends on the rounding of every step (above)
    s = _inputs(case, seed)
    P = _Plain(s)
    conf = torch.tensor(s["confs"], **P.f64)
    if case["kind"] == "score":
        H = max(m.heavy for m in s["models"])
        e, intra, xyz = np.zeros(len(conf)), np.zeros(len(conf)), np.zeros((len(conf), H, 3))
        n = case["poses"]
        for k, m in enumerate(s["models"]):
            a, b, x = P.model(m).score(conf[k * n:(k + 1) * n, :m.conf_size])
            e[k * n:(k + 1) * n], intra[k * n:(k + 1) * n], xyz[k * n:(k + 1) * n, :m.heavy] = a.cpu(), b.cpu(), x.cpu()
        return e, intra, xyz
    P.model(s["models"][0])
    got = [P.eval(conf[k:k + 500]) for k in range(0, len(conf), 500)]
    return tuple(torch.cat([g[j] for g in got]).cpu().numpy() for j in (0, 1))
