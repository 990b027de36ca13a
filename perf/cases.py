"""Workloads of the contact library for timing: what programs call, over the sizes they call it with.

kind      entry point                                        who calls it so
polyline  zdemx.polyline.pair_contacts, host arrays          the polyline.py drop-in: one pair of STL meshes
pairs     zdemx._lib.pair_contacts_device, CUDA tensors      pair sweeps, contact sets of another solver
host      zdemx.contact.pair_contacts_batch, host arrays     the same from numpy, with the loop points
adjoint   zdemx.autograd.pair_contacts and its backward      shape / pose / stiffness gradients
scene     zdemx.dem.Scene.step or .step_graph, .state        DEM runs (zdem_gpu, with and without --graph)
rollout   zdemx.rollout.DiffScene.rollout and its backward   calibration of k and e through a trajectory

Meshes: "ico" draws each side's mesh from noised icospheres of 80, 320, 1280 and 5120 triangles (the pair
sweep's mix), a number names one of these sizes, "hull" takes convex hulls of 30 to 400 points on an
ellipsoid (uneven triangle counts, long thin triangles).  Depth: "overlap" puts every pair 0 to 0.1 radii
into contact, "broad" spreads the gap as a sphere broad phase leaves it, many pairs apart.
"""
import math
import os
import sys
import tempfile
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zedm-x_b200"))

from zdemx import _lib, autograd, polyline, synth, workloads  # noqa: E402
from zdemx.contact import MeshLibrary, pair_contacts_batch  # noqa: E402
from zdemx.dem import Scene  # noqa: E402
from zdemx.rollout import DiffScene  # noqa: E402

RADIUS = 1e-3
LEVELS = {80: 1, 320: 2, 1280: 3, 5120: 4}


def listed():
    return [
        # one pair of particle meshes through the polyline mirror: the smallest call, all latency
        {"name": "polyline_pair", "kind": "polyline", "tris": 320, "split": False},
        # one pair of fine scans with --split-contacts: several separate contacts
        {"name": "polyline_fine_split", "kind": "polyline", "tris": 5120, "split": True},
        # the contact set of a small assembly, fewer pairs than the GPU has SMs
        {"name": "pairs_64", "kind": "pairs", "n": 64, "mesh": "ico", "depth": "overlap", "split": True},
        # a broad phase's candidates of a mid-size scene of convex particles
        {"name": "pairs_hull_6000", "kind": "pairs", "n": 6000, "mesh": "hull", "depth": "broad", "split": True},
        # fine meshes only: few pairs with many segments each
        {"name": "pairs_fine_1500", "kind": "pairs", "n": 1500, "mesh": "5120", "depth": "overlap", "split": True},
        # the pair sweep (benchmark size)
        {"name": "pairs_sweep", "kind": "pairs", "n": 65536, "mesh": "ico", "depth": "overlap", "split": True},
        # the sweep called from numpy with loop points, as a post-processing program does
        {"name": "host_8192", "kind": "host", "n": 8192, "mesh": "ico", "depth": "overlap", "split": True},
        # forward and backward of the contact geometry (benchmark size)
        {"name": "adjoint_16384", "kind": "adjoint", "n": 16384, "mesh": "320", "depth": "overlap", "split": True},
        # two particles pressed together: the smallest DEM step, one contact pair
        {"name": "scene_two", "kind": "scene", "scene": "two", "n": 2, "steps": 10, "graph": True},
        # the pour (benchmark's shapes): many candidates, few contacts, walls; the clearance cache at work
        {"name": "scene_pour_30000", "kind": "scene", "scene": "pour", "n": 30000, "steps": 10, "graph": True},
        # a bed of 729 particles on a plane, one Scene.step per step as zdem_gpu without --graph runs it
        {"name": "scene_bed_729", "kind": "scene", "scene": "bed", "n": 729, "steps": 4, "graph": False},
        # gradients of k, e and the velocities through a few steps of the same bed
        {"name": "rollout_729", "kind": "rollout", "n": 729, "steps": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["polyline", "pairs", "pairs", "pairs", "host", "adjoint", "scene", "scene", "rollout"])
    if kind == "polyline":
        return {"kind": kind, "tris": rng.choice(list(LEVELS)), "split": rng.random() < 0.5, "offset": round(rng.uniform(1.6, 1.9), 4)}
    if kind == "pairs":
        mesh = rng.choice(["ico", "ico", "hull", "80", "320", "1280", "5120"])
        return {"kind": kind, "n": _log(rng, 1, 2000 if mesh == "5120" else 40000), "mesh": mesh,
                "depth": rng.choice(["overlap", "broad"]), "split": rng.random() < 0.85}
    if kind == "host":
        return {"kind": kind, "n": _log(rng, 64, 8000), "mesh": rng.choice(["ico", "hull", "320", "1280"]),
                "depth": rng.choice(["overlap", "broad"]), "split": rng.random() < 0.85}
    if kind == "adjoint":
        return {"kind": kind, "n": _log(rng, 8, 16000), "mesh": rng.choice(["80", "320", "hull"]), "depth": "overlap",
                "split": True}
    if kind == "scene":
        scene = rng.choice(["two", "pour", "bed"])
        n = {"two": 2, "pour": _log(rng, 100, 30000), "bed": rng.randint(2, 9) ** 3}[scene]
        graph = scene == "pour" or rng.random() < 0.5
        return {"kind": kind, "scene": scene, "n": n, "steps": rng.randint(2, 12), "graph": graph}
    return {"kind": kind, "n": rng.randint(3, 9) ** 3, "steps": rng.randint(1, 3)}


# ------------------------------------------------------------------------------------------------ inputs
_CTX = []


def _ctx():
    """The context a program keeps for its pair calls."""
    if not _CTX:
        _CTX.append(_lib.Context(0))
    return _CTX[0]


def _meshes(mesh, n, rng):
    """(MeshLibrary, ids): build_mesh of up to 256 meshes a size; the ids a pair's sides are drawn from."""
    per = min(256, max(2, 2 * n))
    raw = []
    if mesh == "hull":
        for _ in range(min(per, 64)):
            raw.append(synth.ellipsoid_hull(int(rng.integers(30, 401)), (1.0, 0.8, 0.6), RADIUS, rng))
    else:
        for tris in LEVELS if mesh == "ico" else [int(mesh)]:
            raw.extend(synth.noised_icospheres(LEVELS[tris], per, RADIUS, 0.15, rng))
    with ThreadPoolExecutor(8) as ex:
        built = list(ex.map(lambda t: _lib.mesh_build(t, True), raw))
    off = np.zeros(len(raw) + 1, np.int64)
    off[1:] = np.cumsum([len(t) for t, _ in built])
    props = np.asarray([p["raw"] for _, p in built])
    return MeshLibrary(np.concatenate([t.reshape(-1, 9) for t, _ in built]), off, props[:, 5].copy(), props[:, 6].copy(),
                       props)


def _pairs(case, seed):
    rng = np.random.default_rng([seed, 11])
    n = case["n"]
    lib = _meshes(case["mesh"], n, rng)
    pm = rng.integers(0, lib.n_mesh, size=(n, 2)).astype(np.int32)
    lo, hi = (0.0, 0.1) if case["depth"] == "overlap" else (-0.15, 0.35)
    if case["mesh"] == "hull":
        lo, hi = lo + 0.3, hi + 0.45  # a hull's mean radius is well below its circumradius
    pp = synth.pair_poses(rng, n, RADIUS, lo, hi)
    pp[:, 3:7] = synth.random_unit_quat(rng, n)
    return lib, pm, pp


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _polyline_inputs(case, seed):
    rng = np.random.default_rng([seed, 12])
    tris = [synth.noised_icosphere(LEVELS[case["tris"]], RADIUS, 0.15, rng) for _ in range(2)]
    t = synth.random_dirs(rng, 1)[0] * (case.get("offset", 1.75) * RADIUS)
    return {"A": tris[0], "B": tris[1], "qA": synth.random_unit_quat(rng), "tB": t, "qB": synth.random_unit_quat(rng)}


def _bed(dirpath, n, seed):
    side = round(n ** (1.0 / 3.0))
    return workloads.calibration_scene(dirpath, n_side=side, seed=seed, spacing=1.8e-3)


def _scene(case, seed):
    with tempfile.TemporaryDirectory() as d:
        if case["scene"] == "two":
            cfg = workloads.two_particle_scene(d, seed=seed)
        elif case["scene"] == "pour":
            cfg = workloads.pour_scene(d, n=case["n"], seed=seed, spacing=1.8e-3)
        else:
            cfg = _bed(d, case["n"], seed)
        sc = Scene(cfg)
    st = sc.state()[0]
    if case["scene"] == "two":
        st[1, 0] = 1.75e-3  # already pressed together
    return {"scene": sc, "start": st, "out": sc.state()}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "polyline":
        return {"case": case, **_polyline_inputs(case, seed)}
    if kind == "scene":
        return {"case": case, **_scene(case, seed)}
    if kind == "rollout":
        with tempfile.TemporaryDirectory() as d:
            sc = Scene(_bed(d, case["n"], seed))
        st = sc.state()[0]
        goal = st[:, 0:3] + np.random.default_rng([seed, 14]).normal(scale=1e-5, size=(len(st), 3))
        return {"case": case, "ds": DiffScene(sc), "start": _cuda(st), "goal": _cuda(goal)}
    lib, pm, pp = _pairs(case, seed)
    if kind == "host":
        return {"case": case, "lib": lib, "pm": pm, "pp": pp}
    meshes = {"tris": _cuda(lib.tris), "tri_off": _cuda(lib.tri_off), "mean_edge": _cuda(lib.mean_edge),
              "bbox_diag": _cuda(lib.bbox_diag)}
    pairs = {"mesh": _cuda(pm), "pose": _cuda(pp)}
    if kind == "pairs":
        n, cap = case["n"], 64 + (24 if case["mesh"] == "5120" else 6) * case["n"]
        out = {"ncontact": torch.zeros(n, dtype=torch.int32, device="cuda"),
               "contact_off": torch.zeros(n + 1, dtype=torch.int64, device="cuda"),
               "stats": torch.zeros(n, 4, dtype=torch.int32, device="cuda"),
               "geom": torch.zeros(cap, 20, dtype=torch.float64, device="cuda"),
               "info": torch.zeros(cap, 4, dtype=torch.int32, device="cuda")}
        return {"case": case, "meshes": meshes, "pairs": pairs, "out": out}
    # adjoint: the loss weighs every pair's force and torque on A; the contacts are kept in buffers
    w = _cuda(np.random.default_rng([seed, 13]).normal(size=(case["n"], 6)))
    k = torch.tensor(1e7, dtype=torch.float64, device="cuda")
    cap = 64 + 6 * case["n"]
    kept = {key: torch.zeros(cap, 3, dtype=torch.float64, device="cuda") for key in ("Sn", "Gn", "xc0", "F_A")}
    kept["contact_id"] = torch.zeros(cap, dtype=torch.int32, device="cuda")
    return {"case": case, "meshes": meshes, "pairs": pairs, "w": w, "k": k, "kept": kept}


# ------------------------------------------------------------------------------------------------ passes
def run(state):
    case = state["case"]
    return RUN[case["kind"]](case, state)


def _run_polyline(case, s):
    manifold, loops, _, ids = polyline.pair_contacts(s["A"], s["B"], qA=s["qA"], tB=s["tB"], qB=s["qB"], k=1e7,
                                                     split_contacts=case["split"], ctx=_ctx())
    return _table(loops, ids, {key: [x[key] or (0.0, 0.0, 0.0) for x in manifold["contacts"]]
                               for key in ("Sn", "Gn", "xc0", "F_A")})


def _table(loops, ids, vectors):
    """A pair's contacts in arrays of a fixed size: 128 contacts, 8192 loop points."""
    out = {"ids": np.full(128, -1, np.int64), "nvert": np.zeros(128, np.int64), "points": np.zeros((8192, 3))}
    n = len(loops)
    if n:
        out["ids"][:n] = ids
        out["nvert"][:n] = [len(p) for p in loops]
        out["points"][: out["nvert"].sum()] = np.concatenate(loops)
    for key, rows in vectors.items():
        out[key] = np.zeros((128, 3))
        out[key][:n] = np.reshape(rows, (n, 3))
    return out


def _run_pairs(case, s):
    _lib.pair_contacts_device(_ctx(), s["meshes"], s["pairs"], s["out"], k=1e7, split=case["split"])
    return s["out"]


def _run_host(case, s):
    r = pair_contacts_batch(_ctx(), s["lib"], s["pm"], s["pp"], k=1e7, split=case["split"], want_points=True)
    # the arrays the call filled, to their capacity
    return {**r, **{key: r[key].base for key in ("geom", "info", "points", "point_off")}}


def _run_adjoint(case, s):
    m, p = s["meshes"], s["pairs"]
    tris, pose, k = (x.detach().requires_grad_() for x in (m["tris"], p["pose"], s["k"]))
    out = autograd.pair_contacts(tris, pose, m["tri_off"], m["mean_edge"], m["bbox_diag"], p["mesh"], k=k,
                                 split=case["split"])
    w = s["w"][out["pair"]]
    torque = torch.cross(out["xc0"] - pose[out["pair"], 0:3], out["F_A"], dim=1)
    loss = (w[:, 0:3] * out["F_A"]).sum() + (w[:, 3:6] * torque).sum() / RADIUS
    grads = torch.autograd.grad(loss, (tris, pose, k))
    with torch.no_grad():
        for key, kept in s["kept"].items():
            kept[: len(out[key])] = out[key]
    return {**s["kept"], "loss": loss, "grads": grads}


def _run_scene(case, s):
    sc = s["scene"]
    sc.set_state(s["start"])
    if case["graph"]:
        sc.step_graph(case["steps"])
    else:
        sc.step(case["steps"])
    info = sc.info()
    return {"state": sc.state(out=s["out"]), "counts": [info[c] for c in ("contacts", "segments", "comps", "loops", "pairs")]}


def _run_rollout(case, s):
    ds = s["ds"]
    k = torch.tensor(ds.feng_k, dtype=torch.float64, device="cuda", requires_grad=True)
    e = torch.tensor(0.5, dtype=torch.float64, device="cuda", requires_grad=True)
    v = s["start"][:, 7:10].clone().requires_grad_()
    end, _ = ds.rollout(torch.cat([s["start"][:, 0:7], v, s["start"][:, 10:16]], 1), k, e, case["steps"])
    loss = ((end[:, 0:3] - s["goal"]) ** 2).sum()
    return {"end": end, "loss": loss, "grads": torch.autograd.grad(loss, (k, e, v))}


RUN = {"polyline": _run_polyline, "pairs": _run_pairs, "host": _run_host, "adjoint": _run_adjoint, "scene": _run_scene,
       "rollout": _run_rollout}


# ------------------------------------------------------------------------------------------------ work
MEAN_TRIS = {"ico": 1700.0, "hull": 426.0}  # triangles of a mesh, on average
TEMPLATE_TRIS = {"two": 640.0, "pour": 3 * 124.0 + 320 + 1280, "bed": 320.0}


def work(case):
    """Bytes of one pass: 72 a triangle of the meshes, 120 a pair for its ids and poses, 28 for its counts,
    176 a contact (about two a pair in contact); for a scene 128 in and 160 out a particle and step.
    Gradients as many bytes again as what they belong to."""
    kind, n = case["kind"], case["n"] if "n" in case else 1
    if kind == "polyline":
        return {"bytes": 2 * 72.0 * case["tris"] + 148 + 2 * 176, "flops": 0.0}
    if kind in ("scene", "rollout"):
        tris = TEMPLATE_TRIS[case.get("scene", "bed")]
        passes = 3 if kind == "rollout" else 1
        return {"bytes": passes * case["steps"] * (288.0 * n + 72 * tris), "flops": 0.0}
    meshes = min(64 if case["mesh"] == "hull" else 1024 if case["mesh"] == "ico" else 256, 2 * n)
    tris = meshes * (MEAN_TRIS[case["mesh"]] if case["mesh"] in MEAN_TRIS else float(case["mesh"]))
    contacts = 2.0 * n if case["depth"] == "overlap" else 0.5 * n
    per = 72 * tris + 148 * n + 176 * contacts
    return {"bytes": per * (3 if kind == "adjoint" else 1), "flops": 0.0}


# ------------------------------------------------------------------------------------------------ exact
def exact(case, seed):
    """The loops of a polyline pair (one component, no --split-contacts) by numpy in FP64; None for the other
    cases: thousands of pairs take numpy minutes, and the order and direction of their loops are fixed by
    the reference program's sort, not by the geometry."""
    if case["kind"] != "polyline" or case["split"]:
        return None
    s = _polyline_inputs(case, seed)
    tol = 1e-6
    A, B = _place(s["A"], s["qA"], np.zeros(3)), _place(s["B"], s["qB"], s["tB"])
    V, edges = _snap(_segments(A, B), tol)
    loops = _loops(V, _split(V, edges, tol), tol)
    vectors = {"Sn": [], "Gn": [], "xc0": [], "F_A": []}
    for p in loops:
        q = np.roll(p, -1, 0)
        dx = q - p
        Sn = 0.5 * np.cross(p, q).sum(0)
        Gn = (-((p * q).sum(1) + (dx * dx).sum(1) / 3) / 3) @ dx
        area = np.linalg.norm(Sn)
        for key, row in zip(vectors, (Sn, Gn, np.cross(-Sn / area, Gn) / area, -0.5 * 1e7 * Sn)):
            vectors[key].append(row)
    return {**_table(loops, np.zeros(len(loops)), vectors), "ids": None, "nvert": None}


def _place(tris, q, t):
    w, u = q[0], q[1:]
    h = 2.0 * np.cross(u, tris)
    return tris + w * h + np.cross(u, h) + t


def _segments(A, B):
    """(n, 2, 3): the cuts of every pair of triangles that share a segment, in (A, B) order."""
    hit = np.ones((len(A), len(B)), bool)
    for k in range(3):
        hit &= (A.max(1)[:, None, k] >= B.min(1)[None, :, k]) & (A.min(1)[:, None, k] <= B.max(1)[None, :, k])
    ia, ib = np.nonzero(hit)
    T = (A[ia], B[ib])
    n = [np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]) for x in T]
    n = [x / np.linalg.norm(x, axis=1, keepdims=True) for x in n]
    tau = np.cross(n[0], n[1])
    tau /= np.maximum(np.linalg.norm(tau, axis=1, keepdims=True), 1e-300)
    pts, use = [], []
    for side in range(2):
        E, F, m = T[side], T[1 - side], n[1 - side]
        for i in range(3):
            p, u = E[:, i], E[:, (i + 1) % 3] - E[:, i]
            den = (m * u).sum(1)
            t = ((F[:, 0] - p) * m).sum(1) / np.where(np.abs(den) < 1e-30, np.inf, den)
            x = p + u * np.clip(t, 0.0, 1.0)[:, None]
            ok = (np.abs(den) >= 1e-30) & (t >= -1e-10) & (t <= 1.0 + 1e-10)
            for j in range(3):
                ok &= (np.cross(F[:, (j + 1) % 3] - F[:, j], x - F[:, j]) * m).sum(1) >= -1e-10
            for y, o in zip(pts, use):  # a point found before
                ok &= ~(o & (((x - y) ** 2).sum(1) <= 1e-18))
            pts.append(x)
            use.append(ok)
    P, use = np.stack(pts, 1), np.stack(use, 1)
    t = (P * tau[:, None]).sum(2)
    i0, i1 = np.where(use, t, np.inf).argmin(1), np.where(use, t, -np.inf).argmax(1)
    r = np.arange(len(P))
    S = np.stack([P[r, i0], P[r, i1]], 1)
    return S[(use.sum(1) >= 2) & (i0 != i1) & (((S[:, 1] - S[:, 0]) ** 2).sum(1) >= 1e-18)]


def _snap(S, tol):
    """Endpoints within tol of one another, and of one another's, become one vertex at their mean."""
    P = S.reshape(-1, 3)
    near = np.linalg.norm(P[:, None] - P[None], axis=2) <= tol
    label = np.arange(len(P))
    while len(P):
        new = np.where(near, label[None], len(P)).min(1)
        if (new == label).all():
            break
        label = new
    _, v = np.unique(label, return_inverse=True)
    V = np.zeros((v.max() + 1 if len(v) else 0, 3))
    np.add.at(V, v, P)
    V /= np.bincount(v)[:, None] if len(v) else 1.0
    return V, [(a, b) for a, b in v.reshape(-1, 2) if a != b]


def _split(V, edges, tol):
    """Each edge cut at the vertices that lie on its inside."""
    out = []
    for a, b in edges:
        d = V[b] - V[a]
        t = np.clip((V - V[a]) @ d / max(d @ d, 1e-300), 0.0, 1.0)
        on = (((V - V[a] - t[:, None] * d) ** 2).sum(1) <= tol * tol) & (t > 1e-6) & (t < 1 - 1e-6)
        on[[a, b]] = False
        on &= bool(d @ d > 1e-12)
        chain = [a, *sorted(np.nonzero(on)[0], key=lambda x: t[x]), b]
        out += list(zip(chain[:-1], chain[1:]))
    return out


def _loops(V, edges, tol):
    """Closed walks over unused edges, from the vertices with two edges first, never straight back."""
    near = [[] for _ in V]
    for e, (a, b) in enumerate(edges):
        near[a].append((b, e))
        near[b].append((a, e))
    used, loops = set(), []
    for s in sorted(range(len(V)), key=lambda v: (len(near[v]) != 2, -len(near[v]))):
        for nxt, e in near[s]:
            if e in used:
                continue
            used.add(e)
            path, prev, cur = [s], s, nxt
            while cur != s:
                path.append(cur)
                free = [x for x in near[cur] if x[1] not in used]
                if not free:
                    path = []
                    break
                to, e2 = next((x for x in free if x[0] != prev), free[0])
                used.add(e2)
                prev, cur = cur, to
            if len(path) >= 3 and np.linalg.norm(np.ptp(V[path], axis=0)) >= 2 * tol:
                loops.append(V[path])
    return loops
