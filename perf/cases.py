"""The workloads that performance work on this framework is measured on.

Each case is one call pattern of a user's program through the public interface:

* ``flat`` / ``tet`` / ``hex`` / ``surface``: an optimiser that the program keeps is given new
  vertex positions (device array), restarted and iterated; the moved positions and the minimum
  quality come back. A moving-mesh simulation does this once per time step.
* ``batch``: the same for many independent flat meshes in one ``BatchDMO``.
* ``learned``: the tet optimiser in learned mode with a network trained beforehand.
* ``train``: training steps of the proposal network on collected pairs.
* ``build``: the connectivity and colouring of a new mesh.
* ``inspect``: per-element qualities, histogram and statistics of a mesh.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

import volumesurfacediscretemeshoptimization_b200 as V
from volumesurfacediscretemeshoptimization_b200 import _capi
from volumesurfacediscretemeshoptimization_b200 import meshgen as G


def listed():
    return [
        # the small flat benchmark mesh: a user's interactive 2D smoothing, bound by launches
        {"name": "flat_tri_64", "kind": "flat", "elem": "tri", "n": 64, "iters": 20, "fix_boundary": True,
         "quality": "MEAN_RATIO"},
        # a toy volume mesh: the smallest volume call, bound by launches
        {"name": "tet_10", "kind": "tet", "n": 10, "iters": 10, "refine": 0.0, "fix_boundary": True,
         "quality": "MEAN_RATIO"},
        # the headline benchmark: 117,649 vertices, 20 iterations
        {"name": "tet_48", "kind": "tet", "n": 48, "iters": 20, "refine": 0.0, "fix_boundary": True,
         "quality": "MEAN_RATIO"},
        # a production-sized volume mesh: 1,030,301 vertices, 6 M tetrahedra
        {"name": "tet_100", "kind": "tet", "n": 100, "iters": 5, "refine": 0.0, "fix_boundary": True,
         "quality": "MEAN_RATIO"},
        # an irregular mesh (locally refined, uneven valence) whose boundary moves too, the
        # reference's own default
        {"name": "tet_30_refined_free", "kind": "tet", "n": 30, "iters": 10, "refine": 0.15, "fix_boundary": False,
         "quality": "MEAN_RATIO"},
        # hexahedra: 35,937 vertices
        {"name": "hex_32", "kind": "hex", "n": 32, "iters": 10, "fix_boundary": True, "quality": "MEAN_RATIO"},
        # a triangle surface with feature lines: icosphere of 163,842 vertices
        {"name": "surface_tri_7", "kind": "surface", "elem": "tri", "level": 7, "iters": 10, "noise": 1e-3},
        # many 2D meshes of 500 to 50,000 vertices together, triangles and quads
        {"name": "batch_256", "kind": "batch", "count": 256, "v_min": 500, "v_max": 50000, "iters": 5},
        # learned mode on a mesh that the network has not seen
        {"name": "learned_64", "kind": "learned", "n": 64, "iters": 10},
        # training the proposal network at the batch size its recipe uses
        {"name": "train_8192", "kind": "train", "batch": 8192, "steps": 50},
        # building the headline mesh from device arrays
        {"name": "build_tet_48", "kind": "build", "elem": "tet", "n": 48, "refine": 0.0},
        # looking at the headline mesh: element qualities, histogram, minimum
        {"name": "inspect_tet_48", "kind": "inspect", "n": 48},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fixed = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in fixed:
            return case


def _draw(rng):
    kind = rng.choice(["flat", "tet", "tet", "tet", "hex", "surface", "surface", "batch", "learned", "train", "build",
                       "inspect"])
    if kind == "flat":
        elem = rng.choice(["tri", "tri", "quad"])
        fix = elem == "quad" or rng.random() < 0.6
        quality = "MIN_ANGLE" if elem == "tri" and rng.random() < 0.25 else "MEAN_RATIO"
        return {"kind": kind, "elem": elem, "n": _log_int(rng, 16, 500), "iters": rng.randint(5, 20),
                "fix_boundary": fix, "quality": quality}
    if kind == "tet":
        n = _log_int(rng, 6, 80)
        return {"kind": kind, "n": n, "iters": rng.randint(2, 12), "refine": rng.choice([0.0, 0.05, 0.15, 0.3]),
                "fix_boundary": rng.random() < 0.7, "quality": "MIN_ANGLE" if n < 30 and rng.random() < 0.15 else "MEAN_RATIO"}
    if kind == "hex":
        return {"kind": kind, "n": _log_int(rng, 6, 40), "iters": rng.randint(3, 10), "fix_boundary": rng.random() < 0.7,
                "quality": "MEAN_RATIO"}
    if kind == "surface":
        if rng.random() < 0.5:
            return {"kind": kind, "elem": "tri", "level": rng.randint(3, 7), "iters": rng.randint(3, 10),
                    "noise": rng.choice([1e-3, 1e-4])}
        return {"kind": kind, "elem": "quad", "nu": _log_int(rng, 24, 512), "nv": _log_int(rng, 16, 256),
                "iters": rng.randint(3, 10), "noise": rng.choice([1e-3, 1e-4])}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 4, 256), "v_min": 500, "v_max": _log_int(rng, 1000, 50000),
                "iters": rng.randint(2, 5)}
    if kind == "learned":
        return {"kind": kind, "n": _log_int(rng, 10, 64), "iters": rng.randint(3, 10)}
    if kind == "train":
        return {"kind": kind, "batch": 128 * _log_int(rng, 4, 128), "steps": rng.randint(10, 50)}
    if kind == "build":
        elem = rng.choice(["tet", "tet", "hex", "tri", "quad"])
        top = {"tet": 60, "hex": 40, "tri": 500, "quad": 500}[elem]
        case = {"kind": kind, "elem": elem, "n": _log_int(rng, 8, top)}
        return {**case, "refine": rng.choice([0.0, 0.05, 0.15])} if elem == "tet" else case
    return {"kind": kind, "n": _log_int(rng, 10, 80)}


# ---- inputs ------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _tet_lattice(n, refine):
    """The mesh of ``meshgen.tet_cube`` without its jitter (made in less time); ``refine``: share
    of the tetrahedra that get a vertex at their centre."""
    m = n + 1
    k, j, i = np.meshgrid(*[np.arange(m, dtype=np.int32)] * 3, indexing="ij")
    xyz = np.stack([i.ravel(), j.ravel(), k.ravel()], 1) * (1.0 / n)
    base = ((k * m + j) * m + i)[:n, :n, :n].reshape(-1)
    step = [1, m, m * m]
    el = np.empty((n ** 3, 6, 4), np.int32)
    for t, p in enumerate([(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]):
        b = step[p[0]]
        c = b + step[p[1]]
        even = (p[1] - p[0]) % 3 == 1
        for corner, off in enumerate([0, b if even else c, c if even else b, c + step[p[2]]]):
            np.add(base, off, out=el[:, t, corner])
    el = el.reshape(-1, 4)
    if refine > 0:
        pick = np.random.default_rng(n).random(len(el)) < refine
        split = el[pick]
        centre = len(xyz) + np.arange(len(split), dtype=np.int32)
        xyz = np.concatenate([xyz, xyz[split].mean(1)])
        parts = []
        for c in range(4):
            t = split.copy()
            t[:, c] = centre
            parts.append(t)
        el = np.concatenate([el[~pick]] + parts)
    free = np.all((xyz > 1e-9) & (xyz < 1 - 1e-9), axis=1)
    # new vertices sit in cells a quarter as tall: their jitter is smaller
    scale = np.where(np.arange(len(xyz)) < (n + 1) ** 3, 0.3, 0.06) / n
    if refine > 0:
        scale *= 0.5
    return xyz, np.ascontiguousarray(el, np.int32), free, scale


@functools.lru_cache(maxsize=None)
def _hex_lattice(n):
    xyz, el = G.hex_cube(n, None)
    xyz = xyz.astype(np.float64)
    return xyz, el, np.all((xyz > 1e-9) & (xyz < 1 - 1e-9), axis=1), np.full(len(xyz), 0.3 / n)


@functools.lru_cache(maxsize=None)
def _surface(elem, a, b):
    return G.icosphere(a) if elem == "tri" else G.torus_quads(a, b)


def _points(case, seed):
    """(points, elements, element type) of a case's mesh, the points jittered by the seed."""
    kind = case["kind"]
    elem = case.get("elem", "hex" if kind == "hex" else "tet")
    if kind == "surface":
        xyz, el = _surface(elem, case.get("level", case.get("nu")), case.get("nv", 0))
        tangential = 0.35 if elem == "tri" or case["noise"] >= 1e-3 else 0.2
        return G.perturb_surface(xyz, el, seed, tangential, case["noise"], normal_absolute=True), el, \
            _capi.TRI if elem == "tri" else _capi.QUAD
    if elem == "tri":
        return *G.tri_grid(case["n"], seed, 0.4), _capi.TRI
    if elem == "quad":
        return *G.quad_grid(case["n"], seed, 0.4), _capi.QUAD
    xyz, el, free, scale = _hex_lattice(case["n"]) if elem == "hex" else _tet_lattice(case["n"], case.get("refine", 0.0))
    u = np.random.default_rng(seed).uniform(-1.0, 1.0, size=(len(xyz), 3)) * (scale * free)[:, None]
    return (xyz + u).astype(np.float32), el, _capi.HEX if elem == "hex" else _capi.TET


_MESH = {_capi.TRI: V.DMOMeshTri, _capi.QUAD: V.DMOMeshQuad, _capi.TET: V.DMOMeshTet, _capi.HEX: V.DMOMeshHex}


class _Handle:
    """An optimiser that a program keeps, with the positions of its next run on the device."""

    def __init__(self, case, seed):
        xyz, el, kind = _points(case, seed)
        self.mesh = _MESH[kind](xyz, el)
        self.x = torch.from_numpy(np.ascontiguousarray(xyz)).cuda()
        self.out = torch.empty_like(self.x)
        self.iters = case.get("iters", 0)
        quality = getattr(V.QualityCriterium, case.get("quality", "MEAN_RATIO"))
        if case["kind"] == "surface":
            self.opt = (V.DMOTriClass if kind == _capi.TRI else V.DMOQuadClass)(self.mesh, n_iter=max(self.iters, 1))
        else:
            cls = {_capi.TRI: V.DMOTriFlatClass, _capi.QUAD: V.DMOQuadFlatClass, _capi.TET: V.DMOTetClass,
                   _capi.HEX: V.DMOHexClass}[kind]
            self.opt = cls(self.mesh, quality, n_iter=max(self.iters, 1), fix_boundary=case.get("fix_boundary", True))

    def run(self):
        _capi.check(_capi.lib().vsdmo_mesh_set_positions(self.mesh.h, C.c_void_p(self.x.data_ptr()), 1, _capi.DEVICE))
        self.opt.restart()
        self.opt.iterate(self.iters)
        self.mesh.positions_to_device(self.out.data_ptr())
        return {"positions": self.out, "min_quality": self.opt.getQuality()}


def _pairs(n, iters, seed):
    """Training pairs (ring, displacement) from plain iterations of a jittered cube."""
    xyz, el, _ = _points({"kind": "tet", "n": n}, seed)
    mesh = V.DMOMeshTet(xyz, el)
    opt = V.DMOTetClass(mesh, n_iter=iters)
    cap = (mesh.info["nV"] - mesh.info["nSurf"]) * iters
    feats = torch.empty(cap * 96, device="cuda")
    targets = torch.empty(cap * 3, device="cuda")
    torch.cuda.synchronize()
    rows = opt.collect_pairs(iters, feats.data_ptr(), targets.data_ptr(), cap)
    opt.close()
    mesh.close()
    return feats, targets, rows


def _train(model, data, steps, batch, lr, seed):
    return model.train(None, None, steps=steps, batch=batch, lr=lr, seed=seed,
                       device_ptrs=(data[0].data_ptr(), data[1].data_ptr()), n_rows=data[2])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        g = np.random.default_rng(case["count"])
        sizes = np.exp(g.uniform(math.log(case["v_min"]), math.log(case["v_max"]), size=case["count"]))
        meshes = []
        for i, v in enumerate(sizes):
            n = max(4, int(round(math.sqrt(v))))
            make = G.tri_grid if i % 2 == 0 else G.quad_grid
            meshes.append((_capi.TRI if i % 2 == 0 else _capi.QUAD, *make(n, seed=seed * 1000 + i, jitter=0.4)))
        batch = V.BatchDMO(meshes)
        x = torch.from_numpy(np.concatenate([m[1] for m in meshes])).cuda()
        return {"kind": kind, "batch": batch, "x": x, "out": torch.empty_like(x), "iters": case["iters"]}
    if kind == "train":
        return {"kind": kind, "data": _pairs(24, 12, seed), "model": V.ProposalModel(seed=seed), "case": dict(case)}
    if kind == "build":
        xyz, el, t = _points(case, seed)
        return {"kind": kind, "type": t, "xyz": torch.from_numpy(np.ascontiguousarray(xyz)).cuda(),
                "el": torch.from_numpy(np.ascontiguousarray(el)).cuda(), "out": torch.empty(xyz.shape, device="cuda")}
    if kind == "inspect":
        h = _Handle({"kind": "tet", "n": case["n"]}, seed)
        return {"kind": kind, "handle": h, "q": torch.empty(h.mesh.info["nE"], device="cuda")}
    h = _Handle({**case, "kind": "tet"} if kind == "learned" else case, seed)
    if kind == "learned":
        model = V.ProposalModel(seed=seed)
        _train(model, _pairs(20, 12, seed + 1), 1500, 4096, 1e-3, seed)
        h.opt.set_model(model)
    return {"kind": kind, "handle": h}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b, L = state["batch"], _capi.lib()
        _capi.check(L.vsdmo_batch_set_positions(b.h, C.c_void_p(state["x"].data_ptr()), _capi.DEVICE))
        b.restart()
        b.iterate(state["iters"])
        _capi.check(L.vsdmo_batch_get_positions(b.h, C.c_void_p(state["out"].data_ptr()), _capi.DEVICE))
        return {"positions": state["out"], "min_quality": b.stats(state["iters"])[0]}
    if kind == "train":
        c = state["case"]
        loss = _train(state["model"], state["data"], c["steps"], c["batch"], 1e-3, 7)
        return {"loss": loss, "params": state["model"].get_params()}
    if kind == "build":
        x, el = state["xyz"], state["el"]
        mesh = _MESH[state["type"]](None, None, device_ptrs=(x.data_ptr(), el.data_ptr(), len(x), len(el)))
        mesh.positions_to_device(state["out"].data_ptr(), original_order=False)
        out = {"positions": state["out"], "permutation": mesh.permutation(), "colors_free": mesh.array(V.A_COL_FREE),
               "colors_feature": mesh.array(V.A_COL_FEATURE), "colors_inner": mesh.array(V.A_COL_INNER)}
        mesh.close()
        return out
    h = state["handle"]
    if kind == "inspect":
        h.opt.getElementQualities(state["q"].data_ptr())
        low, mean = h.opt.quality_stats()
        return {"qualities": state["q"], "histogram": h.opt.getQualityHistogram(10), "min": low, "mean": mean}
    return h.run()


# ---- what a pass cannot do without --------------------------------------------------------------------

def _counts(case):
    """(vertices, vertices that move, elements, corners per element) of a case's mesh."""
    kind = case["kind"]
    elem = case.get("elem", "hex" if kind == "hex" else "tet")
    if kind == "surface":
        if elem == "tri":
            v = 10 * 4 ** case["level"] + 2
            return v, v, 2 * v - 4, 3
        v = case["nu"] * case["nv"]
        return v, v, v, 4
    n = case["n"]
    if elem in ("tri", "quad"):
        return n * n, (n - 2) ** 2, (n - 1) ** 2 * (2 if elem == "tri" else 1), 3 if elem == "tri" else 4
    e, extra = (n ** 3, 0) if elem == "hex" else (6 * n ** 3, int(6 * n ** 3 * case.get("refine", 0.0)))
    v = (n + 1) ** 3 + extra
    return v, (n - 1) ** 3 + extra, e + 3 * extra, 8 if elem == "hex" else 4


def work(case):
    kind = case["kind"]
    if kind == "train":
        b = case["batch"] * case["steps"]
        weights = 96 * 128 + 2 * 128 * 128 + 128 * 3
        return {"bytes": 4.0 * 99 * b, "flops": 6.0 * weights * b}
    if kind == "batch":
        span = math.log(case["v_max"] / case["v_min"])
        v = case["count"] * (case["v_max"] - case["v_min"]) / max(span, 1e-9)
        return {"bytes": 24.0 * v + 18.0 * 1.5 * v, "flops": v * case["iters"] * 3 * 64 * 12}
    v, moving, e, k = _counts(case)
    if kind == "build":
        # points and elements in; points, elements, ring records, colours and permutation out
        return {"bytes": 12.0 * v + 4.0 * k * e + 16.0 * v + 4.0 * k * e + 12.0 * k * e + 8.0 * v, "flops": 0}
    if kind == "inspect":
        return {"bytes": 12.0 * v + 16.0 * e + 4.0 * e, "flops": 60.0 * e}
    # every level judges every candidate by one element at least; every ring is set up once
    candidates = 3 * (512 if k in (4, 8) and kind in ("tet", "hex") else 64)
    if kind == "learned":
        candidates = 64
    flops = moving * case["iters"] * (candidates * 14 + 100 * k * e / max(v, 1))
    if kind == "learned":
        flops += moving * case["iters"] * 2.0 * (96 * 128 + 2 * 128 * 128 + 128 * 3)
    return {"bytes": 24.0 * v + 4.0 * k * e, "flops": float(flops)}


def exact(case, seed):
    """Element qualities and their statistics in 64 bits; the searches have no such value: which
    candidate wins a near tie depends on the rounding."""
    if case["kind"] != "inspect":
        return None
    xyz, el, _ = _points(case, seed)
    p = xyz.astype(np.float64)[el]
    e0, e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0], p[:, 3] - p[:, 0]
    vol = np.einsum("ij,ij->i", e0, np.cross(e1, e2)) / 6.0
    length = sum((d * d).sum(1) for d in (e0, e1, e2, e1 - e0, e2 - e0, e2 - e1))
    q = np.where(vol < 0, vol, 12.0 * np.cbrt(9.0 * vol * vol) / length)
    return {"qualities": q, "histogram": None, "min": float(q.min()), "mean": float(q.mean())}
