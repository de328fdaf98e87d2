"""The work that programs have this framework do, as cases to be timed.

A case is one call of a public entry point on seeded inputs:

* ``refine``: a CDT in host memory to its refined mesh in host memory
  (``refine.refine``, the GPU_Refine_Quality of the framework);
* ``cdt``: points and segments to their constrained Delaunay triangulation
  (``triangulate.build_cdt_gpu``);
* ``mesh``: points and segments to the refined mesh
  (``triangulate.triangulate_refine``);
* ``batch``: independent domains through the persistent engine
  (``refine.refine_batch_persistent``);
* ``train``: Adam training of the placement network on labelled candidates
  (``refine.mlp_train``).

Inputs follow the benchmark's configurations: uniform points, a mixture of 64
Gaussians with 10 % background, a jittered grid with concentric circles, and
batched domains of log-uniform size.

How many vertices a mesh gets depends on the input.  A mesh is returned whole,
in arrays whose shapes depend on the case alone: the rows that every such mesh
has are the library's own arrays, the rest is put into zero-filled arrays of
the caller's with room for the largest.
"""
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np

from gpu_cdt_refine_b200 import inputs, refine, triangulate

NET = os.path.join(os.path.dirname(refine.__file__), "data", "placement_mlp.npy")

RUPPERT, CHEW = 1, 0


def _refine(points, dist="clustered", theta=20.0, policy=refine.Offcenter, mode=RUPPERT, exact_pred=False,
            learned=False, area=0.0):
    """area: bound on a triangle's area in units of domain area / points (0: none)."""
    return {"kind": "refine", "points": points, "dist": dist, "theta": theta, "policy": policy, "mode": mode,
            "exact_pred": exact_pred, "learned": learned, "area": area}


def listed():
    return [
        # a single small part, as a mesher inside an interactive tool refines it: launch and host latency
        dict(_refine(500, "uniform"), name="refine_500"),
        # the small plain configuration: 10,000 uniform points, 500 segments
        dict(_refine(10_000, "uniform"), name="refine_10k"),
        # the other mode and the other insertion policy on an ordinary clustered input of an odd size
        dict(_refine(100_003, mode=CHEW, policy=refine.Circumcenter), name="refine_100k_chew_cc"),
        # the adversarial configuration (near-cocircular points) at a quarter of its size, exact predicates
        dict(_refine(245_000, "adversarial", theta=20.7, exact_pred=True), name="refine_245k_exact"),
        # the learned placement configuration at the size its network was trained on
        dict(_refine(200_000, learned=True), name="refine_200k_learned"),
        # the large clustered configuration: the benchmark's headline
        dict(_refine(2_000_000), name="refine_2m"),
        # triangulation of a small and of a large input
        {"name": "cdt_20k", "kind": "cdt", "points": 20_011, "dist": "uniform"},
        {"name": "cdt_1m", "kind": "cdt", "points": 1_000_000, "dist": "clustered"},
        # the whole flow, with an area bound as finite-element programs set it
        {"name": "mesh_300k_area", "kind": "mesh", "points": 301_117, "dist": "uniform", "theta": 20.0, "area": 0.6},
        # batched domains: a few, and more than the GPU has multiprocessors
        {"name": "batch_16", "kind": "batch", "domains": 16, "nmin": 200, "nmax": 50_000},
        {"name": "batch_256", "kind": "batch", "domains": 256, "nmin": 200, "nmax": 50_000},
        # training of the placement network (forward, backward, Adam) on an input's worth of candidates
        {"name": "train_100k", "kind": "train", "rows": 100_000, "epochs": 2, "batch": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["refine", "refine", "refine", "refine", "cdt", "mesh", "batch", "train"])
    dist = rng.choice(["uniform", "clustered", "clustered"])
    theta = rng.choice([15.0, 18.0, 20.0])
    if kind == "refine":
        c = _refine(_log(rng, 500, 1_000_000), dist, theta, rng.choice([refine.Circumcenter, refine.Offcenter]),
                    rng.choice([RUPPERT, CHEW]), rng.random() < 0.25)
        opt = rng.random()
        if opt < 0.15:  # the network places points between off-center and circumcenter
            c.update(learned=True, policy=refine.Offcenter)
        elif opt < 0.3:
            c.update(dist="uniform", area=rng.uniform(0.5, 1.5))
        elif opt < 0.4:
            c.update(dist="adversarial", points=_log(rng, 20_000, 400_000), theta=20.7, mode=RUPPERT,
                     policy=refine.Offcenter, exact_pred=rng.random() < 0.5)
        return c
    if kind == "cdt":
        return {"kind": "cdt", "points": _log(rng, 2_000, 1_000_000), "dist": dist}
    if kind == "mesh":
        return {"kind": "mesh", "points": _log(rng, 1_000, 500_000), "dist": dist, "theta": theta,
                "area": rng.uniform(0.5, 1.5) if dist == "uniform" else 0.0}
    if kind == "batch":
        return {"kind": "batch", "domains": _log(rng, 8, 256), "nmin": 200, "nmax": _log(rng, 2_000, 50_000)}
    return {"kind": "train", "rows": _log(rng, 5_000, 100_000), "epochs": rng.randint(1, 2),
            "batch": rng.choice([256, 1024, 4096])}


def _points(case, seed):
    n = case["points"]
    if case["dist"] == "uniform":
        return inputs.uniform_points(n, 0.0, 1000.0, seed)
    return inputs.cluster_points(n, 64, 1.0e4, 5.0, 200.0, 0.10, seed)


def _max_area(case):
    return case["area"] * 1.0e6 / case["points"] if case.get("area") else 0.0


def _domain(n, uniform, seed):
    rng = np.random.default_rng(seed)
    if uniform:
        pts = inputs.uniform_points(n, 0.0, 1000.0, seed)
    else:
        pts = inputs.cluster_points(n, int(rng.integers(1, 9)), 1000.0, 5.0, 100.0, 0.0, seed)
    return inputs.build_cdt(pts, inputs.pick_segments(pts, max(1, n // 20), seed + 1))


def _sizes(case):
    """Points of each domain of a batch: evenly over the logarithm of the range."""
    lo, hi, count = case["nmin"], case["nmax"], case["domains"]
    return [int(round(lo * (hi / lo) ** ((k + 0.5) / count))) for k in range(count)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        rng = np.random.default_rng(seed)
        n = case["rows"]
        # bounded features, and descendant-count-like targets that depend on them
        x = np.tanh(rng.normal(0.0, 0.7, (n, refine.MLP_FEATURES))).astype(np.float32)
        y = np.maximum(0.0, 1.5 + x[:, :8].sum(axis=1) + x[:, 25] * x[:, 3] + rng.normal(0, 0.5, n))
        return {"case": case, "params": refine.mlp_init(seed % 1000, float(y.mean())), "x": x,
                "y": y.astype(np.float32)}
    if kind == "batch":
        sizes = _sizes(case)
        with ThreadPoolExecutor(os.cpu_count() or 1) as ex:
            doms = list(ex.map(lambda k: _domain(sizes[k], k % 2 == 0, 2 * (seed + 1000 * k)), range(len(sizes))))
        order = np.random.default_rng(seed).permutation(len(doms))  # domains come in no order of size
        return {"case": case, "doms": [doms[k] for k in order], "thetas": [(15.0, 18.0, 20.0)[k % 3] for k in order],
                "keep": {}}
    if case["dist"] == "adversarial":
        g = max(16, int(round(math.sqrt(case["points"] / 2.0))))
        cdt = inputs.adversarial(seed, g=g, nc=max(4, g * 200 // 700), nseg=g * g // 25)
    else:
        pts = _points(case, seed)
        seg = inputs.pick_segments(pts, max(1, case["points"] // 20), seed + 1)
        if kind != "refine":
            return {"case": case, "pts": pts, "seg": seg, "keep": {}}
        cdt = triangulate.build_cdt_gpu(pts, seg)
    net = np.load(NET).astype(np.float32) if case["learned"] else None
    return {"case": case, "cdt": cdt, "net": net, "keep": {}}


def _room(case):
    """(points, triangles, segments) that every mesh of the case has, and that none exceeds."""
    n = case["points"]
    if case["kind"] == "cdt":
        return (n, 2 * n - 500, n // 20 - n // 200), (n, 2 * n, n // 20 + 500)
    low = {15.0: 1.45, 18.0: 1.75}.get(case["theta"], 2.03)
    high = 8.0 if case["dist"] == "adversarial" else low + 1.0
    return ((int(low * n), int(1.93 * low * n), int(0.15 * n)),
            (int(high * n) + 4000, int(2 * high * n) + 8000, int(high * n) // 2 + 1000))


def _arrays(cdt):
    return [cdt.pointlist, cdt.trianglelist, cdt.neighborlist, cdt.segmentlist]


def _kept(state, key, rows, like):
    buf = state["keep"].get(key)
    if buf is None:
        buf = state["keep"][key] = np.zeros((rows,) + like.shape[1:], like.dtype)
    return buf


def _mesh(state, cdt):
    (p0, t0, s0), (p1, t1, s1) = _room(state["case"])
    out = []
    for key, a, lo, hi in zip("ptns", _arrays(cdt), (p0, t0, t0, s0), (p1, t1, t1, s1)):
        head = a[:lo]
        if a.shape[0] < lo:
            head = _kept(state, key + "0", lo, a)
            head[:a.shape[0]] = a
        rest = _kept(state, key, hi - lo, a)
        k = max(0, a.shape[0] - lo)
        rest[:k] = a[lo:]
        rest[k:state["keep"].get(key + "k", k)] = 0  # rows of a longer earlier mesh
        state["keep"][key + "k"] = k
        out += [head, rest]
    return out + [cdt.numberofpoints, cdt.numberoftriangles, cdt.numberofsegments]


def _joined(state, meshes):
    """Each array of the meshes end to end, in arrays that the caller keeps."""
    out = []
    for key, most, arrs in zip("ptns", (3, 6, 6, 1), zip(*[_arrays(m) for m in meshes])):
        buf = _kept(state, key, most * sum(_sizes(state["case"])) + 4000, arrs[0])
        n = sum(a.shape[0] for a in arrs)
        np.concatenate(arrs, out=buf[:n])
        buf[n:state["keep"].get(key + "k", n)] = 0
        state["keep"][key + "k"] = n
        out.append(buf)
    return out + [np.array([[m.numberofpoints, m.numberoftriangles, m.numberofsegments] for m in meshes])]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "refine":
        pred = refine.PRED_EXACT if case["exact_pred"] else refine.PRED_REFERENCE
        mesh, _ = refine.refine(state["cdt"], case["theta"], case["policy"], case["mode"], predicates=pred,
                                mlp=state["net"], max_area=_max_area(case))
        return _mesh(state, mesh)
    if kind == "cdt":
        return _mesh(state, triangulate.build_cdt_gpu(state["pts"], state["seg"]))
    if kind == "mesh":
        mesh, _, _ = triangulate.triangulate_refine(state["pts"], state["seg"], case["theta"],
                                                    max_area=_max_area(case))
        return _mesh(state, mesh)
    if kind == "batch":
        meshes, _ = refine.refine_batch_persistent(state["doms"], state["thetas"])
        return _joined(state, meshes)
    params, loss = refine.mlp_train(state["params"], state["x"], state["y"], epochs=case["epochs"],
                                    batch=case["batch"], seed=0)
    return [params, np.array([loss], np.float32)]


def work(case):
    """Bytes of the input read once and of the output written once; operations:
    the predicates and constructions that the output's size asks for.  A
    refinement at these angles leaves about 2.1 vertices per input vertex."""
    kind = case["kind"]
    if kind == "train":  # two products of the network forward, four backward, for every row and epoch
        rows = case["rows"] * case["epochs"]
        return {"bytes": case["rows"] * 4 * 33 + 2 * 4 * 6337, "flops": rows * 6 * (32 * 64 + 64 * 64 + 64)}
    n = sum(_sizes(case)) if kind == "batch" else case["points"]
    raw = n * 16 + n / 20 * 8                    # points and segments
    cdt = n * 2 * 24                             # triangles and neighbours
    refined = 2.1 * n * (16 + 2 * 24) + n / 20 * 3 * 8
    if case.get("area"):
        refined *= max(1.0, 1.0 / case["area"])
    if kind == "cdt":
        return {"bytes": raw * 2 + cdt, "flops": n * 6 * 50}
    if kind == "mesh":
        return {"bytes": raw + refined, "flops": n * 6 * 50 + n * 6 * 150}
    return {"bytes": raw + cdt + refined, "flops": n * 6 * 150}


def exact(case, seed):
    """No case has one within seconds: a refined mesh and a triangulation are
    combinatorial (their arrays are compared bit for bit), and a trained
    network is the end of some hundred dependent 16-bit steps."""
    return None
