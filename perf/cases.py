"""The workloads whose speed this library is judged by: builds, searches and
batched clouds through the public Python API, from the smallest calls (where
launches and latency count) to the ten-million-point benchmark.

`listed()` gives the fixed cases, `draw(rng)` one more of the same ranges;
`prepare`, `run`, `work` and `exact` are described at each.
"""
import math

import numpy as np
import torch

import cudakdtree_b200 as ck

# record layouts in use: plain points (2 to 4 float or int coordinates), the
# benchmark's 16-byte {float3; payload with the split dim in bits 30..31}, and
# the reference's 32-byte {float4; int dim}
LAYOUTS = {
    "float2": ("float32", 2, 8, None), "float3": ("float32", 3, 12, None),
    "float4": ("float32", 4, 16, None), "int2": ("int32", 2, 8, None),
    "int3": ("int32", 3, 12, None), "int4": ("int32", 4, 16, None),
    "packed16": ("float32", 3, 16, (12, 30, 2)), "record32": ("float32", 4, 32, (16, 0, 32)),
}
METHODS = ("stack_based", "stack_free", "cct")


def listed():
    return [
        # one small cloud, built again for every frame or object: launches
        {"name": "build_1k", "op": "build", "n": 1000, "layout": "float3",
         "builder": "default", "data": "uniform"},
        # the headline benchmark's build: 10M clustered points with payload
        {"name": "build_10m", "op": "build", "n": 10_000_000, "layout": "packed16",
         "builder": "default", "data": "mixture"},
        # a build next to other large allocations: the bounded-memory builder
        {"name": "build_inplace_1m", "op": "build", "n": 1_000_003, "layout": "float4",
         "builder": "inplace", "data": "uniform"},
        # closest-point lookups (registration, snapping), a query per point
        {"name": "fcp_1m", "op": "fcp", "n": 1_000_000, "nq": 1_000_000, "k": 1,
         "layout": "float3", "method": "stack_free", "data": "uniform", "cutoff": 0.0},
        # an interactive lookup: a few hundred queries against a kept tree
        {"name": "knn_few", "op": "knn", "n": 100_000, "nq": 777, "k": 8,
         "layout": "float3", "method": "stack_based", "data": "uniform", "cutoff": 0.0},
        # the ordinary search: 1M points, 1M queries, a short list
        {"name": "knn_1m_k8", "op": "knn", "n": 1_000_000, "nq": 1_000_000, "k": 8,
         "layout": "float3", "method": "cct", "data": "uniform", "cutoff": 0.0},
        # the headline benchmark's search
        {"name": "knn_10m_k16", "op": "knn", "n": 10_000_000, "nq": 10_000_000, "k": 16,
         "layout": "packed16", "method": "stack_based", "data": "mixture", "cutoff": 0.0},
        # wide records and long lists (feature matching)
        {"name": "knn_float4_k64", "op": "knn", "n": 4_000_000, "nq": 500_000, "k": 64,
         "layout": "record32", "method": "stack_based", "data": "wide", "cutoff": 0.0},
        # integer coordinates (voxels, quantised scans), long lists
        {"name": "knn_int3_k64", "op": "knn", "n": 4_000_000, "nq": 500_000, "k": 64,
         "layout": "int3", "method": "stack_based", "data": "uniform", "cutoff": 0.0},
        # searches seeded by a trained radius model, k = 32, mixed queries
        {"name": "learned_k32", "op": "learned", "n": 4_000_000, "nq": 2_000_000, "k": 32,
         "layout": "packed16", "method": "stack_based", "data": "mixture", "cutoff": 0.0},
        # many independent clouds built and searched in one call
        {"name": "clouds_1k", "op": "clouds", "clouds": 1024, "lo": 256, "hi": 65536,
         "queries": 1024, "k": 8},
        # the spatial tree: built and searched (a frame of a moving point set)
        {"name": "spatial_1m", "op": "spatial", "n": 1_000_000, "nq": 500_000, "k": 8,
         "layout": "float3", "method": "cct", "data": "mixture", "cutoff": 0.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["build", "build", "fcp", "knn", "knn", "knn", "knn", "learned", "clouds",
                     "spatial"])
    if op == "clouds":
        return {"op": op, "clouds": _log_int(rng, 16, 1024), "lo": _log_int(rng, 32, 1024),
                "hi": _log_int(rng, 4096, 65536), "queries": _log_int(rng, 32, 1024),
                "k": _log_int(rng, 1, 16)}
    if op == "build":
        builder = rng.choice(["default", "default", "thrust", "bitonic", "inplace"])
        return {"op": op, "n": _log_int(rng, 100, 4_000_000 if builder in ("bitonic", "inplace")
                                        else 10_000_000),
                "layout": rng.choice(sorted(LAYOUTS)), "builder": builder,
                "data": rng.choice(["uniform", "mixture"])}
    c = {"op": op, "n": _log_int(rng, 1000, 10_000_000), "nq": 0, "k": 1,
         "layout": rng.choice(sorted(LAYOUTS)), "method": rng.choice(METHODS),
         "data": rng.choice(["uniform", "mixture"]), "cutoff": 0.0}
    if op == "fcp":
        c["nq"] = _log_int(rng, 100, 2_000_000)
    elif op == "knn":
        c["k"] = _log_int(rng, 1, 128)
        c["nq"] = _log_int(rng, 100, 20_000_000 // max(4, c["k"]))
    elif op == "learned":
        c["layout"] = rng.choice(["float2", "float3", "packed16", "float4", "int3"])
        c["n"] = _log_int(rng, 50_000, 4_000_000)
        c["k"] = _log_int(rng, 4, 64)
        c["nq"] = _log_int(rng, 10_000, 20_000_000 // max(4, c["k"]))
    else:  # spatial
        c["layout"] = rng.choice(["float2", "float3", "float4"])
        c["method"] = rng.choice(["stack_based", "cct"])
        c["n"] = _log_int(rng, 1000, 2_000_000)
        c["k"] = _log_int(rng, 1, 32)
        c["nq"] = _log_int(rng, 100, 500_000)
    if op in ("fcp", "knn") and rng.random() < 0.25:
        # searches within a radius: some find their k points, some do not
        c["cutoff"] = 0.02
    return c


def _layout(name):
    scalar, dims, stride, dim = LAYOUTS[name]
    off, shift, bits = dim if dim else (-1, 0, 32)
    return ck.layout_for(scalar, dims, stride=stride, dim_offset=off, dim_shift=shift,
                         dim_bits=bits)


def _coords(n, name, data, gen, mixed=0.0):
    """[n, D] coordinates: uniform in the unit cube; a mixture of 64 Gaussians
    (sigma 0.01; a share `mixed` of them uniform); `wide`: uniform xyz and a
    normal fourth coordinate.  Integer layouts scale them to +-2^20."""
    scalar, dims, _, _ = LAYOUTS[name]
    p = torch.rand((n, dims), device="cuda", generator=gen)
    if data == "mixture":
        centre_gen = torch.Generator(device="cuda")
        centre_gen.manual_seed(3)
        centres = torch.rand((64, dims), device="cuda", generator=centre_gen)
        which = torch.randint(0, 64, (n,), device="cuda", generator=gen)
        g = centres[which] + 0.01 * torch.randn((n, dims), device="cuda", generator=gen)
        keep = torch.rand((n, 1), device="cuda", generator=gen) < mixed
        p = torch.where(keep, p, g)
    elif data == "wide":
        p[:, 3] = torch.randn(n, device="cuda", generator=gen)
    if scalar == "int32":
        return ((p * 2 - 1) * 2 ** 20).to(torch.int32)
    return p


def _records(coords, name):
    """The record array (int32 words for records with more than the point)."""
    _, dims, stride, dim = LAYOUTS[name]
    if dim is None:
        return coords.contiguous()
    n = coords.shape[0]
    rec = torch.zeros((n, stride // 4), dtype=torch.int32, device=coords.device)
    rec[:, :dims] = coords.view(torch.int32)
    if dim[2] < 32:  # payload: the input index
        rec[:, dim[0] // 4] = torch.arange(n, dtype=torch.int32, device=coords.device)
    return rec


def _cloud_sizes(case):
    """Cloud sizes log-uniform in [lo, hi), the same for every seed (a plan
    is made for sizes)."""
    rng = np.random.Generator(np.random.MT19937(5))
    return np.floor(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]),
                                       size=case["clouds"]))).astype(np.int64)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] == "clouds":
        offs = np.concatenate([[0], np.cumsum(_cloud_sizes(case))]).astype(np.int64)
        return (torch.rand((int(offs[-1]), 3), device="cuda", generator=gen),
                torch.rand((case["clouds"] * case["queries"], 3), device="cuda", generator=gen),
                offs)
    pts = _coords(case["n"], case["layout"], case["data"], gen)
    if case["op"] == "build":
        return (pts,)
    mixed = 0.3 if case["op"] == "learned" else 0.0
    return pts, _coords(case["nq"], case["layout"], case["data"], gen, mixed)


def _cutoff(case):
    """Search radius options of fcp / knn (none: unbounded)."""
    if not case.get("cutoff"):
        return {}
    if LAYOUTS[case["layout"]][0] == "int32":
        return {"cutoff_d2": int((case["cutoff"] * 2 ** 21) ** 2)}
    return {"cutoff": case["cutoff"]}


def prepare(case, seed):
    """What a program holds before the call: points, queries, and for the
    searches the built tree (with its plan or trained model)."""
    op = case["op"]
    if op == "clouds":
        pts, queries, offs = _inputs(case, seed)
        qoffs = np.arange(case["clouds"] + 1, dtype=np.int64) * case["queries"]
        plan = ck.BatchPlan(offs, qoffs, num_dims=3, k=case["k"])
        return {"case": case, "pts": pts, "work": torch.empty_like(pts), "queries": queries,
                "plan": plan}
    lay = _layout(case["layout"])
    if op == "build":
        rec = _records(_inputs(case, seed)[0], case["layout"])
        return {"case": case, "layout": lay, "pts": rec, "work": torch.empty_like(rec)}
    pts, queries = _inputs(case, seed)
    if op == "spatial":
        return {"case": case, "layout": lay, "pts": pts.contiguous(), "queries": queries}
    tree = _records(pts, case["layout"])
    bounds = ck.build_tree(tree, layout=lay)
    state = {"case": case, "layout": lay, "tree": tree, "bounds": bounds, "queries": queries}
    if op == "learned":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed + 1)
        train = _coords(100_000, case["layout"], case["data"], gen, 0.3)
        model = ck.RadiusModel(seed=1, quantile=0.9, num_dims=LAYOUTS[case["layout"]][1])
        model.fit(tree, train, case["k"], layout=lay, world_bounds=bounds, epochs=5)
        state["model"] = model
    return state


def run(state):
    """One pass.  Builds: the unbuilt records are restored, then built in
    place (records, world bounds).  Searches: (ids, squared distances)."""
    case = state["case"]
    op = case["op"]
    if op == "build":
        state["work"].copy_(state["pts"])
        bounds = ck.build_tree(state["work"], layout=state["layout"], builder=case["builder"])
        return state["work"], bounds
    if op == "clouds":
        state["work"].copy_(state["pts"])
        ids, d2 = state["plan"].run(state["work"], state["queries"])
        return state["work"], ids, d2
    if op == "spatial":
        tree = ck.spatial_build(state["pts"], state["layout"])
        ids, d2 = tree.knn(state["queries"], case["k"], case["method"])
        return tree.prim_ids(), ids, d2
    if op == "fcp":
        return ck.fcp(state["tree"], state["queries"], case["method"], layout=state["layout"],
                      world_bounds=state["bounds"], with_d2=True, **_cutoff(case))
    if op == "learned":
        return ck.knn_learned(state["tree"], state["queries"], case["k"], state["model"],
                              case["method"], layout=state["layout"],
                              world_bounds=state["bounds"])[:2]
    return ck.knn(state["tree"], state["queries"], case["k"], case["method"],
                  layout=state["layout"], world_bounds=state["bounds"], **_cutoff(case))


def work(case):
    """Bytes: inputs read and outputs written once (of a tree no more nodes
    than the queries' paths and answers name).  Flops: a squared distance
    for every point on a path and in an answer; a build compares."""
    if case["op"] == "clouds":
        total, nq = int(_cloud_sizes(case).sum()), case["clouds"] * case["queries"]
        return {"bytes": 2 * 12 * total + nq * (12 + 8 * case["k"]),
                "flops": 8 * nq * (case["k"] + math.log2(max(2, total / case["clouds"])))}
    scalar, dims, stride, _ = LAYOUTS[case["layout"]]
    n = case["n"]
    if case["op"] == "build":
        return {"bytes": 2 * n * stride + 8 * dims, "flops": n * math.log2(max(2, n))}
    nq, k = case["nq"], case["k"]
    nodes = nq * (k + math.log2(max(2, n)))
    answer = 4 + (8 if scalar == "int32" else 4)
    done = {"bytes": min(n, nodes) * stride + nq * (4 * dims + answer * k),
            "flops": nodes * 3 * dims}
    if case["op"] == "spatial":  # reads all points, writes a permutation and nodes
        done["bytes"] = n * (stride + 4 + 12 / 4) + nq * (4 * dims + answer * k)
    return done


def _nearest_d2(pts, queries, k, cutoff2):
    """[nq, k] ascending squared distances in 64 bits, cut off at cutoff2."""
    pts, queries = pts.double(), queries.double()
    out = []
    step = max(1, 2 ** 27 // max(1, pts.shape[0]))
    for i in range(0, queries.shape[0], step):
        q = queries[i:i + step]
        d2 = torch.zeros((q.shape[0], pts.shape[0]), dtype=torch.float64, device=pts.device)
        for d in range(pts.shape[1]):
            d2 += (q[:, d:d + 1] - pts[None, :, d]) ** 2
        near = d2.topk(min(k, pts.shape[0]), dim=1, largest=False, sorted=True).values
        if near.shape[1] < k:
            near = torch.nn.functional.pad(near, (0, k - near.shape[1]), value=math.inf)
        out.append(torch.where(near < cutoff2, near, cutoff2))
    return torch.cat(out)


def exact(case, seed):
    """World bounds of a build, squared distances of a search (by comparing
    every query with every point, where that is quick enough)."""
    op = case["op"]
    if op == "build":
        p = _inputs(case, seed)[0].double()
        return None, torch.stack([p.min(0).values, p.max(0).values])
    if op == "clouds":
        sizes = _cloud_sizes(case)
        if int((sizes * case["queries"]).sum()) > 2 ** 34 or case["clouds"] > 2048:
            return None
        pts, queries, offs = _inputs(case, seed)
        m = case["queries"]
        d2 = torch.cat([_nearest_d2(pts[offs[c]:offs[c + 1]], queries[c * m:(c + 1) * m],
                                    case["k"], math.inf) for c in range(case["clouds"])])
        return None, None, d2
    if case["n"] * case["nq"] > 2 ** 34 or LAYOUTS[case["layout"]][0] == "int32":
        return None
    pts, queries = _inputs(case, seed)
    cut = float(np.float32(case["cutoff"]) * np.float32(case["cutoff"])) or math.inf
    d2 = _nearest_d2(pts, queries, case["k"], cut)
    if op == "spatial":
        return None, None, d2
    return None, d2[:, 0] if op == "fcp" else d2
