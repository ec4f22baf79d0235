"""The work that programs built on this library have it do, as timed cases.

Every case goes through the public Python interface (``atrbvh_b200``): rebuilds
of a scene through a build plan, builds through the builder classes, segmented
batches, refits of a resident tree, ray queries, whole frames of rays and the
serving loop.  All cases of one process share one context, as a program with
one GPU stream does.

Builds, refits and traversal are discrete (comparisons, minima, maxima, and
single-precision arithmetic in a fixed order), so every output is compared
exactly; where 64-bit arithmetic gives the same quantity another way (the hit
distances of a small ray query), ``exact`` does so.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import atrbvh_b200 as ab

SCENES = {"uniform": ab.SCENE_UNIFORM, "clustered": ab.SCENE_CLUSTERED}

_shared: dict = {}


def _ctx() -> ab.Context:
    if "ctx" not in _shared:
        _shared["ctx"] = ab.Context(0)
    return _shared["ctx"]


def _server() -> ab.Server:
    """The process's request server: three lanes, ATRBVH(9,2), 24 GB."""
    if "server" not in _shared:
        _shared["server"] = ab.Server(0, hbm_budget=24 << 30, lanes=3, max_batch_requests=32)
        _shared["mesh_id"] = 0
    return _shared["server"]


class _Raw:
    """Device memory of the library, for torch to wrap without a copy; the
    object that owns it lives as long as the tensor."""

    def __init__(self, owner, ptr: int, shape: tuple, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 2,
                                         "strides": None}


def _wrap(owner, ptr, shape, typestr="<i4") -> torch.Tensor:
    return torch.as_tensor(_Raw(owner, int(ptr), shape, typestr), device="cuda")


def _tree_arrays(owner, view, nodes: int) -> dict:
    i4 = {k: _wrap(owner, getattr(view, k), (nodes,)) for k in ("parent", "left", "right", "data")}
    return {**i4, "bbox_min": _wrap(owner, view.bbox_min, (nodes, 4), "<f4"),
            "bbox_max": _wrap(owner, view.bbox_max, (nodes, 4), "<f4"),
            "area": _wrap(owner, view.area, (nodes,), "<f4")}


def _collapsed_arrays(owner, view, n: int) -> dict:
    return {"data": _wrap(owner, view.data, (2 * n - 1,)),
            "triangle_count": _wrap(owner, view.triangle_count, (2 * n - 1,)),
            "triangle_indices": _wrap(owner, view.triangle_indices, (n,))}


def _compact_arrays(owner, view, nodes: int, woop: int) -> dict:
    """The layout's first `nodes` node records and `woop` Woop entries."""
    return {"nodes": _wrap(owner, view.nodes, (nodes, 16)), "woop": _wrap(owner, view.woop, (woop, 4), "<f4"),
            "tri_index": _wrap(owner, view.tri_index, (woop,)), "num_nodes": view.num_nodes, "num_woop": view.num_woop}


def _ray_results(n: int) -> tuple[torch.Tensor, dict]:
    """A result buffer of n rays (int4 each) and views of its triangle ids and distances."""
    buf = torch.zeros((n, 4), dtype=torch.int32, device="cuda")
    return buf, {"triangle": buf[:, 0], "t": buf.view(torch.float32)[:, 1]}


def _cuda(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(a).cuda()


# ---- the cases -------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # A small movable object rebuilt every frame through its plan, then
        # handed to the tracer (the layout's sizes are read): the smallest build.
        dict(name="rebuild_1k", kind="rebuild", n=1003, scene="uniform", bits=30, treelet=9, iterations=2, max_leaf=0,
             flatten=True),
        # The plain single build: 65,536 uniform triangles, leaves of at most 4.
        dict(name="rebuild_64k", kind="rebuild", n=65536, scene="uniform", bits=30, treelet=9, iterations=2, max_leaf=4,
             flatten=False),
        # The benchmark's scene: a whole level rebuilt with its traversal layout.
        dict(name="rebuild_4m", kind="rebuild", n=4194304, scene="clustered", bits=30, treelet=9, iterations=2,
             max_leaf=0, flatten=True),
        # The largest scene of the quality sweep, to node arrays.
        dict(name="rebuild_16m", kind="rebuild", n=16777216, scene="uniform", bits=30, treelet=9, iterations=2,
             max_leaf=0, flatten=False),
        # A renderer loading a scene: builder classes one after another, 63-bit
        # codes, an odd triangle count.
        dict(name="load_1m_63bit", kind="load", n=1000003, scene="clustered", bits=63, optimizer="atrbvh", treelet=9,
             iterations=2, max_leaf=4),
        # The other optimiser: offline quality build of a medium mesh.
        dict(name="load_300k_trbvh", kind="load", n=300007, scene="uniform", bits=30, optimizer="trbvh", treelet=7,
             iterations=3, max_leaf=8),
        # Many meshes of very uneven sizes built at once and queried together.
        dict(name="batch_512", kind="batch", meshes=512, largest=262144, sizes=0, treelet=9, iterations=2, rays=500009),
        # A deforming mesh: new vertices every frame, boxes refitted.
        dict(name="refit_1m", kind="refit", n=1000003, scene="uniform", bits=30),
        # A handful of picking rays against a resident mesh: the smallest call.
        dict(name="pick_1k", kind="query", n=20011, scene="uniform", rays=1000, any_hit=False, sort=False),
        # Incoherent rays sorted for coherence, then traced.
        dict(name="query_1m_sorted", kind="query", n=500009, scene="uniform", rays=1000003, any_hit=False, sort=True),
        # A frame of the benchmark: primary rays, one diffuse bounce, and two
        # ambient-occlusion rays per pixel (any hit) in batches of 2^20.
        dict(name="frame_1080p", kind="frame", n=4194304, scene="clustered", width=1920, height=1080, ao=2),
        # The serving loop under a burst: builds kept resident, then refits,
        # each with its rays, host memory to host memory.
        dict(name="serve_16", kind="serve", builds=16, refits=8, largest=200000, sizes=0, rays=65536),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["rebuild", "rebuild", "rebuild", "load", "load", "batch", "refit", "query", "query", "frame",
                       "serve"])
    scene = rng.choice(["uniform", "clustered"])
    if kind == "rebuild":
        return dict(kind=kind, n=_log_int(rng, 1000, 8 << 20), scene=scene, bits=rng.choice([30, 30, 63]),
                    treelet=rng.choice([5, 7, 9, 9]), iterations=rng.choice([1, 2, 2, 3]),
                    max_leaf=rng.choice([0, 0, 4, 8]), flatten=rng.choice([True, False]))
    if kind == "load":
        opt = rng.choice(["none", "atrbvh", "atrbvh", "trbvh"])
        return dict(kind=kind, n=_log_int(rng, 2000, 1 << 20), scene=scene, bits=rng.choice([30, 63]), optimizer=opt,
                    treelet=7 if opt == "trbvh" else rng.choice([5, 7, 9, 9]), iterations=rng.choice([1, 2, 3]),
                    max_leaf=rng.choice([4, 4, 8, 16]))
    if kind == "batch":
        return dict(kind=kind, meshes=_log_int(rng, 16, 500), largest=_log_int(rng, 4096, 262144),
                    sizes=rng.randrange(1000), treelet=rng.choice([5, 7, 9, 9]), iterations=rng.choice([1, 2, 2]),
                    rays=_log_int(rng, 1000, 1 << 20))
    if kind == "refit":
        return dict(kind=kind, n=_log_int(rng, 1000, 4 << 20), scene=scene, bits=rng.choice([30, 63]))
    if kind == "query":
        return dict(kind=kind, n=_log_int(rng, 2000, 1 << 20), scene=scene, rays=_log_int(rng, 200, 2 << 20),
                    any_hit=rng.choice([False, False, True]), sort=rng.choice([False, True]))
    if kind == "frame":
        return dict(kind=kind, n=_log_int(rng, 10000, 4 << 20), scene=scene, width=rng.randrange(160, 1921),
                    height=rng.randrange(120, 1081), ao=rng.choice([1, 2]))
    return dict(kind=kind, builds=rng.randrange(4, 17), refits=rng.randrange(1, 5),
                largest=_log_int(rng, 10000, 200000), sizes=rng.randrange(1000), rays=_log_int(rng, 4096, 65536))


# ---- inputs ----------------------------------------------------------------------

def _prepare_rebuild(c: dict, seed: int) -> dict:
    scene = ab.SceneWrapper(_ctx(), ab.gen_scene(SCENES[c["scene"]], c["n"], seed))
    plan = ab.BuildPlan(scene, morton_bits=c["bits"], optimizer=ab.Batch.ATRBVH, treelet=c["treelet"],
                        iterations=c["iterations"], max_leaf=c["max_leaf"], flatten=c["flatten"])
    n, owner = c["n"], (plan, scene)
    out = {"tree": _tree_arrays(owner, plan.tree().view(), 2 * n - 1),
           "collapsed": _collapsed_arrays(owner, plan.collapsed().view(), n)}
    if c["flatten"]:
        # The first build, at load time.  Outputs cover the plan's buffers to
        # their capacity: the unused ends, which no run writes, are cleared.
        plan.run(graph=False)
        out["compact"] = _compact_arrays(owner, plan.compact().view(), n - 1, 4 * n)
        for k in ("nodes", "woop", "tri_index"):
            out["compact"][k].zero_()
    return {"scene": scene, "plan": plan, "out": out}


def _prepare_load(c: dict, seed: int) -> dict:
    return {"scene": ab.SceneWrapper(_ctx(), ab.gen_scene(SCENES[c["scene"]], c["n"], seed))}


def _prepare_batch(c: dict, seed: int) -> dict:
    sizes = ab.gen_batch_sizes(c["meshes"], 256, c["largest"], c["sizes"])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    v = ab.gen_batch_scene(sizes, seed)
    batch = ab.Batch(_ctx(), v, off)
    # Each queried mesh gets a run of rays in its own box.
    rng = np.random.RandomState(seed % (1 << 31))
    groups = min(64, c["rays"])
    mesh = np.sort(rng.choice(c["meshes"], size=groups, replace=groups > c["meshes"])).astype(np.uint32)
    ray_off = np.linspace(0, c["rays"], groups + 1).astype(np.uint32)
    parts = []
    for g in range(groups):
        p = v[off[mesh[g]]:off[mesh[g] + 1], :, :3].reshape(-1, 3)
        k = int(ray_off[g + 1] - ray_off[g])
        parts.append(ab.gen_rays_random(k, p.min(axis=0), p.max(axis=0), seed + g))
    rays = _cuda(np.concatenate(parts))
    buf, hits = _ray_results(c["rays"])
    return {"batch": batch, "rays": rays, "ray_off": ray_off, "mesh": mesh, "buf": buf, "hits": hits,
            "nodes": 2 * int(off[-1]) - c["meshes"]}


def _prepare_refit(c: dict, seed: int) -> dict:
    v = ab.gen_scene(SCENES[c["scene"]], c["n"], seed)
    scene = ab.SceneWrapper(_ctx(), v)
    tree = ab.LBVHBuilder(c["bits"] == 63).BuildTree(scene)
    ab.AgglomerativeTreeletOptimizer(9, 2).Optimize(tree)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    moved = _cuda(v)
    moved[:, :, :3] += 0.001 * torch.randn((c["n"], 3, 3), generator=gen, device="cuda")
    return {"scene": scene, "tree": tree, "moved": moved, "out": _tree_arrays(tree, tree.view(), 2 * c["n"] - 1)}


def _resident_layout(c: dict, seed: int) -> tuple:
    v = ab.gen_scene(SCENES[c["scene"]], c["n"], seed)
    scene = ab.SceneWrapper(_ctx(), v)
    tree = ab.LBVHBuilder(False).BuildTree(scene)
    ab.AgglomerativeTreeletOptimizer(9, 2).Optimize(tree)
    collapsed, _ = ab.BVHTreeCollapser().Collapse(tree)
    return scene, ab.CudaBVH(collapsed, scene)


def _query_rays(c: dict, seed: int, scene: ab.SceneWrapper) -> np.ndarray:
    return _segment_rays(c, seed, *scene.bounds())


def _segment_rays(c: dict, seed: int, lo, hi) -> np.ndarray:
    """Random rays in the scene's box, of a length that leaves it."""
    rays = ab.gen_rays_random(c["rays"], lo, hi, seed + 1)
    rays[:, 1, 3] = 4.0
    return rays


def _prepare_query(c: dict, seed: int) -> dict:
    scene, bvh = _resident_layout(c, seed)
    n = c["rays"]
    buf, hits = _ray_results(n)
    s = {"scene": scene, "bvh": bvh, "rays": _cuda(_query_rays(c, seed, scene)), "buf": buf, "hits": hits}
    if c["sort"]:
        s["sorted"] = torch.empty((n, 2, 4), dtype=torch.float32, device="cuda")
        s["slot_to_id"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["id_to_slot"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return s


AO_BATCH = 1 << 20


def _prepare_frame(c: dict, seed: int) -> dict:
    scene, bvh = _resident_layout(c, seed)
    n = c["width"] * c["height"]
    s = {"scene": scene, "bvh": bvh, "seed": seed, "rays": _cuda(ab.gen_rays_pinhole(c["width"], c["height"])),
         "bounce": torch.empty((n, 2, 4), dtype=torch.float32, device="cuda"),
         "ao_rays": torch.empty((AO_BATCH, 2, 4), dtype=torch.float32, device="cuda")}
    s["primary"], primary = _ray_results(n)
    s["indirect"], indirect = _ray_results(n)
    s["ao_hits"], ao = _ray_results(n * c["ao"])
    s["out"] = {"primary": primary, "bounce": s["bounce"], "indirect": indirect, "ao": ao}
    return s


def _prepare_serve(c: dict, seed: int) -> dict:
    server = _server()
    rng = np.random.RandomState(seed % (1 << 31))
    meshes, moved, rays = [], [], []
    for k, n in enumerate(ab.gen_batch_sizes(c["builds"], 1000, c["largest"], c["sizes"])):
        v = ab.gen_scene(ab.SCENE_UNIFORM, int(n), seed * 64 + k)
        meshes.append(ab.pinned_like(v))
        rays.append(ab.pinned_like(ab.gen_rays_random(c["rays"], (0, 0, 0), (1, 1, 1), seed * 64 + k).reshape(-1, 8)))
        if k < c["refits"]:
            w = v.copy()
            w[:, :, :3] += rng.normal(0.0, 0.001, size=w[:, :, :3].shape).astype(np.float32)
            moved.append(ab.pinned_like(w))
    results = ab.pinned_like(np.zeros((c["builds"] + c["refits"], c["rays"], 4), np.int32))
    first = _shared["mesh_id"] + 1
    _shared["mesh_id"] += c["builds"]
    return {"server": server, "meshes": meshes, "moved": moved, "rays": rays, "results": results, "first": first}


def prepare(case: dict, seed: int) -> dict:
    make = {"rebuild": _prepare_rebuild, "load": _prepare_load, "batch": _prepare_batch, "refit": _prepare_refit,
            "query": _prepare_query, "frame": _prepare_frame, "serve": _prepare_serve}[case["kind"]]
    s = make(case, seed)
    s["case"] = case
    _ctx().synchronize()
    torch.cuda.synchronize()  # torch's copies ran on its own stream
    return s


# ---- one pass ----------------------------------------------------------------------

def _run_rebuild(s: dict) -> dict:
    s["plan"].run()
    if not s["case"]["flatten"]:
        return s["out"]
    view = s["plan"].compact().view()  # the layout's sizes, for the tracer
    return {**s["out"], "compact": {**s["out"]["compact"], "num_nodes": view.num_nodes, "num_woop": view.num_woop}}


def _run_load(s: dict) -> dict:
    c, scene = s["case"], s["scene"]
    tree = ab.LBVHBuilder(c["bits"] == 63).BuildTree(scene)
    if c["optimizer"] == "atrbvh":
        ab.AgglomerativeTreeletOptimizer(c["treelet"], c["iterations"]).Optimize(tree)
    elif c["optimizer"] == "trbvh":
        ab.TRBVHOptimizer(c["treelet"], c["iterations"]).Optimize(tree)
    collapsed, sah = ab.BVHTreeCollapser().Collapse(tree, max_leaf=c["max_leaf"])
    bvh = ab.CudaBVH(collapsed, scene)
    # How much of the layout is used depends on the scene.  Leaves hold at most
    # max_leaf triangles, so this much of it always is.
    n = c["n"]
    return {"tree": _tree_arrays(tree, tree.view(), 2 * n - 1),
            "collapsed": _collapsed_arrays(collapsed, collapsed.view(), n), "sah": sah,
            "compact": _compact_arrays(bvh, bvh.view(), -(-n // c["max_leaf"]) - 1, 3 * n + 1)}


def _run_batch(s: dict) -> dict:
    c, b = s["case"], s["batch"]
    b.build(ab.Batch.ATRBVH, c["treelet"], c["iterations"], graph=True)
    sah = b.collapse()
    b.flatten()
    b.trace(s["rays"].data_ptr(), c["rays"], s["ray_off"], s["mesh"], s["buf"].data_ptr())
    v = ab.TreeView()
    ab.check(ab.lib().atr_batch_mesh_view(b.handle, 0, ab.C.byref(v)))
    return {"trees": _tree_arrays(b, v, s["nodes"]), "sah": sah, "hits": s["hits"]}


def _run_refit(s: dict) -> dict:
    s["scene"].set_vertices(device_ptr=s["moved"].data_ptr())
    ab.Refit(s["tree"], s["scene"])
    return s["out"]


def _run_query(s: dict) -> dict:
    c = s["case"]
    if not c["sort"]:
        s["bvh"].trace(s["rays"].data_ptr(), c["rays"], s["buf"].data_ptr(), any_hit=c["any_hit"])
        return s["hits"]
    ab.sort_rays(s["scene"].ctx, s["rays"].data_ptr(), c["rays"], s["sorted"].data_ptr(),
                 out_slot_to_id_ptr=s["slot_to_id"].data_ptr(), out_id_to_slot_ptr=s["id_to_slot"].data_ptr())
    s["bvh"].trace(s["sorted"].data_ptr(), c["rays"], s["buf"].data_ptr(), any_hit=c["any_hit"])
    return {"hits": s["hits"], "rays": s["sorted"], "slot_to_id": s["slot_to_id"], "id_to_slot": s["id_to_slot"]}


def _run_frame(s: dict) -> dict:
    c, scene, bvh = s["case"], s["scene"], s["bvh"]
    n, k = c["width"] * c["height"], c["ao"]
    bvh.trace(s["rays"].data_ptr(), n, s["primary"].data_ptr())
    ab.check(ab.lib().atr_gen_bounce_rays(scene.ctx.handle, scene.handle, s["rays"].data_ptr(), s["primary"].data_ptr(),
                                          n, s["seed"], s["bounce"].data_ptr()))
    bvh.trace(s["bounce"].data_ptr(), n, s["indirect"].data_ptr())
    for lo, hi in ab.ray_batches(n, k, AO_BATCH):
        ab.gen_ao_rays(scene, s["rays"].data_ptr(), s["primary"].data_ptr(), lo, hi - lo, k, 0.1, s["seed"],
                       s["ao_rays"].data_ptr())
        bvh.trace(s["ao_rays"].data_ptr(), (hi - lo) * k, s["ao_hits"].data_ptr() + 16 * lo * k, any_hit=True)
    return s["out"]


def _run_serve(s: dict) -> dict:
    c, server = s["case"], s["server"]
    # Refits follow their mesh's build; meshes of a pass before are replaced.
    tickets = [server.submit(ab.REQ_BUILD, s["first"] + k, s["meshes"][k], s["rays"][k], s["results"][k])
               for k in range(c["builds"])]
    done = [server.wait(t) for t in tickets]
    tickets = [server.submit(ab.REQ_REFIT, s["first"] + k, s["moved"][k], s["rays"][k], s["results"][c["builds"] + k])
               for k in range(c["refits"])]
    done += [server.wait(t) for t in tickets]
    for r in done:
        if r["status"] != ab.ATR_OK:
            raise RuntimeError(f"request failed: {r['error']}")
    return {"triangle": s["results"][:, :, 0], "t": s["results"].view(np.float32)[:, :, 1],
            "sah": [r["sah"] for r in done]}


def run(state: dict):
    go = {"rebuild": _run_rebuild, "load": _run_load, "batch": _run_batch, "refit": _run_refit, "query": _run_query,
          "frame": _run_frame, "serve": _run_serve}[state["case"]["kind"]]
    return go(state)


# ---- what a pass cannot do without ----------------------------------------------------

TREE = 104      # bytes of a triangle's two nodes: links, data, box, area
COLLAPSED = 20  # two data words, two counts, one list entry
COMPACT = 76    # a Woop triangle with its index entries, and a node for every four triangles
RAY = 48        # 32 bytes in, 16 out
VISIT = 4096    # bytes of layout that one ray looks at, at most


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "rebuild":
        return {"bytes": case["n"] * (48 + TREE + COLLAPSED + (COMPACT if case["flatten"] else 0)), "flops": 0}
    if kind == "load":
        return {"bytes": case["n"] * (48 + TREE + COLLAPSED + COMPACT), "flops": 0}
    if kind == "batch":
        n = (case["largest"] - 256) / math.log(case["largest"] / 256) * case["meshes"]  # log-uniform sizes
        return {"bytes": int(n * (48 + TREE + COLLAPSED + COMPACT)) + RAY * case["rays"], "flops": 0}
    if kind == "refit":
        # New vertices read and kept; links read, boxes and areas written.
        return {"bytes": case["n"] * (96 + 2 * (16 + 36)), "flops": 0}
    if kind == "query":
        r = case["rays"]
        sort = r * (32 + 32 + 8) if case["sort"] else 0
        return {"bytes": r * RAY + min(r * VISIT, case["n"] * COMPACT) + sort, "flops": 0}
    if kind == "frame":
        r = case["width"] * case["height"]
        layout = min(r * VISIT, case["n"] * COMPACT)
        return {"bytes": r * RAY * 2 + r * 32 + r * case["ao"] * (RAY + 32) + layout, "flops": 0}
    n = (case["largest"] - 1000) / math.log(case["largest"] / 1000)
    built = case["builds"] * n * (48 + TREE + COLLAPSED + COMPACT)
    rays = (case["builds"] + case["refits"]) * case["rays"]
    return {"bytes": int(built + case["refits"] * n * (48 + 104)) + rays * RAY, "flops": 0}


def tolerance(case: dict):
    return "exact"


# ---- the same in 64 bits ----------------------------------------------------------------

def exact(case: dict, seed: int):
    """Hit distances of an unsorted closest-hit query against every triangle,
    in 64 bits (the triangle, where two tie, is a matter of order)."""
    if case["kind"] != "query" or case["sort"] or case["any_hit"] or case["n"] * case["rays"] > 2e10:
        return None
    v = ab.gen_scene(SCENES[case["scene"]], case["n"], seed)
    p = v[:, :, :3].reshape(-1, 3)
    hi = np.maximum(p.max(axis=0), np.finfo(np.float32).tiny)
    rays = _cuda(_segment_rays(case, seed, p.min(axis=0), hi)).double()
    tri = _cuda(v)[:, :, :3].double()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    t_best = rays[:, 1, 3].clone()
    step = max(1, 20_000_000 // case["n"])
    for lo in range(0, case["rays"], step):
        o, d = rays[lo:lo + step, 0, :3, None], rays[lo:lo + step, 1, :3, None]

        def cross(x, y):
            return x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]

        dd = [d[:, k] for k in range(3)]
        e1k, e2k = [e1[:, k] for k in range(3)], [e2[:, k] for k in range(3)]
        s = [o[:, k] - a[:, k] for k in range(3)]
        h = cross(dd, e2k)
        det = e1k[0] * h[0] + e1k[1] * h[1] + e1k[2] * h[2]
        u = (s[0] * h[0] + s[1] * h[1] + s[2] * h[2]) / det
        q = cross(s, e1k)
        w = (dd[0] * q[0] + dd[1] * q[1] + dd[2] * q[2]) / det
        t = (e2k[0] * q[0] + e2k[1] * q[1] + e2k[2] * q[2]) / det
        tmin, tmax = rays[lo:lo + step, 0, 3, None], rays[lo:lo + step, 1, 3, None]
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > tmin) & (t < tmax)
        t_best[lo:lo + step] = torch.where(ok, t, tmax.expand_as(t)).min(dim=1).values
    return {"triangle": None, "t": t_best}
