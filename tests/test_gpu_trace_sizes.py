"""Traversal at the ray counts where a launch changes shape: rays per warp
follow the count (1, 2, 4, ... 32), warps fetch again, launches follow one
another on the context's ray counter; and at stack depths past the register and
the 16 entries in shared memory, in both stack sizes and over several meshes."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def deep(ctx):
    """A layout of more than 20 levels: points that close in on a corner, among others."""
    v = O.gen_scene(O.SCENE_UNIFORM, 3001, 4)
    k = np.arange(1500)
    v[:1500, :, :3] *= (0.97 ** (k % 150))[:, None, None].astype(np.float32)
    mn, mx = O.scene_aabb(v)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder(True).BuildTree(scene)
    col, _ = ab.BVHTreeCollapser().Collapse(tree, max_leaf=2)
    bvh = ab.CudaBVH(col, scene)
    cp = O.flatten(O.collapse(O.build_lbvh(v, mn, mx, bits=63)[0], max_leaf=2), v)
    assert bvh.view().max_depth > 20
    return scene, col, bvh, cp, mn, mx


# One ray; partly filled warps; either side of 1, 2, 4, 8 and 16 rays a warp on
# 148 SMs of 40 warps (5,920); several fetches a warp.
@pytest.mark.parametrize("n", [1, 31, 5919, 5921, 11841, 23681, 47361, 94721, 300001])
def test_trace_matches_oracle_at_any_ray_count(ctx, deep, n):
    import torch
    scene, col, bvh, cp, mn, mx = deep
    rays = ab.gen_rays_random(n, mn, mx, seed=n)
    rd = torch.from_numpy(rays).cuda()
    for any_hit in (False, True, False):
        res = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        bvh.trace(rd.data_ptr(), n, res.data_ptr(), any_hit=any_hit)
        ctx.synchronize()
        want = O.trace(cp, rays, any_hit=any_hit)
        assert np.array_equal(res.cpu().numpy()[:, :2], want[:, :2])


@pytest.mark.parametrize("w,h", [(1, 1), (37, 29), (640, 480)])
def test_camera_rays_match_oracle(ctx, deep, w, h):
    """Rays of one origin over a small layout, which are fetched later, and such
    rays among others."""
    import torch
    scene, col, bvh, cp, mn, mx = deep
    n = w * h
    assert bvh.view().num_nodes * 64 + bvh.view().num_woop * 16 <= 4_000_000
    rays = ab.gen_rays_pinhole(w, h).reshape(-1, 8)
    mixed = rays.copy()
    mixed[1::3] = ab.gen_rays_random(n, mn, mx, seed=n).reshape(-1, 8)[1::3]
    for r in (rays, mixed):
        rd = torch.from_numpy(r).cuda()
        for any_hit in (False, True):
            res = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            bvh.trace(rd.data_ptr(), n, res.data_ptr(), any_hit=any_hit)
            ctx.synchronize()
            assert np.array_equal(res.cpu().numpy()[:, :2], O.trace(cp, r, any_hit=any_hit)[:, :2])


def test_captured_trace_replays_beside_direct_ones(ctx, deep):
    """A captured trace keeps a ray counter of its own."""
    import torch
    scene, col, bvh, cp, mn, mx = deep
    n = 7001
    rays = ab.gen_rays_random(n, mn, mx, seed=9)
    rd = torch.from_numpy(rays).cuda()
    a, b = (torch.zeros((n, 4), dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    stream = torch.cuda.ExternalStream(ctx.stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        bvh.trace(rd.data_ptr(), n, a.data_ptr())
    want = O.trace(cp, rays)
    for _ in range(3):
        a.zero_()
        b.zero_()
        torch.cuda.synchronize()
        graph.replay()
        bvh.trace(rd.data_ptr(), n, b.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(a.cpu().numpy()[:, :2], want[:, :2])
        assert np.array_equal(b.cpu().numpy()[:, :2], want[:, :2])


def test_contexts_trace_side_by_side(deep):
    """Threads with a context each, as the server's lanes: launch shapes are the context's."""
    import threading

    import torch
    scene, col, bvh, cp, mn, mx = deep
    n, threads = 20011, 6
    rays = ab.gen_rays_random(n, mn, mx, seed=3)
    want = O.trace(cp, rays)
    rd = torch.from_numpy(rays).cuda()
    image = bvh.serialize()
    res = torch.zeros((threads, n, 4), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    start = threading.Barrier(threads)
    errors = []

    def work(k):
        try:
            start.wait()
            c = ab.Context(0)
            own = ab.CudaBVH.from_image(c, image)
            own.trace(rd.data_ptr(), n, res[k].data_ptr())
            c.synchronize()
            own.close()
            c.close()
        except BaseException as e:  # reported after the join
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    got = res.cpu().numpy()
    for k in range(threads):
        assert np.array_equal(got[k][:, :2], want[:, :2]), k


# ---- deep stacks ---------------------------------------------------------------
# A ray's stack grows while the nearer of two boxes it meets is the larger subtree's.

def _corner(levels: int, copies: int) -> np.ndarray:
    """Triangles across the first octant whose boxes start at the origin, each
    about half the one before along one axis: the 63-bit radix tree is a chain with
    the smaller boxes on the left.  Copies of the smallest lengthen it by their
    number's logarithm (equal codes)."""
    half = np.array([[0.75 * 2.0 ** -((k + 2 - a) // 3 + 1) for a in range(3)] for k in range(levels)])
    half = np.concatenate([half, np.repeat(half[-1:], copies, 0)])
    v = np.zeros((len(half), 3, 4), np.float32)
    for a in range(3):
        v[:, a, a] = 2 * half[:, a]
    return v


def _shrinking(n: int, f: float) -> np.ndarray:
    """As _corner, each a little smaller: ATRBVH makes long chains of them."""
    half = 0.5 * (1 + f) ** -np.arange(n, dtype=float)
    v = np.zeros((n, 3, 4), np.float32)
    for a in range(3):
        v[:, a, a] = 2 * half * (1 + 0.1 * a)
    return v


def _rays_out(v: np.ndarray, n: int, seed: int) -> np.ndarray:
    """Rays that leave from inside the boxes, at the scale of one of the triangles."""
    rng = np.random.default_rng(seed)
    size = v[rng.integers(0, len(v), n)][:, [0, 1, 2], [0, 1, 2]]
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = size * rng.uniform(0.02, 0.3, (n, 3))
    d = size * rng.uniform(0.05, 1.0, (n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1)[:, None]
    rays[:, 7] = 1e30
    return rays


def _stack_peak(cp, ray) -> int:
    """Entries a ray's stack holds at most, the one in the register included."""
    nodes = cp.nodes.reshape(-1, 16)
    box = nodes[:, :12].view(np.float32)
    o, inv = ray[:3].astype(float), 1.0 / ray[4:7].astype(float)
    stack, peak, at = [], 0, 0
    while True:
        if at >= 0:
            spans = []
            for k in (0, 1):
                n = box[at // 4].astype(float)
                a = (n[[4 * k, 4 * k + 2, 8 + 2 * k]] - o) * inv
                b = (n[[4 * k + 1, 4 * k + 3, 9 + 2 * k]] - o) * inv
                spans.append((max(ray[3], np.minimum(a, b).max()), min(ray[7], np.maximum(a, b).min())))
            order = (1, 0) if spans[1][0] < spans[0][0] else (0, 1)
            go = [int(nodes[at // 4, 12 + k]) for k in order if spans[k][1] >= spans[k][0]]
            stack += go[1:]
            peak = max(peak, len(stack))
            if go:
                at = go[0]
                continue
        if not stack:
            return peak
        at = stack.pop()


@pytest.mark.parametrize("levels,copies,depth,peak", [(16, 0, 15, 15), (17, 0, 16, 16), (18, 0, 17, 17), (50, 0, 49, 49),
                                                      (60, 4, 62, 62), (60, 8, 63, 63), (60, 512, 69, 69)])
def test_deep_stacks(ctx, levels, copies, depth, peak):
    """Stacks around the shared-memory entries, and layouts either side of the
    63 levels that the smaller stack takes."""
    import torch
    v = _corner(levels, copies)
    mn, mx = np.zeros(3, np.float32), np.ones(3, np.float32)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder(True).BuildTree(scene)
    col, _ = ab.BVHTreeCollapser().Collapse(tree, max_leaf=1)
    bvh = ab.CudaBVH(col, scene)
    cp = O.flatten(O.collapse(O.build_lbvh(v, mn, mx, bits=63)[0], max_leaf=1), v)
    assert bvh.view().max_depth == depth
    n = 5003
    rays = _rays_out(v, n, levels)
    assert max(_stack_peak(cp, r) for r in rays[:200]) == peak
    rd = torch.from_numpy(rays).cuda()
    for any_hit in (False, True):
        res = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        bvh.trace(rd.data_ptr(), n, res.data_ptr(), any_hit=any_hit)
        ctx.synchronize()
        assert np.array_equal(res.cpu().numpy()[:, :2], O.trace(cp, rays, any_hit=any_hit)[:, :2]), any_hit


def test_deep_stacks_over_several_meshes(ctx):
    import torch
    meshes = [_shrinking(400, 0.05), O.gen_scene(O.SCENE_UNIFORM, 300, 3)]
    off = np.concatenate([[0], np.cumsum([len(v) for v in meshes])]).astype(np.uint32)
    batch = ab.Batch(ctx, np.concatenate(meshes), off)
    batch.build(ab.Batch.ATRBVH, 9, 2)
    batch.collapse(max_leaf=1)
    batch.flatten()
    n = 3001
    rays, want = [], []
    for k, v in enumerate(meshes):
        mn, mx = O.scene_aabb(v)
        cp = O.flatten(O.collapse(O.atrbvh(O.build_lbvh(v, mn, mx)[0], 9, 2), max_leaf=1), v)
        rays.append(_rays_out(v, n, 5) if k == 0 else ab.gen_rays_random(n, mn, mx, seed=2).reshape(-1, 8))
        want.append(O.trace(cp, rays[-1]))
        if k == 0:
            assert max(_stack_peak(cp, r) for r in rays[0][:100]) > 64
    assert batch.compact_view(0).max_depth > 63
    rd = torch.from_numpy(np.concatenate(rays)).cuda()
    res = torch.full((2 * n, 4), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    batch.trace(rd.data_ptr(), 2 * n, [0, n, 2 * n], [0, 1], res.data_ptr())
    ctx.synchronize()
    assert np.array_equal(res.cpu().numpy()[:, :2], np.concatenate(want)[:, :2])


# ---- layouts far beyond L2 -----------------------------------------------------

@pytest.mark.parametrize("n,least,most", [(6_300_000, 600e6, 1100e6), (11_000_000, 1100e6, 2e9)])
def test_large_layouts(ctx, n, least, most):
    """The sizes from which warps step otherwise: on the device's own layout the
    oracle's traversal finds the same, alone and beside another mesh."""
    import torch
    v = ab.gen_scene(ab.SCENE_UNIFORM, n, 5)
    scene = ab.SceneWrapper(ctx, v)
    mn, mx = scene.bounds()
    tree = ab.LBVHBuilder().BuildTree(scene)
    col, _ = ab.BVHTreeCollapser().Collapse(tree)
    bvh = ab.CudaBVH(col, scene)
    col.close()
    tree.close()
    view = bvh.view()
    assert least < view.num_nodes * 64 + view.num_woop * 16 < most
    # More than twice the rays that 148 SMs hold at once (189,440).
    rays = ab.gen_rays_random(400_009, mn, mx, seed=8).reshape(-1, 8)
    cp = O.Compact(*bvh.download())
    rd = torch.from_numpy(rays).cuda()
    res = torch.full((len(rays), 4), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    want = {}
    for any_hit in (False, True):
        bvh.trace(rd.data_ptr(), len(rays), res.data_ptr(), any_hit=any_hit)
        ctx.synchronize()
        want[any_hit] = O.trace(cp, rays, any_hit=any_hit)[:, :2]
        assert np.array_equal(res.cpu().numpy()[:, :2], want[any_hit]), any_hit
    bvh.close()
    scene.close()
    small = O.gen_scene(O.SCENE_UNIFORM, 300, 3)
    batch = ab.Batch(ctx, np.concatenate([small, v]), np.array([0, 300, 300 + n], np.uint32))
    batch.build(ab.Batch.NONE)
    batch.collapse()
    batch.flatten()
    m = len(rays) - 1000
    batch.trace(rd.data_ptr(), len(rays), [0, m, len(rays)], [1, 0], res.data_ptr())
    ctx.synchronize()
    got = res.cpu().numpy()[:, :2]
    assert np.array_equal(got[:m], want[False][:m])
    few = O.flatten(O.collapse(O.build_lbvh(small, *O.scene_aabb(small))[0]), small)
    assert np.array_equal(got[m:], O.trace(few, rays[m:])[:, :2])
    batch.close()
