"""Traversal at the ray counts where a launch changes shape: rays per warp
follow the count (1, 2, 4, ... 32), warps fetch again, launches follow one
another on the context's ray counter, and layouts are deeper than the part of
the stack in shared memory."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def deep(ctx):
    """A layout of 30 and more levels: points that close in on a corner, among others."""
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
