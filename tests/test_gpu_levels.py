"""Who takes which treelet roots: level passes, the cluster at the top, and the
dataflow pass where a top does not fit the cluster."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("parent", "left", "right", "data", "area")


def _chain(seed: int) -> np.ndarray:
    """About 300 triangles whose radix tree is a chain of 30 levels: ten small
    triangles in every cell along the corner that the codes close in on."""
    rng = np.random.default_rng(seed)
    cells = []
    for k in range(10):
        for axis in range(3):
            lo = np.full(3, 0.0)
            size = np.full(3, 2.0 ** -(k + 1))
            size[:axis] = 2.0 ** -(k + 1)
            size[axis + 1:] = 2.0 ** -k
            lo[axis] = 2.0 ** -(k + 1)
            cells.append((lo, size))
    v = np.zeros((len(cells) * 10, 3, 4), np.float32)
    for c, (lo, size) in enumerate(cells):
        for j in range(10):
            p = lo + size * rng.uniform(0.1, 0.9, 3)
            v[c * 10 + j, :, :3] = p + size * rng.uniform(-0.02, 0.02, (3, 3))
    v[0, 0, :3] = 0.0
    v[1, 0, :3] = 1.0
    return v


def _same(got, want, label):
    for f in FIELDS:
        assert np.array_equal(getattr(got, f), getattr(want, f)), (label, f)
    assert np.array_equal(got.bbox_min[:, :3], want.bbox_min[:, :3])
    assert np.array_equal(got.bbox_max[:, :3], want.bbox_max[:, :3])


# 200 chains have more roots above the level passes than the cluster kernel
# holds (2,048): the dataflow pass takes them.  Three fit.
@pytest.mark.parametrize("count", [3, 200])
@pytest.mark.parametrize("optimizer", [ab.Batch.ATRBVH, ab.Batch.TRBVH])
def test_deep_tops(ctx, optimizer, count):
    meshes = [_chain(k) for k in range(count)]
    off = np.concatenate([[0], np.cumsum([len(v) for v in meshes])]).astype(np.uint32)
    batch = ab.Batch(ctx, np.concatenate(meshes), off)
    tsize, iters = (9, 2) if optimizer == ab.Batch.ATRBVH else (7, 3)
    batch.build(optimizer, tsize, iters)
    ctx.synchronize()  # reports device-side errors
    run = O.atrbvh if optimizer == ab.Batch.ATRBVH else O.trbvh
    for m in sorted({0, 1, count // 2, count - 1}):
        base = O.build_lbvh(meshes[m], *O.scene_aabb(meshes[m]))[0]
        _same(batch.mesh(m), run(base, tsize, iters), m)


# Around the sizes where roots appear, where a level outgrows the cluster's
# width, and where the cluster gives way to the dataflow pass (131,072).
@pytest.mark.parametrize("n", [6, 7, 9, 10, 20, 2701, 131072, 131073])
def test_sizes(ctx, n):
    v = O.gen_scene(O.SCENE_CLUSTERED if n > 100 else O.SCENE_UNIFORM, n, n)
    mn, mx = O.scene_aabb(v)
    base = O.build_lbvh(v, mn, mx, threads=0)[0]
    for optimizer, run in ((ab.AgglomerativeTreeletOptimizer(9, 2), lambda: O.atrbvh(base, 9, 2, threads=0)),
                           (ab.TRBVHOptimizer(7, 3), lambda: O.trbvh(base, 7, 3, threads=0))):
        scene = ab.SceneWrapper(ctx, v, mn, mx)
        tree = ab.LBVHBuilder().BuildTree(scene)
        optimizer.Optimize(tree)
        ctx.synchronize()
        _same(ab.BVHTreeInstanceManager().DeviceToHostTree(tree), run(), n)
        tree.close()
        scene.close()


@pytest.mark.parametrize("n", [2, 13, 127, 128, 129])
def test_small_trees_by_one_climb(ctx, n):
    """TRBVH of up to 128 triangles takes one climb an iteration."""
    v = O.gen_scene(O.SCENE_UNIFORM, n, n)
    mn, mx = O.scene_aabb(v)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder().BuildTree(scene)
    before = ctx.launch_count()
    ab.TRBVHOptimizer(7, 3).Optimize(tree)
    assert (ctx.launch_count() - before <= 6) == (n <= 128)
    ctx.synchronize()
    _same(ab.BVHTreeInstanceManager().DeviceToHostTree(tree), O.trbvh(O.build_lbvh(v, mn, mx)[0], 7, 3), n)


def test_nan_areas_do_not_hang_trbvh(ctx):
    """A triangle with an infinite vertex and a flat axis has a NaN area."""
    v = O.gen_scene(O.SCENE_UNIFORM, 300, 5)
    v[17, 0, 0] = np.inf
    v[17, :, 1] = 0.25
    mn, mx = np.zeros(3, np.float32), np.ones(3, np.float32)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder().BuildTree(scene)
    ab.TRBVHOptimizer(7, 2).Optimize(tree)
    ctx.synchronize()
    got = ab.BVHTreeInstanceManager().DeviceToHostTree(tree)
    want = O.trbvh(O.build_lbvh(v, mn, mx)[0], 7, 2)
    for f in ("parent", "left", "right", "data"):
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
