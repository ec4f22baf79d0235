"""Compact2 layouts at the sizes where the path sums change hands: meshes with
no, one or a few nodes of at least 128 inner nodes, alone and in a batch, with
and without collapsed leaves."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 127, 128, 129, 130, 257, 1031]


def _expected(v, max_leaf):
    mn, mx = O.scene_aabb(v)
    return O.flatten(O.collapse(O.atrbvh(O.build_lbvh(v, mn, mx)[0], 9, 2), max_leaf=max_leaf), v)


@pytest.mark.parametrize("max_leaf", [0, 1, 4])
def test_layouts_equal_the_oracle(ctx, max_leaf):
    meshes = [O.gen_scene(O.SCENE_UNIFORM, n, n) for n in SIZES]
    for v in meshes:  # large triangles overlap: uncapped leaves then hold many
        v[:, 1:, :3] += (v[:, 1:, :3] - v[:, :1, :3]) * (20.0 if max_leaf == 0 else 0.0)
    off = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.uint32)
    batch = ab.Batch(ctx, np.concatenate(meshes), off)
    batch.build(1, 9, 2)
    batch.collapse(max_leaf=max_leaf)
    batch.flatten()
    for m, v in enumerate(meshes):
        want = _expected(v, max_leaf)
        scene = ab.SceneWrapper(ctx, v, *O.scene_aabb(v))
        tree = ab.LBVHBuilder().BuildTree(scene)
        ab.AgglomerativeTreeletOptimizer(9, 2).Optimize(tree)
        col, _ = ab.BVHTreeCollapser().Collapse(tree, max_leaf=max_leaf)
        bvh = ab.CudaBVH(col, scene)
        assert bvh.view().max_depth <= batch.compact_view(m).max_depth
        for nodes, woop, tri in (bvh.download(), batch.compact(m)):
            assert np.array_equal(nodes, want.nodes)
            assert np.array_equal(woop.view(np.int32), want.woop.view(np.int32))
            assert np.array_equal(tri, want.tri_index)


class _Words:
    """A device array of int32 at an address, for torch."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (ptr, False), "version": 2}


@pytest.mark.parametrize("n", [100, 1031])
def test_the_root_is_part_of_the_layout_whatever_its_data_says(ctx, n):
    """A collapsed tree's arrays are the caller's to write through its view."""
    import torch
    v = O.gen_scene(O.SCENE_UNIFORM, n, n)
    scene = ab.SceneWrapper(ctx, v, *O.scene_aabb(v))
    tree = ab.LBVHBuilder().BuildTree(scene)
    col, _ = ab.BVHTreeCollapser().Collapse(tree, max_leaf=4)
    want = ab.CudaBVH(col, scene).serialize()
    data = torch.as_tensor(_Words(col.view().data, 2 * n - 1), device="cuda")
    assert int(data[0]) < 0
    data[0] = 5
    torch.cuda.synchronize()
    assert ab.CudaBVH(col, scene).serialize() == want
