"""The LBVH build where its blocks widen (512 leaves past 2,097,152 triangles):
last blocks of 1 and 513 leaves, equal keys, and meshes that share blocks."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O
from tests._util import assert_trees_equal

pytestmark = pytest.mark.gpu

WIDE = 1 << 21


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [WIDE, WIDE + 1, WIDE + 513])
def test_single_mesh(ctx, n, bits):
    v = O.gen_scene(O.SCENE_UNIFORM, n, 5)
    v[n // 2:n // 2 + 3000] = v[0]  # equal keys across block edges
    mn, mx = O.scene_aabb(v)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder(bits == 63).BuildTree(scene)
    want, _, _ = O.build_lbvh(v, mn, mx, bits=bits, threads=8)
    assert_trees_equal(ab.BVHTreeInstanceManager().DeviceToHostTree(tree), want, f"{n} triangles")
    tree.close()
    scene.close()


@pytest.mark.parametrize("optimizer", [0, 1])
def test_meshes_sharing_blocks(ctx, optimizer):
    sizes = [2, 3, 509, 512, 513, 1025, WIDE - 7, 2, 511, 40000]
    meshes = [O.gen_scene(O.SCENE_UNIFORM, n, n) for n in sizes]
    batch = ab.Batch(ctx, np.concatenate(meshes), np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32))
    batch.build(optimizer, 9, 1)
    for m, v in enumerate(meshes):
        want, _, _ = O.build_lbvh(v, *O.scene_aabb(v), threads=8)
        if optimizer:
            want = O.atrbvh(want, 9, 1, threads=8)
        assert_trees_equal(batch.mesh(m), want, f"mesh {m} ({sizes[m]} triangles)")
