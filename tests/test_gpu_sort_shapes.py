"""The sorts where their launches change shape: meshes of one tile (one launch),
tiles of 3, 6 and 12 keys a thread, prefix chunks folded or carried, and ray
keys with digits that all rays share."""
from __future__ import annotations

import numpy as np
import pytest

import atrbvh_b200 as ab
import oracle as O
from tests._util import scene_case

pytestmark = pytest.mark.gpu


def _check_keys(ctx, v, bits):
    mn, mx = O.scene_aabb(v)
    scene = ab.SceneWrapper(ctx, v, mn, mx)
    tree = ab.LBVHBuilder(bits == 63).BuildTree(scene)
    keys, order = tree.sorted_keys()
    want = O.morton(v, mn, mx, bits=bits).astype(np.uint64)
    idx = np.argsort(want, kind="stable")
    assert np.array_equal(order, idx.astype(np.uint32))
    assert np.array_equal(keys, want[idx])
    tree.close()
    scene.close()


# One tile (3,072), then tiles of 768, 1,536 and 3,072 keys; two chunks of 256
# tiles are walked by the prefixes.
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [2, 31, 3071, 3072, 3073, 196608, 196609, 393216, 393217, 786433])
def test_lbvh_order_at_tile_boundaries(ctx, n, bits):
    _check_keys(ctx, O.gen_scene(O.SCENE_CLUSTERED if n % 2 else O.SCENE_UNIFORM, n, n), bits)


# Where tiles grow to 1,536 and 3,072 keys, and three chunks: carried.
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [131072, 131073, 360448, 360449, 1572864, 1572865])
def test_lbvh_order_where_tiles_and_prefixes_change(ctx, n, bits):
    _check_keys(ctx, O.gen_scene(O.SCENE_CLUSTERED if n % 2 else O.SCENE_UNIFORM, n, n), bits)


@pytest.mark.parametrize("n", [3072, 5000])
def test_equal_keys_keep_their_order(ctx, n):
    v = np.repeat(O.gen_scene(O.SCENE_UNIFORM, 7, 3), -(-n // 7), axis=0)[:n]
    _check_keys(ctx, np.ascontiguousarray(v), 30)


def test_chunks_beyond_the_fold_are_carried(ctx):
    n = 4 * 256 * 3072 + 1
    _check_keys(ctx, O.gen_scene(O.SCENE_UNIFORM, n, 8), 30)


@pytest.mark.parametrize("sizes", [[2, 3072, 17], [2, 3073, 17]])
def test_batches_of_small_meshes(ctx, sizes):
    meshes = [O.gen_scene(O.SCENE_UNIFORM, n, n) for n in sizes]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    batch = ab.Batch(ctx, np.concatenate(meshes), off)
    batch.build(0)
    for m, v in enumerate(meshes):
        got, want = batch.mesh(m), O.build_lbvh(v, *O.scene_aabb(v))[0]
        for f in ("parent", "left", "right", "data", "area"):
            assert np.array_equal(getattr(got, f), getattr(want, f)), (m, f)


def _rays(kind, n):
    rays = O.gen_rays_random(n, (0, 0, 0), (1, 1, 1), seed=n)
    rays[:, 1, 3] = 2.0
    if kind == "one origin":
        rays[:, 0] = rays[0, 0]
    elif kind == "one direction":
        rays[:, 1] = rays[0, 1]
    elif kind == "identical":
        rays[:] = rays[0]
    elif kind == "pairs":
        rays[1::2] = rays[:len(rays[1::2])][::-1]
    elif kind == "far":  # an end point far away: every origin coordinate about equal
        rays[0, 1, 3] = 1e30
    return np.ascontiguousarray(rays)


@pytest.mark.parametrize("kind", ["random", "one origin", "one direction", "identical", "pairs", "far"])
@pytest.mark.parametrize("n", [1, 2, 769, 20001])
def test_ray_order_with_shared_digits(ctx, kind, n):
    import torch
    rays = _rays(kind, n)
    perm, _ = O.sort_rays(rays)
    rd = torch.from_numpy(rays).cuda()
    out = torch.zeros_like(rd)
    s2i, i2s = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ab.sort_rays(ctx, rd.data_ptr(), n, out.data_ptr(), None, s2i.data_ptr(), i2s.data_ptr())
    ctx.synchronize()
    assert np.array_equal(s2i.cpu().numpy(), np.asarray(perm))
    assert np.array_equal(out.cpu().numpy().view(np.int32), rays[perm].view(np.int32))
    assert np.array_equal(i2s.cpu().numpy()[np.asarray(perm)], np.arange(n))
