"""TRBVH where its level passes find no memory: it runs in 20 bytes of scratch a
triangle, as it did before it had level passes, and gives the same trees."""
from __future__ import annotations

import concurrent.futures as cf
import multiprocessing

import numpy as np
import pytest

import atrbvh_b200 as ab

pytestmark = pytest.mark.gpu

# Every size about a treelet's, a few beyond a block of leaves, and one that makes
# the level passes' scratch (about 80 bytes a triangle) large beside a pool's blocks.
SIZES = [2, 3, 6, 7, 8, 13, 14, 15, 31, 255, 257, 3000, 65537, 6_000_000]
ITERATIONS = 3
LEAVE = 256 << 20  # bytes left free on the device: 20 a triangle fit, 80 do not


def _build(squeeze: bool):
    import torch
    ctx = ab.Context(0)
    off = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.uint32)
    verts = np.concatenate([ab.gen_scene(ab.SCENE_UNIFORM, n, 40 + k) for k, n in enumerate(SIZES)])
    batch = ab.Batch(ctx, verts, off)
    batch.set_params([7] * len(SIZES), [1 + k % ITERATIONS for k in range(len(SIZES))])
    batch.build(ab.Batch.NONE)  # the pool keeps what the radix trees need
    ctx.synchronize()
    hold = None
    if squeeze:
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - LEAVE, dtype=torch.uint8, device="cuda")
    before = ctx.launch_count()
    batch.build(ab.Batch.TRBVH, 7, ITERATIONS)
    ctx.synchronize()
    launches = ctx.launch_count() - before
    del hold
    torch.cuda.empty_cache()
    trees = [batch.mesh(m) for m in range(len(SIZES))]
    batch.close()
    ctx.close()
    return trees, launches


def _compare():
    want, by_levels = _build(False)
    got, tight = _build(True)
    fields = ("parent", "left", "right", "data", "bbox_min", "bbox_max", "area")
    differ = [(SIZES[m], f) for m, (a, b) in enumerate(zip(got, want)) for f in fields
              if not np.array_equal(getattr(a, f).view(np.uint32), getattr(b, f).view(np.uint32))]
    return by_levels, tight, differ


def test_trbvh_without_memory_for_level_passes():
    # In a process of its own: an allocation that fails takes back what the pools
    # of this process's other contexts keep, and then succeeds.
    with cf.ProcessPoolExecutor(1, mp_context=multiprocessing.get_context("spawn")) as pool:
        by_levels, tight, differ = pool.submit(_compare).result(timeout=300)
    assert tight < by_levels - 3 * ITERATIONS, "the level passes found memory"
    assert not differ, differ
