"""Serving loop: requests submitted together (continuous batching over two
lanes) give the same results as the same requests run one at a time, builds
equal the plain single-mesh pipeline, and admission by memory evicts idle
resident meshes."""
from __future__ import annotations

import time

import numpy as np
import pytest

import atrbvh_b200 as ab

pytestmark = pytest.mark.gpu


def _mesh(n: int, seed: int) -> np.ndarray:
    return ab.gen_scene(ab.SCENE_UNIFORM, n, seed)


def _rays(v: np.ndarray, count: int, seed: int) -> np.ndarray:
    p = v[:, :, :3].reshape(-1, 3)
    return ab.gen_rays_random(count, p.min(0), p.max(0), seed=seed)


def _jitter(v: np.ndarray, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    w = (v + rng.normal(0, 0.001, v.shape).astype(np.float32)).astype(np.float32)
    w[:, :, 3] = 0
    return w


def _workload(seed: int = 0):
    """Builds of log-uniform sizes and refits of some of them, with rays."""
    rng = np.random.default_rng(seed)
    reqs = []
    built = []
    for i in range(18):
        if built and rng.random() < 0.35:
            mid, base = built[int(rng.integers(len(built)))]
            w = _jitter(base, 1000 + i)
            reqs.append((ab.REQ_REFIT, mid, w, _rays(w, int(rng.integers(2000, 9000)), 50 + i)))
        else:
            n = int(np.exp(rng.uniform(np.log(1000), np.log(120000))))
            v = _mesh(n, 100 + i)
            reqs.append((ab.REQ_BUILD, i, v, _rays(v, int(rng.integers(2000, 9000)), 10 + i)))
            built.append((i, v))
    return reqs


def _run(server: ab.Server, reqs, together: bool, gap_s: float = 0.0):
    outs = [np.full((len(r[3]), 4), -7, np.int32) for r in reqs]
    results = [None] * len(reqs)
    if together:
        tickets = []
        for (kind, mid, v, rays), out in zip(reqs, outs):
            tickets.append(server.submit(kind, mid, v, rays, out))
            if gap_s:
                time.sleep(gap_s)
        for k, t in enumerate(tickets):
            results[k] = server.wait(t)
    else:
        for k, ((kind, mid, v, rays), out) in enumerate(zip(reqs, outs)):
            results[k] = server.wait(server.submit(kind, mid, v, rays, out))
    return outs, results


def test_server_mix_equals_alone():
    reqs = _workload(0)
    mix = ab.Server(lanes=2, max_batch_requests=8)
    outs_mix, res_mix = _run(mix, reqs, together=True, gap_s=0.002)
    st = mix.stats()
    mix.close()
    alone = ab.Server(lanes=1, max_batch_requests=1)
    outs_alone, res_alone = _run(alone, reqs, together=False)
    alone.close()
    assert all(r["status"] == 0 for r in res_mix), [r["error"] for r in res_mix if r["status"]]
    assert all(r["status"] == 0 for r in res_alone)
    assert max(r["batch_requests"] for r in res_mix) > 1, "no request shared a lane batch"
    assert st["completed"] == len(reqs) and st["failed"] == 0
    assert st["p99_ms"] >= st["p50_ms"] > 0
    for k in range(len(reqs)):
        assert np.array_equal(outs_mix[k], outs_alone[k]), f"request {k} kind {reqs[k][0]}"
        assert np.float32(res_mix[k]["sah"]) == np.float32(res_alone[k]["sah"]), k
        assert (outs_mix[k][:, 0] >= 0).any()


def test_server_build_equals_plain_pipeline(ctx):
    v = _mesh(30000, 7)
    rays = _rays(v, 20000, 3)
    srv = ab.Server(lanes=2)
    out = np.zeros((len(rays), 4), np.int32)
    r = srv.wait(srv.submit(ab.REQ_BUILD, 1, v, rays, out))
    srv.close()
    assert r["status"] == 0
    import torch
    scene = ab.SceneWrapper(ctx, v)
    tree = ab.LBVHBuilder().BuildTree(scene)
    ab.AgglomerativeTreeletOptimizer(9, 2).Optimize(tree)
    col, sah = ab.BVHTreeCollapser().Collapse(tree)
    bvh = ab.CudaBVH(col, scene)
    rd = torch.from_numpy(rays.reshape(-1)).cuda()
    res = torch.zeros(len(rays) * 4, dtype=torch.int32, device="cuda")
    bvh.trace(rd.data_ptr(), len(rays), res.data_ptr())
    ctx.synchronize()
    want = res.cpu().numpy().reshape(-1, 4)
    assert np.array_equal(out[:, :2], want[:, :2])
    assert np.float32(r["sah"]) == np.float32(sah)


def test_server_budget_evicts_idle_meshes():
    n = 50000
    # Room for about two resident meshes of this size beside one in flight.
    srv = ab.Server(lanes=1, hbm_budget=int(n * 404 * 2.5 + n * 460), max_batch_requests=1)
    meshes = [_mesh(n, 40 + i) for i in range(5)]
    for i, v in enumerate(meshes):
        assert srv.wait(srv.submit(ab.REQ_BUILD, i, v))["status"] == 0
    st = srv.stats()
    assert st["evictions"] >= 2 and st["resident_meshes"] <= 3
    # The oldest mesh was evicted; the newest is resident.
    w = _jitter(meshes[0], 1)
    assert srv.wait(srv.submit(ab.REQ_REFIT, 0, w))["status"] == ab.ERR_NOT_RESIDENT
    w = _jitter(meshes[4], 2)
    rays = _rays(w, 5000, 9)
    out = np.zeros((len(rays), 4), np.int32)
    assert srv.wait(srv.submit(ab.REQ_REFIT, 4, w, rays, out))["status"] == 0
    assert (out[:, 0] >= 0).any()
    srv.release(4)
    with pytest.raises(ab.AtrError):
        srv.release(4)
    srv.close()


def test_server_rejects_bad_requests():
    srv = ab.Server(lanes=1, max_batch_triangles=1000)
    v = _mesh(2000, 1)
    with pytest.raises(ab.AtrError):
        srv.submit(ab.REQ_BUILD, 0, v)  # above the batch cap
    with pytest.raises(ab.AtrError):
        srv.submit(5, 0, v[:10])
    r = srv.wait(srv.submit(ab.REQ_REFIT, 123, v[:10]))
    assert r["status"] == ab.ERR_NOT_RESIDENT
    srv.close()


def test_server_pinned_request_buffers_equal_pageable():
    """Requests whose vertex, ray and result buffers are page-locked (copied to
    and from the device directly, no staging copy), mixed in one lane batch
    with pageable ones, give the same results as pageable requests alone."""
    reqs = _workload(1)
    pinned = []
    for k, (kind, mid, v, rays) in enumerate(reqs):
        if k % 2 == 0:
            v, rays = ab.pinned_like(v), ab.pinned_like(rays)
        pinned.append((kind, mid, v, rays))
    mix = ab.Server(lanes=2, max_batch_requests=8)
    outs = [np.full((len(r[3]), 4), -7, np.int32) for r in pinned]
    outs = [ab.pinned_like(o) if k % 3 == 0 else o for k, o in enumerate(outs)]
    tickets = [mix.submit(kind, mid, v, rays, out) for (kind, mid, v, rays), out in zip(pinned, outs)]
    res_mix = [mix.wait(t) for t in tickets]
    st = mix.stats()
    mix.close()
    alone = ab.Server(lanes=1, max_batch_requests=1)
    outs_alone, res_alone = _run(alone, reqs, together=False)
    alone.close()
    assert all(r["status"] == 0 for r in res_mix), [r["error"] for r in res_mix if r["status"]]
    assert st["host_copy_ms"] >= 0 and st["lane_batch_ms"] > 0
    for k in range(len(reqs)):
        assert np.array_equal(outs[k], outs_alone[k]), f"request {k}"
        assert np.float32(res_mix[k]["sah"]) == np.float32(res_alone[k]["sah"]), k


def _buffers(reqs, kind):
    """The requests' arrays page-locked, pageable, or by turns."""
    if kind == "pageable":
        return reqs, [np.full((len(r[3]), 4), -7, np.int32) for r in reqs]
    pin = [kind == "pinned" or k % 2 == 0 for k in range(3 * len(reqs))]
    out = []
    for k, (what, mid, v, rays) in enumerate(reqs):
        v = ab.pinned_like(v) if pin[3 * k] else v
        out.append((what, mid, v, ab.pinned_like(rays) if pin[3 * k + 1] and len(rays) else rays))
    res = [np.full((len(r[3]), 4), -7, np.int32) for r in reqs]
    return out, [ab.pinned_like(o) if pin[3 * k + 2] and len(o) else o for k, o in enumerate(res)]


def _submit_all(srv, reqs, outs):
    stamps, tickets = [], []
    for (kind, mid, v, rays), out in zip(reqs, outs):
        stamps.append(time.perf_counter())
        tickets.append(srv.submit(kind, mid, v, rays if len(rays) else None, out if len(rays) else None))
    return stamps, [srv.wait(t) for t in tickets]


def _joining(n=1_200_000, refits=3):
    """A build that lasts (several ms, for the submissions behind it) and, at once,
    refits of its mesh: one without rays."""
    v = _mesh(n, 21)
    none = np.zeros((0, 8), np.float32)
    reqs = [(ab.REQ_BUILD, 5, v, _rays(v, 6000, 1))]
    for k in range(refits):
        w = _jitter(v, 300 + k)
        reqs.append((ab.REQ_REFIT, 5, w, none if k == 1 else _rays(w, 4000 + k, 2 + k)))
    return reqs


def _same(outs, res, want_outs, want_res):
    assert all(r["status"] == 0 for r in res), [r["error"] for r in res if r["status"]]
    for k in range(len(outs)):
        assert np.array_equal(outs[k], want_outs[k]), k
        assert np.float32(res[k]["sah"]) == np.float32(want_res[k]["sah"]), k


@pytest.mark.parametrize("kind", ["pageable", "pinned", "mixed"])
def test_server_refits_follow_the_build_they_wait_for(kind):
    """Refits that wait for a build are the second part of its batch; two of one
    mesh apply in order, one has no rays."""
    reqs, outs = _buffers(_joining(), kind)
    srv = ab.Server(lanes=1, max_batch_requests=8)
    _, res = _submit_all(srv, reqs, outs)
    alone = ab.Server(lanes=1, max_batch_requests=1)
    want_outs = [np.full((len(r[3]), 4), -7, np.int32) for r in reqs]
    want = [alone.wait(alone.submit(k, m, v, r if len(r) else None, o if len(r) else None))
            for (k, m, v, r), o in zip(reqs, want_outs)]
    assert [r["batch_requests"] for r in res] == [len(reqs)] * len(reqs)
    assert srv.stats()["lane_batches"] == 1
    srv.close()
    alone.close()
    _same(outs, res, want_outs, want)


def test_server_builds_do_not_wait_for_refits_that_join():
    reqs, outs = _buffers(_joining(refits=7), "pageable")
    srv = ab.Server(lanes=1, max_batch_requests=8)
    stamps, res = _submit_all(srv, reqs, outs)
    srv.close()
    assert res[0]["batch_requests"] == len(reqs)
    done = [s + r["latency_ms"] / 1e3 for s, r in zip(stamps, res)]
    # Seven refits stage 58 MB each, copy it and refit 1,200,000 triangles.
    assert min(done[1:]) - done[0] > 1e-3, [r["latency_ms"] for r in res]


def test_server_join_ends_at_the_batch_limit():
    reqs, outs = _buffers(_joining(), "pageable")
    srv = ab.Server(lanes=1, max_batch_requests=2)
    _, res = _submit_all(srv, reqs, outs)
    st = srv.stats()
    alone = ab.Server(lanes=1, max_batch_requests=1)
    want_outs, want = _buffers(reqs, "pageable")[1], None
    _, want = _submit_all(alone, reqs, want_outs)
    srv.close()
    alone.close()
    assert res[0]["batch_requests"] == res[1]["batch_requests"] == 2 and st["max_batch_requests_seen"] == 2
    _same(outs, res, want_outs, want)


def test_server_refits_wait_for_every_build_of_their_mesh():
    """Build, refit, build, refit of one id at once: both refits are of the second build."""
    a, b = _mesh(800000, 31), _mesh(800000, 32)
    r = _rays(a, 5000, 4)
    reqs = [(ab.REQ_BUILD, 9, a, r), (ab.REQ_REFIT, 9, _jitter(b, 1), r),
            (ab.REQ_BUILD, 9, b, r), (ab.REQ_REFIT, 9, _jitter(b, 2), r)]
    outs = _buffers(reqs, "pageable")[1]
    srv = ab.Server(lanes=1, max_batch_requests=8)
    _, res = _submit_all(srv, reqs, outs)
    srv.close()
    order = [0, 2, 1, 3]
    alone = ab.Server(lanes=1, max_batch_requests=1)
    want_outs, want = [None] * 4, [None] * 4
    for k in order:
        want_outs[k] = np.full((len(r), 4), -7, np.int32)
        want[k] = alone.wait(alone.submit(*reqs[k], want_outs[k]))
    alone.close()
    _same(outs, res, want_outs, want)
