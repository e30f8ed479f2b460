"""GPU parity of the batched form: one persistent launch builds many meshes,
one launch traces rays of all of them.  Every mesh's bytes must equal a
separate rq_build of that mesh (itself bit-exact with the oracle), and every
hit must equal a separate rq_trace on that mesh."""
import numpy as np
import pytest
import torch

import pyoracle as O
import rq
from rq import workloads as W

pytestmark = pytest.mark.gpu


def make_batch(ctx, sizes, seed=5):
    pos, idx, descs = W.batched_meshes(sizes, seed=seed)
    p = torch.from_numpy(pos).cuda()
    i = torch.from_numpy(idx.view(np.int32)).cuda()
    b = rq.Batch(ctx, descs)
    b.build(p, i)
    ctx.sync_check()
    return pos, idx, descs, p, i, b


SIZES = [2, 4, 6, 64, 100, 998, 4096, 20000, 65536, 3, 130]


def test_batch_bytes_equal_separate_builds(ctx):
    pos, idx, descs, p, i, b = make_batch(ctx, SIZES)
    for m, (vo, nv, to, nt) in enumerate(descs):
        pm, im = pos[vo:vo + nv], idx[to:to + nt]
        s = rq.Bvh.build(ctx, torch.from_numpy(pm).cuda(), torch.from_numpy(im.view(np.int32)).cuda())
        got = b.download(m)
        want = s.download()
        for g, w, name in zip(got, want, ("nodes2", "tris", "nodes4", "perm")):
            assert g.tobytes() == w.tobytes(), f"mesh {m} ({nt} triangles): {name} differs"
        assert b.info(m)["depth4"] == s.info()["depth4"]
        s.destroy()
    # and one mesh against the oracle directly
    vo, nv, to, nt = descs[7]
    o = O.lbvh_build(pos[vo:vo + nv].reshape(-1), idx[to:to + nt].reshape(-1))
    n2, tr, n4, pm = b.download(7)
    assert n2.tobytes() == o["nodes2"].tobytes() and n4.tobytes() == o["nodes4"].tobytes()
    b.destroy()


def test_batch_rebuild_is_stable(ctx):
    pos, idx, descs, p, i, b = make_batch(ctx, SIZES)
    first = [b.download(m) for m in range(len(descs))]
    b.build(p, i)
    ctx.sync_check()
    for m in range(len(descs)):
        assert all(x.tobytes() == y.tobytes() for x, y in zip(first[m], b.download(m)))
    b.destroy()


@pytest.mark.parametrize("tri_flags", [0, rq.RQ_TRI_MT])
def test_batch_trace_equals_separate_traces(ctx, tri_flags):
    pos, idx, descs, p, i, b = make_batch(ctx, SIZES)
    rays, mesh, flags = W.batched_rays(descs, 500, 700, seed=11)
    rays_t = torch.from_numpy(rays).cuda()
    hits, stats = b.trace(rays_t, torch.from_numpy(mesh.view(np.int32)).cuda(),
                          torch.from_numpy(flags.view(np.int32)).cuda(), flags=tri_flags, stats=True)
    h = rq.hits_numpy(hits)
    st = rq.stats_numpy(stats)
    for m, (vo, nv, to, nt) in enumerate(descs):
        s = rq.Bvh.build(ctx, torch.from_numpy(pos[vo:vo + nv]).cuda(),
                         torch.from_numpy(idx[to:to + nt].view(np.int32)).cuda())
        sel = np.nonzero(mesh == m)[0]
        for f in (0, 1):
            part = sel[flags[sel] == f]
            hh, _, ss = rq.trace(ctx, s, torch.from_numpy(rays[part]).cuda(), flags=f | tri_flags, stats=True)
            assert rq.hits_numpy(hh).tobytes() == h[part].tobytes(), (m, f)
            assert rq.stats_numpy(ss).tobytes() == st[part].tobytes(), (m, f)
        s.destroy()
    assert 0.3 < h["hit"].mean() < 0.9
    b.destroy()


def test_batched_workload_sampled(ctx):
    # the batched configuration's 512 meshes (log-uniform 64..65,536), one build
    sizes = W.batched_sizes(512, seed=2)
    pos, idx, descs, p, i, b = make_batch(ctx, sizes, seed=2)
    rng = np.random.default_rng(1)
    for m in rng.choice(len(descs), 6, replace=False):
        vo, nv, to, nt = descs[m]
        o = O.lbvh_build(pos[vo:vo + nv].reshape(-1), idx[to:to + nt].reshape(-1))
        n2, tr, n4, pm = b.download(int(m))
        assert n2.tobytes() == o["nodes2"].tobytes() and n4.tobytes() == o["nodes4"].tobytes(), m
    # the same batch built with clusters for its large meshes: every mesh's
    # bytes unchanged, and the largest against the oracle
    want = [b.download(m) for m in range(len(descs))]
    for bt, cl, min_tris in ((1024, 2, 16384), (512, 4, 8192)):
        b.set_tuning({"build_threads": bt, "build_blocks": b.tuning()["max_build_blocks"], "build_cluster": cl,
                      "cluster_min_tris": min_tris})
        b.build(p, i)
        ctx.sync_check()
        for m in range(len(descs)):
            assert all(x.tobytes() == y.tobytes() for x, y in zip(want[m], b.download(m))), (bt, cl, m)
    m = int(np.argmax(sizes))
    vo, nv, to, nt = descs[m]
    o = O.lbvh_build(pos[vo:vo + nv].reshape(-1), idx[to:to + nt].reshape(-1))
    n2, tr, n4, pm = b.download(m)
    assert n2.tobytes() == o["nodes2"].tobytes() and n4.tobytes() == o["nodes4"].tobytes(), m
    b.destroy()


def test_batch_rejects_bad_descriptors(ctx):
    with pytest.raises(rq.RqError):
        rq.Batch(ctx, [(0, 3, 0, 2), (0, 3, 1, 2)])  # overlapping triangle ranges
    with pytest.raises(rq.RqError):
        rq.Batch(ctx, [(0, 3, 0, 0)])  # empty mesh


def test_every_launch_shape_gives_identical_results(ctx):
    pos, idx, descs, p, i, b = make_batch(ctx, SIZES)
    rays, mesh, flags = W.batched_rays(descs, 300, 300, seed=12)
    rays_t = torch.from_numpy(rays).cuda()
    mesh_t = torch.from_numpy(mesh.view(np.int32)).cuda()
    flags_t = torch.from_numpy(flags.view(np.int32)).cuda()
    want_tree = [b.download(m) for m in range(len(descs))]
    depths = [b.info(m)["depth4"] for m in range(len(descs))]
    want_hits = b.trace(rays_t, mesh_t, flags_t)[0].cpu().numpy()
    base = b.tuning()
    assert base["build_cluster"] == 1
    assert base["build_threads"] == 512 and base["trace_threads"] == 128 and base["max_build_blocks"] >= 1
    for bt, blocks in ((256, 1), (1024, 3), (512, base["max_build_blocks"])):
        b.set_tuning({"build_threads": bt, "build_blocks": blocks, "build_cluster": 1})
        b.build(p, i)
        ctx.sync_check()
        for m in range(len(descs)):
            assert all(x.tobytes() == y.tobytes() for x, y in zip(want_tree[m], b.download(m))), (bt, blocks, m)
    # thread-block clusters: every mesh (threshold 0, the 2-triangle ones
    # included), the large ones only, and grids that round down to whole
    # clusters or hold fewer blocks than one cluster
    for bt, blocks, cl, min_tris in ((1024, 8, 2, 0), (256, 8, 4, 0), (512, 5, 2, 1000), (1024, 11, 4, 20000),
                                     (512, base["max_build_blocks"], 4, 4096), (256, 1, 4, 0)):
        b.set_tuning({"build_threads": bt, "build_blocks": blocks, "build_cluster": cl, "cluster_min_tris": min_tris})
        b.build(p, i)
        ctx.sync_check()
        for m in range(len(descs)):
            got = b.download(m)
            assert all(x.tobytes() == y.tobytes() for x, y in zip(want_tree[m], got)), (bt, blocks, cl, min_tris, m)
        assert [b.info(m)["depth4"] for m in range(len(descs))] == depths
    for tt in (64, 128, 256):
        for chunk in (32, 64):
            for cap in (0, 64, 80):
                b.set_tuning({"trace_threads": tt, "trace_chunk": chunk, "trace_reg_cap": cap, "stack_entries": 128})
                got = b.trace(rays_t, mesh_t, flags_t)[0].cpu().numpy()
                ctx.sync_check()
                assert got.tobytes() == want_hits.tobytes(), (tt, chunk, cap)
    with pytest.raises(rq.RqError):
        b.set_tuning({"trace_threads": 96})
    with pytest.raises(rq.RqError):
        b.set_tuning({"build_cluster": 3})
    b.destroy()


def test_autotune_keeps_a_measured_shape(ctx):
    pos, idx, descs, p, i, b = make_batch(ctx, SIZES)
    rays, mesh, flags = W.batched_rays(descs, 200, 200, seed=13)
    rays_t = torch.from_numpy(rays).cuda()
    mesh_t = torch.from_numpy(mesh.view(np.int32)).cuda()
    flags_t = torch.from_numpy(flags.view(np.int32)).cuda()
    want = b.trace(rays_t, mesh_t, flags_t)[0].cpu().numpy()
    shape, trials = b.autotune(p, i, rays_t, mesh_t, flags_t, reps=2)
    builds = [t for t in trials if t["build_ms"] > 0]
    traces = [t for t in trials if t["trace_ms"] > 0]
    # 3 block sizes x 2 chunks x budgets {none, 64, 80}, plus 72 at 64 and 128 threads, then 4 refill
    # thresholds for the fastest of those
    assert len(traces) == 26 and len(builds) >= 3
    assert shape["build_ms"] == min(t["build_ms"] for t in builds)
    assert shape["trace_ms"] == min(t["trace_ms"] for t in traces)
    assert shape["stack_entries"] >= 3 * (max(b.info(m)["depth4"] for m in range(len(descs))) + 2) + 1
    got = b.trace(rays_t, mesh_t, flags_t)[0].cpu().numpy()
    assert got.tobytes() == want.tobytes()
    b.destroy()


def test_batch_mesh_sizes_and_places(ctx):
    """Meshes at the edges of the build's blocks and sort tiles, listed in any order, with gaps between their triangle
    ranges and vertices that are not in the meshes' order."""
    sizes = [1, 255, 256, 257, 513, 4095, 4096, 4097, 8193, 2, 70001]
    rng = np.random.default_rng(3)
    pos_l, idx_l, descs, v, t = [], [], [], 0, 5
    idx_l.append(np.zeros((5, 3), np.uint32))
    for n in sizes:
        p = (rng.uniform(-1, 1, (n, 1, 3)) + rng.uniform(-0.05, 0.05, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
        pos_l.append(p)
        idx_l.append(rng.permutation(3 * n).astype(np.uint32).reshape(-1, 3))
        idx_l.append(np.zeros((n % 7, 3), np.uint32))
        descs.append((v, 3 * n, t, n))
        v, t = v + 3 * n, t + n + n % 7
    pos, idx = np.concatenate(pos_l), np.concatenate(idx_l)
    order = rng.permutation(len(descs))
    p, i = torch.from_numpy(pos).cuda(), torch.from_numpy(idx.view(np.int32)).cuda()
    for leaf in (4, 1):
        b = rq.Batch(ctx, [descs[k] for k in order], max_leaf=leaf)
        b.build(p, i)
        b.build(p, i)
        ctx.sync_check()
        for m, k in enumerate(order):
            vo, nv, to, nt = descs[k]
            s = rq.Bvh.build(ctx, p[vo:vo + nv].contiguous(), i[to:to + nt].contiguous(), max_leaf=leaf)
            for g, w, name in zip(b.download(m), s.download(), ("nodes2", "tris", "nodes4", "perm")):
                assert g.tobytes() == w.tobytes(), (nt, name)
            s.destroy()
        b.destroy()


@pytest.mark.parametrize("max_leaf", [1, 16])
def test_batch_collapse_treelets(ctx, max_leaf):
    """Trees of 2,047, 2,049 and more binary nodes (a subtree of at most 2,048 is collapsed by one block), evenly spread
    and as a chain of ever smaller clusters."""
    rng = np.random.default_rng(8)
    pos_l, descs, v, t = [], [], 0, 0
    for n in (1, 2, 1023, 1024, 1025, 1026, 4097, 30000):
        for skew in (False, True):
            c = rng.uniform(0, 1, (n, 1, 3))
            if skew:
                c = c * 0.5 ** rng.integers(0, 10, (n, 1, 1))
            pos_l.append((c + rng.uniform(0, 1e-3, (n, 3, 3))).astype(np.float32).reshape(-1, 3))
            descs.append((v, 3 * n, t, n))
            v, t = v + 3 * n, t + n
    pos = np.concatenate(pos_l)
    idx = np.concatenate([np.arange(3 * d[3], dtype=np.int32).reshape(-1, 3) for d in descs])
    p, i = torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda()
    b = rq.Batch(ctx, descs, max_leaf=max_leaf)
    b.build(p, i)
    ctx.sync_check()
    for m, (vo, nv, to, nt) in enumerate(descs):
        o = O.lbvh_build(pos[vo:vo + nv].reshape(-1), None, max_leaf)
        g = b.download(m)
        for a, name in zip(g, ("nodes2", "tris", "nodes4")):
            assert a.tobytes() == o[name].tobytes(), (nt, name)
        assert np.array_equal(g[3], o["sorted"])
    b.destroy()


def test_batch_groups(ctx):
    """More triangles than one group of meshes holds (16,777,216): meshes of both groups equal a build of their own."""
    pos, idx = rq.scene_grid(1000, 500, seed=6)
    n, count = len(idx), 17
    p = torch.from_numpy(pos).cuda()
    i = torch.from_numpy(idx.view(np.int32)).cuda()
    b = rq.Batch(ctx, [(0, len(pos), k * n, n) for k in range(count)])
    b.build(p, i.repeat(count, 1))
    ctx.sync_check()
    s = rq.Bvh.build(ctx, p, i)
    want = s.download()
    for m in (0, 15, 16):
        for g, w in zip(b.download(m), want):
            assert g.tobytes() == w.tobytes(), m
    s.destroy()
    b.destroy()


def test_batch_rebuilt_to_deeper_trees(ctx):
    """The stack is sized by the first build's depths; meshes that contract and are rebuilt are traced as separate
    builds of them, by rays along which the nested boxes pile up on the stack."""
    from test_gpu_frame import contracting
    n, m = 2000, 1 << 18
    idx = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    rng = np.random.default_rng(0)
    c = np.concatenate([rng.uniform(-1, 1, (n, 2)), rng.uniform(-0.1, 0.1, (n, 1))], 1)
    flat = (c[:, None] + rng.uniform(-0.02, 0.02, (n, 3, 3))).astype(np.float32).reshape(-1, 3)
    deep = [contracting(n, 1.01), contracting(n, 1.008)]
    p = torch.from_numpy(np.tile(flat, (2, 1))).cuda()
    i = torch.from_numpy(np.tile(idx, (2, 1)).view(np.int32)).cuda()
    b = rq.Batch(ctx, [(0, 3 * n, 0, n), (3 * n, 3 * n, n, n)], max_leaf=1)
    b.build(p, i)
    assert max(b.info(k)["depth4"] for k in (0, 1)) == 7
    p.copy_(torch.from_numpy(np.concatenate(deep)))
    b.build(p, i)
    rays = np.zeros(m, rq.RAY)
    rays["org"] = (-1.6, -1.5, -1.55)
    rays["dir"] = rng.uniform(-1, 1, (m, 1)) + rng.uniform(-0.2, 0.2, (m, 3)) - rays["org"]
    rays["tmax"] = 100
    mesh = torch.arange(m, dtype=torch.int32, device="cuda") % 2
    rt = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    hits, _ = b.trace(rt, mesh)
    ctx.sync_check()
    for k in (0, 1):
        s = rq.Bvh.build(ctx, torch.from_numpy(deep[k]).cuda(), max_leaf=1)
        assert s.info()["depth4"] >= 18
        want, _, _ = rq.trace(ctx, s, rt[k::2].contiguous())
        assert torch.equal(hits[k::2], want)
        assert 0.02 < (want[:, 0] != 0).float().mean() < 1
        s.destroy()
    b.destroy()
