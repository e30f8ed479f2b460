"""GPU parity of the median-split build (rq_build with RQ_BUILD_MEDIAN)
against the reference's own SoftwareBVH::build (common/software_bvh.hpp,
compiled from its sources into oracle/_ref) on inputs whose centroid values
never repeat on an axis (then nth_element's left and right sets are unique):
binary nodes byte for byte, each leaf's triangles as a set, and the 4-wide
collapse byte for byte against the reference's fromBVH2.  Committed fixtures
(tests/golden/ref_median_soups.npz, the reference's output) stand in where
the reference library is not built."""
import os

import numpy as np
import pytest
import torch

import pyoracle as O
import rq
from conftest import soup

pytestmark = pytest.mark.gpu

GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_median_soups.npz")


def tie_free_soup(n, seed):
    """A random soup with the triangles whose float32 centroid ((p0+p1)+p2)/3
    repeats a value on some axis removed."""
    v = soup(n, seed).reshape(-1, 3, 3)
    c = ((v[:, 0] + v[:, 1]) + v[:, 2]) / np.float32(3.0)
    keep = np.ones(len(v), bool)
    for a in range(3):
        _, inv, cnt = np.unique(c[:, a], return_inverse=True, return_counts=True)
        keep &= cnt[inv] == 1
    return np.ascontiguousarray(v[keep].reshape(-1, 3))


def gpu_median(ctx, pos, max_leaf):
    p = torch.from_numpy(pos).cuda()
    b = rq.Bvh.build(ctx, p, None, max_leaf=max_leaf, median=True)
    ctx.sync_check()
    out = b.download()
    b.destroy()
    return out  # nodes2, tris, nodes4, perm


def check(n2g, trg, n4g, n2r, trr, n4r):
    assert len(n2g) == len(n2r)
    assert n2g.tobytes() == n2r.tobytes(), "binary nodes"
    for nd in n2r[n2r["left_child"] < 0]:
        f, c = ~int(nd["left_child"]), int(nd["right_child"])
        a = np.sort(trg[f:f + c].view(np.uint8).reshape(c, -1), axis=0)
        b = np.sort(trr[f:f + c].view(np.uint8).reshape(c, -1), axis=0)
        assert np.array_equal(a, b), "leaf triangle sets"
    assert n4g.tobytes() == n4r.tobytes(), "4-wide nodes"


@pytest.mark.skipif(not O.have_ref(), reason="needs oracle/_ref")
@pytest.mark.parametrize("n,seed,max_leaf", [(1, 1, 4), (2, 2, 4), (5, 3, 4), (17, 4, 1), (100, 5, 4),
                                             (1000, 6, 8), (4097, 7, 4), (100000, 8, 4)])
def test_median_matches_reference_live(ctx, n, seed, max_leaf):
    pos = tie_free_soup(n, seed)
    idx = np.arange(len(pos), dtype=np.uint32)
    n2r, trr, n4r = O.ref_build(pos, idx, max_leaf)
    n2g, trg, n4g, perm = gpu_median(ctx, pos, max_leaf)
    check(n2g, trg, n4g, n2r, trr, n4r)
    # the permutation names the triangles written in leaf order
    v = pos.reshape(-1, 3, 3)
    assert np.array_equal(trg["v0"][:, :3], v[perm, 0]) and np.array_equal(trg["v2"][:, :3], v[perm, 2])


def test_median_matches_reference_fixtures(ctx):
    g = np.load(GOLD)
    for key in sorted(k for k in g.files if k.startswith("pos_")):
        tag = key[4:]
        max_leaf = int(g[f"leaf_{tag}"])
        n2g, trg, n4g, _ = gpu_median(ctx, g[key], max_leaf)
        check(n2g, trg, n4g, g[f"nodes2_{tag}"].view(rq.BVH2_NODE), g[f"tris_{tag}"].view(rq.TRIANGLE),
              g[f"nodes4_{tag}"].view(rq.BVH4_NODE))


def test_median_traces_like_lbvh(ctx):
    # another tree over the same triangles: identical closest hits (hit
    # flags, primitive ids, t) except exact-t ties
    pos, idx = rq.scene_grid(64, 32, seed=0)
    p = torch.from_numpy(pos).cuda()
    i = torch.from_numpy(idx.view(np.int32)).cuda()
    bm = rq.Bvh.build(ctx, p, i, median=True)
    bl = rq.Bvh.build(ctx, p, i)
    rays = torch.from_numpy(rq.scene_rays_down(65536, seed=2)).cuda()
    hm = rq.hits_numpy(rq.trace(ctx, bm, rays)[0])
    hl = rq.hits_numpy(rq.trace(ctx, bl, rays)[0])
    assert np.array_equal(hm["hit"], hl["hit"]) and hm["t"].tobytes() == hl["t"].tobytes()
    assert (hm["primitive_id"] != hl["primitive_id"]).mean() < 1e-4
    bm.destroy()
    bl.destroy()


def test_median_build_replayed_from_a_graph(ctx):
    # the median build is stream-ordered (it launches every level a split can
    # reach and reads each level's size on the device), so a rebuild can be
    # captured in a CUDA graph beside an LBVH rebuild and replayed after the
    # vertices move; each replay equals a build outside the graph
    pos_a = tie_free_soup(30000, 61)
    n = len(pos_a) // 3
    pos_b = tie_free_soup(40000, 62)[: 3 * n]
    p = torch.from_numpy(pos_a).cuda()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        bm = rq.Bvh.build(ctx, p, None, median=True, stream=side)  # arrays and scratch before the capture
        bl = rq.Bvh.build(ctx, p, None, stream=side)
        side.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            rq.Bvh.build(ctx, p, None, median=True, into=bm, stream=side)
            rq.Bvh.build(ctx, p, None, into=bl, stream=side)
    for pos in (pos_b, pos_a):
        p.copy_(torch.from_numpy(pos))
        g.replay()
        torch.cuda.synchronize()
        ctx.sync_check()
        got_m, got_l = bm.download(), bl.download()
        want_m = gpu_median(ctx, pos, 4)
        o = O.lbvh_build(pos.reshape(-1), None)
        for a, b in zip(got_m, want_m):
            assert a.tobytes() == b.tobytes()
        assert got_l[0].tobytes() == o["nodes2"].tobytes() and got_l[2].tobytes() == o["nodes4"].tobytes()
    del g
    bm.destroy()
    bl.destroy()


def median_statement(pos, max_leaf):
    """The median build's rules over a soup, one range at a time: binary nodes in pre-order and the permutation."""
    v = pos.reshape(-1, 3, 3).astype(np.float32)
    cent = ((v[:, 0] + v[:, 1]) + v[:, 2]) / np.float32(3.0)
    nodes, perm = [], np.empty(len(v), np.uint32)
    work = [(0, [np.argsort(cent[:, a], kind="stable") for a in range(3)], -1)]
    while work:
        s, orders, right_of = work.pop()
        c, me = len(orders[0]), len(nodes)
        if right_of >= 0:
            nodes[right_of][3] = me
        ids = orders[0]
        nodes.append([v[ids].min((0, 1)), v[ids].max((0, 1)), ~s, c])
        ext = np.array([cent[o[-1], a] - cent[o[0], a] for a, o in enumerate(orders)], np.float32)
        if c <= max_leaf or ext.max() < np.float32(1e-6):
            perm[s:s + c] = ids
            continue
        nodes[me][2] = me + 1
        left = np.zeros(len(v), bool)
        left[orders[int(ext.argmax())][:c // 2]] = True
        work.append((s + c // 2, [o[~left[o]] for o in orders], me))
        work.append((s, [o[left[o]] for o in orders], -1))
    out = np.zeros(len(nodes), rq.BVH2_NODE)
    for k, (lo, hi, lc, rc) in enumerate(nodes):
        out[k] = (lo, lc, hi, rc)
    return out, perm


def tie_soup(n, same):
    """A soup with repeated centroid values on every axis, `same` of its triangles identical."""
    rng = np.random.default_rng(n)
    c = np.round(rng.uniform(-4, 4, (n, 1, 3)) * 16) / 16
    p = (c + np.array([[0, 0, 0], [0.25, 0, 0], [0, 0.25, 0.125]])).astype(np.float32)
    p[rng.permutation(n)[:same]] = p[0]
    return p.reshape(-1, 3)


@pytest.mark.parametrize("n,same,max_leaf", [(1, 0, 4), (5, 0, 4), (17, 5, 1), (1023, 0, 4), (1024, 0, 1), (1025, 0, 1),
                                             (1025, 1025, 4), (2047, 0, 16), (2049, 600, 4), (4099, 0, 2),
                                             (9000, 7000, 4), (9001, 9001, 4), (20000, 0, 4)])
def test_median_matches_its_statement(ctx, n, same, max_leaf):
    """Ranges at the edges of a block's and a tile's size, ties on every axis, leaves by extent above and below them."""
    pos = tie_soup(n, same)
    n2g, trg, _, perm = gpu_median(ctx, pos, max_leaf)
    n2, want = median_statement(pos, max_leaf)
    assert np.array_equal(perm, want)
    assert n2g.tobytes() == n2.tobytes()
    assert np.array_equal(trg["v1"][:, :3], pos.reshape(-1, 3, 3)[want, 1])


@pytest.mark.parametrize("call", ["trace", "shadow_ao", "reflect", "ao_depth", "gbuffer"])
def test_rebuild_to_leaves_too_large_is_reported(ctx, call):
    """The host's largest leaf is from the first build; an in-place rebuild that ends in a leaf of 17 is found on the
    device, by every kernel that cannot hold one."""
    from rq import workloads as W
    first = np.ascontiguousarray(tie_free_soup(40, 9)[:51])
    pos = torch.from_numpy(first).cuda()
    b = rq.Bvh.build(ctx, pos, median=True)
    assert b.info()["max_leaf"] <= 4
    cam, params = W.shadow_camera(), W.shadow_params()
    cam.width, cam.height = params.width, params.height = 32, 16
    gbuf = torch.zeros((32 * 16, 8), dtype=torch.int32, device="cuda")

    def run():
        if call == "trace":
            rq.trace(ctx, b, torch.tensor([[0, 0, -9, 0, 0, 0, 1, 99]], dtype=torch.float32, device="cuda"))
        elif call == "shadow_ao":
            rq.render_shadow_ao(ctx, b, gbuf, params)
        elif call == "reflect":
            rq.render_reflect(ctx, b, gbuf, rq.ReflectParams(width=32, height=16))
        elif call == "ao_depth":
            p = rq.AoDepthParams(width=32, height=16, spp=1)
            rq.render_ao_depth(ctx, b, torch.ones(32 * 16, device="cuda"), p)
        else:
            ctx.set_camera_tuning(1)
            rq.render_gbuffer(ctx, b, cam, gbuf)
        ctx.sync_check()

    try:
        run()
        pos.copy_(torch.from_numpy(np.tile(first[:3], (17, 1))))
        rq.Bvh.build(ctx, pos, median=True, into=b)
        with pytest.raises(rq.RqError) as e:
            run()
        assert e.value.status == rq.RQ_ERR_UNSUPPORTED
    finally:
        ctx.set_camera_tuning(0)
    b.destroy()
