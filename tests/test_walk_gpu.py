"""The device's BVH walks against the oracle's brute force on triangle soups
at the sizes where the tree's shape changes: one triangle (a root with an
empty box), two, a leaf's most and one more, and trees of several levels;
rays of every octant, along the axes (signed zeros in the direction) and in
random directions, from inside and outside the soup.  Answers are the
predicate's bits, so they are compared exactly."""
from __future__ import annotations

import numpy as np
import pytest

from hl2sdk_tools_sharp_b200 import tracer as T

pytestmark = pytest.mark.gpu


def soup(n: int, sky: int, seed: int):
    rng = np.random.default_rng([seed, n, sky])
    c = rng.uniform(-500.0, 500.0, (n, 1, 3))
    v = (c + rng.uniform(-120.0, 120.0, (n, 3, 3))).astype(np.float32).reshape(n, 9)
    ids = np.full(n, 0x02000000, np.int32)
    ids[:sky] = T.TRACE_ID_SKY
    return v, ids


def rays_for(seed: int, count: int = 4096):
    rng = np.random.default_rng([seed, 7])
    o = rng.uniform(-900.0, 900.0, (count, 3)).astype(np.float32)
    d = rng.normal(size=(count, 3)).astype(np.float32)
    axis = np.arange(count) % 8
    for a in range(3):
        only = axis == a
        s = np.where(rng.uniform(size=only.sum()) < 0.5, 1.0, -1.0).astype(np.float32)
        d[only] = np.where(rng.uniform(size=(only.sum(), 3)) < 0.5, np.float32(0.0), np.float32(-0.0))
        d[only, a] = s
    d *= rng.uniform(1.0, 1500.0, (count, 1)).astype(np.float32)
    return T.make_rays(o, d, 1.0)


@pytest.mark.parametrize("n,sky", [(1, 0), (1, 1), (2, 1), (8, 0), (9, 0), (33, 16), (1000, 100)])
def test_soup_equals_brute_force(n, sky, oracle_mod):
    O = oracle_mod
    verts, ids = soup(n, sky, 11)
    rays = rays_for(n)
    tris = O.prepare_triangles(verts, ids)
    flat = rays.view(np.float32).reshape(-1, 7)
    with T.CudaRayTracer(T.make_triangles(verts, ids)) as tr:
        for opts, flags in ((T.RayTraceOptions.stock_exact(), 0),
                            (T.RayTraceOptions(0.0, sky_does_not_block=True), O.SKY_PASS)):
            _, _, bits = O.brute_trace(tris, flat, flags=flags)
            assert np.array_equal(tr.visibility(rays, opts), O.bits_to_bool(bits, len(rays)))
        best, dist, _ = O.brute_trace(tris, flat, flags=O.CLOSEST)
        got = tr.closest(rays)
        assert np.array_equal(got["surface"], np.where(best >= 0, ids[np.maximum(best, 0)], -1))
        hit = best >= 0
        assert np.array_equal(got["fraction"][hit].view(np.uint32), dist[hit].astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("n,sky", [(20000, 1), (20001, 1), (20001, 20000), (30000, 3000)])
def test_soup_of_many_triangles_equals_brute_force(n, sky, oracle_mod):
    """About the size from which a scene keeps one copy of its nodes (one of
    the trees may still be a single triangle): the same answers from every
    entry that walks, and no more than a node's own 64 bytes for each."""
    O = oracle_mod
    verts, ids = soup(n, sky, 12)
    verts = verts.reshape(n, 3, 3)
    verts = (verts.mean(1, keepdims=True) + 0.1 * (verts - verts.mean(1, keepdims=True))).reshape(n, 9)
    rays = rays_for(n, 2048)
    tris = O.prepare_triangles(verts, ids)
    flat = rays.view(np.float32).reshape(-1, 7)
    with T.CudaRayTracer(T.make_triangles(verts, ids)) as tr:
        info = tr.scene_info()
        if n > 20000:
            assert info.device_bytes <= 52 * n + 64 * info.bvh_nodes
        _, _, bits = O.brute_trace(tris, flat)
        want = O.bits_to_bool(bits, len(rays))
        assert want.any() and not want.all()
        assert np.array_equal(tr.visibility(rays, T.RayTraceOptions.stock_exact()), want)
        assert np.array_equal(tr.visibility_recheck(rays, T.RayTraceOptions.stock_exact())[0], want)
        _, _, bits = O.brute_trace(tris, flat, flags=O.SKY_PASS)
        got = tr.visibility(rays, T.RayTraceOptions(0.0, sky_does_not_block=True))
        assert np.array_equal(got, O.bits_to_bool(bits, len(rays)))
        best, dist, _ = O.brute_trace(tris, flat, flags=O.CLOSEST)
        got = tr.closest(rays)
        hit = best >= 0
        assert np.array_equal(got["surface"], np.where(hit, ids[np.maximum(best, 0)], -1))
        assert np.array_equal(got["fraction"][hit].view(np.uint32), dist[hit].astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("octants", [1, 4, 5, 8])
@pytest.mark.parametrize("count", [1, 31, 33, 1000, 65536, 65537, 70001])
def test_warps_of_few_and_many_octants(octants, count, oracle_mod):
    """Each warp's rays lie in so many octants (the last warp's in as many as
    it has rays for): either walk gives the brute force's answers."""
    O = oracle_mod
    verts, ids = soup(500, 50, 21)
    rng = np.random.default_rng([octants, count])
    o = rng.uniform(-900.0, 900.0, (count, 3)).astype(np.float32)
    d = np.abs(rng.normal(size=(count, 3))).astype(np.float32) * np.float32(900.0)
    which = (np.arange(count) % octants + 3) % 8
    d *= np.where((which[:, None] >> np.arange(3)) & 1, np.float32(-1.0), np.float32(1.0))
    rays = T.make_rays(o, d, 1.0)
    tris = O.prepare_triangles(verts, ids)
    flat = rays.view(np.float32).reshape(-1, 7)
    with T.CudaRayTracer(T.make_triangles(verts, ids)) as tr:
        for opts, flags in ((T.RayTraceOptions.stock_exact(), 0),
                            (T.RayTraceOptions(0.0, sky_does_not_block=True), O.SKY_PASS)):
            _, _, bits = O.brute_trace(tris, flat, flags=flags)
            assert np.array_equal(tr.visibility(rays, opts), O.bits_to_bool(bits, len(rays)))
        best, dist, _ = O.brute_trace(tris, flat, flags=O.CLOSEST)
        got = tr.closest(rays)
        hit = best >= 0
        assert np.array_equal(got["surface"], np.where(hit, ids[np.maximum(best, 0)], -1))
        assert np.array_equal(got["fraction"][hit].view(np.uint32), dist[hit].astype(np.float32).view(np.uint32))


def skewed(n, base=0.01, factor=1.4):
    """Triangles in a row, each larger than the one before: a tree that takes
    the large ones off one after the other."""
    k = np.arange(n)
    size = base * factor ** k
    corner = np.stack([4.0 * size, 0.3 * size, -0.2 * size], 1)[:, None, :]
    shape = np.array([[0.0, 0.0, 0.0], [1.0, 0.2, 0.1], [0.1, 1.0, -0.3]])[None]
    return (corner + shape * size[:, None, None]).astype(np.float32).reshape(n, 9)


@pytest.mark.parametrize("n", [20, 66])
def test_skewed_scene_equals_brute_force(n, oracle_mod):
    """A tree deeper than a balanced one: the stacks hold its depth."""
    O = oracle_mod
    verts = skewed(n)
    ids = np.full(n, 0x02000000, np.int32)
    ids[::7] = T.TRACE_ID_SKY
    rng = np.random.default_rng(n)
    at = verts.reshape(n, 3, 3)[rng.integers(0, n, 4096)].mean(1)
    o = (at + rng.normal(size=at.shape) * np.linalg.norm(at, axis=1, keepdims=True)).astype(np.float32)
    rays = T.make_rays(o, ((at - o) * rng.uniform(0.5, 3.0, (4096, 1))).astype(np.float32), 1.0)
    tris = O.prepare_triangles(verts, ids)
    flat = rays.view(np.float32).reshape(-1, 7)
    with T.CudaRayTracer(T.make_triangles(verts, ids)) as tr:
        assert tr.scene_info().bvh_depth > np.ceil(np.log2(n))
        for opts, flags in ((T.RayTraceOptions.stock_exact(), 0),
                            (T.RayTraceOptions(0.0, sky_does_not_block=True), O.SKY_PASS)):
            _, _, bits = O.brute_trace(tris, flat, flags=flags)
            assert np.array_equal(tr.visibility(rays, opts), O.bits_to_bool(bits, len(rays)))
        best, dist, _ = O.brute_trace(tris, flat, flags=O.CLOSEST)
        got = tr.closest(rays)
        hit = best >= 0
        assert hit.any() and np.array_equal(got["surface"], np.where(hit, ids[np.maximum(best, 0)], -1))
        assert np.array_equal(got["fraction"][hit].view(np.uint32), dist[hit].astype(np.float32).view(np.uint32))


@pytest.mark.parametrize("casters", ["skewed", "one opaque", "sky alone"])
def test_walks_that_start_at_the_origins_leaf(casters):
    """The light gather's segments and the transfer rays start their walk near
    their origin and climb; with 20,000 triangles out of their reach added they
    start at the root of one copy of the nodes.  Same lumps: over a map with a
    skewed row of triangles in it, over one opaque triangle, over no opaque
    triangle at all."""
    import dataclasses
    from hl2sdk_tools_sharp_b200 import lighting as L, roomgrid as rg
    w = rg.generate(dataclasses.replace(rg.config_3x3(seed=2), side=2, lights=4, sky_ambient=True))
    off, lst = L.pvs_lists(w)
    verts, ids = np.asarray(w.tri_verts, np.float32).reshape(-1, 9), np.asarray(w.tri_ids)
    sky = (ids & T.TRACE_ID_SKY) != 0
    assert sky.any()
    row = skewed(24, 0.05).reshape(-1, 3, 3) + verts.reshape(-1, 3)[~np.repeat(sky, 3)].mean(0)
    row = row.astype(np.float32).reshape(-1, 9)
    if casters == "skewed":
        verts, ids = np.concatenate([verts, row]), np.concatenate([ids, np.full(len(row), ids[~sky][0], ids.dtype)])
    elif casters == "one opaque":
        verts, ids = np.concatenate([verts[sky], row[-1:]]), np.concatenate([ids[sky], ids[~sky][:1]])
    else:
        verts, ids = verts[sky], ids[sky]
    rng = np.random.default_rng(8)
    far = rng.uniform(-8000.0, 8000.0, (20000, 1, 3)) + rng.uniform(-50.0, 50.0, (20000, 3, 3))
    far[:, :, 2] -= 300000.0
    far = far.reshape(-1, 9).astype(np.float32)
    lumps = []
    with L.LightingStage(w) as st:
        st.upload_bounce(L.face_reflectivity(w), off, lst, threshold=1.0)
        for add in (0, len(far)):
            both = np.concatenate([verts, far[:add]])
            st.tracer.upload_scene(T.make_triangles(both, np.concatenate([ids, np.full(add, T.TRACE_ID_SKY, ids.dtype)])))
            lump, _, _ = st.light_pass()
            lumps.append(lump)
    assert lumps[0].any() and np.array_equal(lumps[0], lumps[1])
