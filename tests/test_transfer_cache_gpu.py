"""The transfer cache on the GPU: ReadPacked decoded on the device
(vrad_transfer_read_packed) against the oracle on the reference's
TransferSetCodecTests cases, and the store and the hit of
TransferCacheBounceTests (src/SourceSharp.Tests/MapTools/Rad/Bounce/
TransferCacheBounceTests.cs:70-117) on the 3x3 room grid: a light pass's
transfers exported (the index and planes the oracle writes for the same
lists), installed on a stage whose lights changed, and that stage's pass
lighting the same lump as one that built its own transfers."""
import dataclasses

import numpy as np
import pytest

from hl2sdk_tools_sharp_b200 import lighting as L, roomgrid as rg, tracer as T, transfer_cache as C
from oracle import transfer_codec_oracle as O
from test_transfer_codec_cpu import packed_refusals, sample, same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tracer():
    tri = T.make_triangles(np.array([[[0, 0, 0], [1, 0, 0], [0, 1, 0]]], np.float32), np.array([1], np.int32))
    t = T.CudaRayTracer(tri)
    yield t
    t.close()


def lists_from(got):
    return None if got is None else [got[1][got[0][p]:got[0][p + 1]] for p in range(len(got[0]) - 1)]


@pytest.mark.parametrize("chunk_bytes", [24, 8, 1 << 20])
def test_device_read_packed_equals_the_oracle(tracer, chunk_bytes):
    s = sample()
    packed = [O.pack(c) for c in O.chunks(s, chunk_bytes)]
    got = lists_from(C.read_packed(tracer, O.index(s), packed, 4))
    assert same(got, O.read_packed(O.index(s), packed, 4))
    # The library's own packing reads the same.
    mine = [C.pack(c) for c in O.chunks(s, chunk_bytes)]
    assert same(lists_from(C.read_packed(tracer, O.index(s), mine, 4)), s)


def test_device_read_packed_refuses_what_the_reference_refuses(tracer):
    packed_refusals(lambda idx, packed, n: lists_from(C.read_packed(tracer, idx, packed, n)))


def test_device_read_packed_on_a_large_random_set(tracer):
    # 300,000 transfers over 5,000 patches in 37 chunks (one list straddles
    # many chunk edges); wrapping deltas both ways.
    rng = np.random.default_rng(11)
    counts = rng.integers(0, 120, 5000)
    counts[17] = 4000
    lists = []
    for c in counts:
        tr = np.zeros(c, O.TRANSFER_DTYPE)
        tr["patch"] = rng.integers(0, 5000, c)
        tr["weight"] = rng.random(c, np.float32)
        lists.append(tr)
    total = int(counts.sum())
    b = 8 * (total // 37 + 1)
    packed = [C.pack(c) for c in O.chunks(lists, b)]
    got = lists_from(C.read_packed(tracer, O.index(lists), packed, 5000))
    assert same(got, lists)


def _stage(w, inp, max_chop=4.0):
    st = L.LightingStage(w, inp)
    off, lst = L.pvs_lists(w)
    st.upload_bounce(L.face_reflectivity(w), off, lst, max_chop=max_chop, threshold=0.1)
    return st


def _edited(inp):
    """The same map with its lights changed (RadWorld.TransferKey reads no
    light, so a light edit keeps the key)."""
    lights = inp.lights.copy()
    lights["intensity"] *= np.float32(0.5)
    lights["intensity"][0] *= np.float32(3.0)
    return dataclasses.replace(inp, lights=lights)


def test_a_replay_bounces_the_same_light_as_a_fresh_build():
    w = rg.generate(rg.config_3x3(seed=2))
    inp = L.prepare(w)
    with _stage(w, inp) as first:
        with pytest.raises(ValueError):
            C.export(first)                      # no pass has bounced yet
        first.light_pass()
        off, tr = first.transfers()
        idx, packed = C.export(first, 1 << 12)
    lists = [tr[off[p]:off[p + 1]] for p in range(len(off) - 1)]
    # The store's bytes: the oracle's index and, inside every packed chunk,
    # the oracle's planes of the oracle's chunk.
    assert idx == O.index(lists)
    assert len(packed) > 3
    assert [O.unpack(p) for p in packed] == O.chunks(lists, 1 << 12)

    edited = _edited(inp)
    with _stage(w, edited) as fresh:
        want_lump, want_ofs, _ = fresh.light_pass()
        want_total, _ = fresh.patch_light()
        want_stats = fresh.bounce_stats()
    with _stage(w, edited) as replay:
        assert C.install(replay, idx, packed)
        lump, ofs, _ = replay.light_pass()
        stats = replay.bounce_stats()
        total, _ = replay.patch_light()
        r_off, r_tr = replay.transfers()
        # A second pass replays them again.
        lump2, _, _ = replay.light_pass()
        again_idx, again = C.export(replay, 1 << 20)
    assert stats.transfers_cached == 1 and want_stats.transfers_cached == 0
    assert stats.transfer_rays == 0 and stats.transfers == want_stats.transfers == len(tr)
    assert stats.bounces == want_stats.bounces
    assert np.array_equal(r_off, off) and np.array_equal(r_tr.view(np.uint64), tr.view(np.uint64))
    assert np.array_equal(total.view(np.uint32), want_total.view(np.uint32))
    assert np.array_equal(ofs, want_ofs)
    assert np.array_equal(lump, want_lump) and np.array_equal(lump2, want_lump)
    assert again_idx == idx and O.read_packed(again_idx, again, len(off) - 1) is not None
    assert b"".join(O.unpack(p) for p in again) == b"".join(O.chunks(lists, 1 << 12))


def test_a_set_of_another_patch_tree_is_refused_and_changes_nothing():
    w = rg.generate(rg.config_3x3(seed=2))
    inp = L.prepare(w)
    with _stage(w, inp, max_chop=16.0) as coarse:
        coarse.light_pass()
        idx, packed = C.export(coarse)
    with _stage(w, inp) as st:
        want, _, _ = st.light_pass()
        n = st.bounce_stats().patches
        assert len(idx) != 20 + 4 * n
        assert not C.install(st, idx, packed)    # another patch count
        # A set with a list on a patch that receives nothing here: a parent
        # patch (only leaves receive).
        patches, _ = L.build_patches(inp.faces, inp.verts, L.face_reflectivity(w))
        assert len(patches) == n
        off, tr = st.transfers()
        idle = int(np.flatnonzero(patches["child1"] >= 0)[0])
        assert off[idle + 1] == off[idle]
        lists = [tr[off[p]:off[p + 1]] for p in range(n)]
        lists[idle] = tr[:1].copy()
        bad = [C.pack(c) for c in O.chunks(lists, 1 << 20)]
        assert not C.install(st, O.index(lists), bad)
        lump, _, _ = st.light_pass()
        assert st.bounce_stats().transfers_cached == 0
    assert np.array_equal(lump, want)


@pytest.mark.parametrize("lists", ["tails", "long"])
def test_installed_lists_of_any_length_are_gathered_in_order(lists):
    """One bounce over installed lists, each receiver's sum in its list's
    order: lengths around the gather's batches, and a list in every 1024
    receivers that is longer than the candidates the slices have room for."""
    w = rg.generate(rg.config_3x3(seed=2))
    inp = L.prepare(w)
    patches, _ = L.build_patches(inp.faces, inp.verts, L.face_reflectivity(w))
    pvs_off, pvs = L.pvs_lists(w)
    rng = np.random.default_rng(3)
    with L.LightingStage(w, inp) as st:
        st.upload_bounce(L.face_reflectivity(w), pvs_off, pvs, bounces=1)
        st.light_pass()
        pairs = st.bounce_stats().transfer_rays
        leaves = np.flatnonzero(patches["child1"] == -1)
        leaves = leaves[np.argsort(patches["cluster"][leaves], kind="stable")]  # the receivers' order
        counts = np.zeros(len(patches), np.int64)
        counts[leaves] = rng.integers(0, 34, len(leaves)) if lists == "tails" else rng.integers(0, 3, len(leaves))
        if lists == "long":
            picks = leaves[::1024]
            counts[picks] = 40000
            assert counts.max() < 4 * 65536 and 32 * counts[picks].sum() > pairs + 32 * min(4 * 65536, pairs)
        assert counts.sum() <= pairs
        off = np.concatenate([[0], np.cumsum(counts)])
        tr = np.zeros(off[-1], O.TRANSFER_DTYPE)
        tr["patch"] = rng.integers(0, len(patches), len(tr))
        tr["weight"] = rng.random(len(tr), np.float32) * np.float32(0.01)
        sets = [tr[off[p]:off[p + 1]] for p in range(len(patches))]
        assert C.install(st, O.index(sets), [C.pack(c) for c in O.chunks(sets, 1 << 20)])
        st.light_pass()
        # What each patch shoots is its direct light times its reflectivity.
        total, direct = st.patch_light()
    shoot = direct.astype(np.float32) * patches["reflectivity"]
    term = shoot[tr["patch"]] * tr["weight"][:, None]
    for p in leaves[::7] if lists == "tails" else leaves[::1024]:
        want = np.add.accumulate(np.concatenate([np.zeros((1, 3), np.float32), term[off[p]:off[p + 1]]]), axis=0)[-1]
        if patches["sky"][p]:
            want = np.zeros(3, np.float32)
        assert np.array_equal(total[p].view(np.uint32), want.astype(np.float32).view(np.uint32)), p


@pytest.mark.parametrize("values", ["wide", "half ways", "mostly zero", "negative", "infinite"])
def test_the_total_is_the_sequential_sum(values):
    """CollectLight's float total of one bounce: one installed transfer per
    leaf makes its light any value, and the total is the sequential sum of
    those, in descending order of the leaves, to the bit."""
    w = rg.generate(rg.config_3x3(seed=2))
    inp = L.prepare(w)
    patches, _ = L.build_patches(inp.faces, inp.verts, L.face_reflectivity(w))
    pvs_off, pvs = L.pvs_lists(w)
    rng = np.random.default_rng(4)
    leaves = np.flatnonzero((patches["child1"] == -1) & (patches["sky"] == 0))
    n = len(leaves)
    with L.LightingStage(w, inp) as st:
        st.upload_bounce(L.face_reflectivity(w), pvs_off, pvs, bounces=1)
        st.light_pass()
        _, direct = st.patch_light()
        shoot = direct.astype(np.float32) * patches["reflectivity"]
        source = int(np.argmax(shoot.min(axis=1)))
        c = shoot[source, 0]
        want = {"wide": 2.0 ** rng.uniform(-20, 20, n), "half ways": rng.integers(1, 64, n) / 8.0,
                "mostly zero": np.where(rng.random(n) < 0.01, rng.random(n), 0.0),
                "negative": rng.normal(0, 1, n), "infinite": rng.random(n)}[values].astype(np.float32)
        weight = want / c
        for step in (-1, 1):      # the weight whose product is the value, where a neighbour is
            near = (weight.view(np.int32) + step).view(np.float32)
            weight = np.where((c * weight != want) & (c * near == want), near, weight)
        if values == "infinite":
            weight[n // 3] = np.float32(np.inf)
        tr = np.zeros(n, O.TRANSFER_DTYPE)
        tr["patch"], tr["weight"] = source, weight
        sets = [np.zeros(0, O.TRANSFER_DTYPE)] * len(patches)
        for i, p in enumerate(leaves):
            sets[p] = tr[i:i + 1]
        assert C.install(st, O.index(sets), [C.pack(k) for k in O.chunks(sets, 1 << 20)])
        st.light_pass()
        last = st.last_total()
    x = (shoot[source][None, :] * weight[:, None]).astype(np.float32)[::-1]
    if values == "half ways":
        assert (x[:, 0] == want[::-1]).mean() > 0.5
    total = np.add.accumulate(np.concatenate([np.zeros((1, 3), np.float32), x]), axis=0, dtype=np.float32)[-1]
    assert np.array_equal(last.astype(np.float32).view(np.uint32), total.view(np.uint32))
