"""The calls a map compile makes into this package, as cases that can be timed.

A case is one call (or one sequence of calls) through the public entry
points, at a size a compile has it at:

  trace       CudaRayTracer.trace_visibility / trace_closest: the IRayTracer
              seam, on CUDA tensors or on host arrays
  direct      LightingStage.direct_device: every sample's direct light with
              its supersampling passes, the map resident
  pass        LightingStage.light_pass_ranges_device: the whole lighting
              stage (gather, transfers, bounces, final pass) of a resident
              map, in one range or both
  compile     a context taking its next map: scene, world and bounce uploads
              from host arrays, both ranges lit, the lumps read back
  ambient     CudaAmbientSampler: leaf ambient's 162-ray cubes
  forward     Network.forward: the warm start's guess for every receiver
  gradient    Network.gradient: one training minibatch, forward and backward

Maps are the seeded room grids of roomgrid.py; leaf ambient runs on the
dm_lockdown geometry the tests keep, with seeded lighting.
"""
from __future__ import annotations

import dataclasses
import functools

import numpy as np
import torch

from hl2sdk_tools_sharp_b200 import ambient as A, bsp as B, learned as N, lighting as L, roomgrid as rg, tracer as T
from hl2sdk_tools_sharp_b200.workload import MAX_TRACE_LENGTH, ambient_directions

LOCKDOWN = "tests/golden/dm_lockdown.lumps.bin"


def listed():
    return [
        # A handful of test lines: the smallest call a host makes (a few
        # faces' shadow segments); launch and call cost.
        {"name": "trace_lines_1k", "kind": "trace", "query": "visibility", "host": False, "rays": 1021, "side": 3},
        # The sky tests of a few hundred faces: sky passes, brushes block.
        {"name": "trace_sky_1m", "kind": "trace", "query": "sky", "host": False, "rays": 1000003, "side": 5},
        # Closest hits of a large batch of sun and sky rays on the 8x8 map.
        {"name": "trace_closest_4m", "kind": "trace", "query": "closest", "host": False, "rays": 4194304, "side": 8},
        # The same seam from a host program: rays in host memory, bits back.
        {"name": "trace_host_250k", "kind": "trace", "query": "visibility", "host": True, "rays": 250001, "side": 4},
        # Direct light alone (no bounce wanted), a soft sun and a few panels
        # of texlights: the preview of a medium map.
        {"name": "direct_4x4_soft_sun", "kind": "direct", "side": 4, "scale": 8.0, "lights": 16, "spread": 2.0,
         "sun_samples": 30, "texlights": 2, "sky": True},
        # The plain small map: coarse luxels, four lights and the sun, LDR
        # alone, the reference's own stop threshold.
        {"name": "pass_3x3_ldr", "kind": "pass", "side": 3, "scale": 16.0, "lights": 4, "ranges": 1, "threshold": 1.0,
         "sky": False},
        # The benchmark map, LDR and HDR.
        {"name": "pass_8x8_both", "kind": "pass", "side": 8, "scale": 8.0, "lights": 64, "ranges": 3,
         "threshold": 0.1, "sky": True},
        # One map of a batch: everything from the host's arrays to its lumps.
        {"name": "compile_4x4_both", "kind": "compile", "side": 4, "scale": 8.0, "lights": 16, "ranges": 3,
         "threshold": 0.1, "sky": True},
        # A small map's candidate samples, from host memory.
        {"name": "ambient_host_768", "kind": "ambient", "host": True, "samples": 768},
        # A large map's candidate samples, on the device.
        {"name": "ambient_100k", "kind": "ambient", "host": False, "samples": 99991},
        # The guess for the 8x8 map's receivers.
        {"name": "forward_1m", "kind": "forward", "rows": 999080},
        # One minibatch of the network's training.
        {"name": "gradient_32k", "kind": "gradient", "rows": 32768},
    ]


def _log_int(rng, lo, hi):
    """A whole number spread over the logarithm of lo..hi."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "direct", "pass", "pass", "compile", "ambient", "forward",
                       "gradient"])
    if kind == "trace":
        return {"kind": kind, "query": rng.choice(["visibility", "sky", "closest"]), "host": rng.random() < 0.25,
                "rays": _log_int(rng, 33, 4194304), "side": rng.randint(2, 8)}
    if kind == "direct":
        side, soft = rng.randint(2, 4), rng.random() < 0.5
        return {"kind": kind, "side": side, "scale": rng.choice([8.0, 16.0]), "lights": rng.randint(1, 2 * side * side),
                "spread": round(rng.uniform(0.5, 5.0), 2) if soft else 0.0, "sun_samples": 30,
                "texlights": rng.randint(0, 2), "sky": rng.random() < 0.7}
    if kind in ("pass", "compile"):
        side = rng.randint(2, 6 if kind == "pass" else 4)
        return {"kind": kind, "side": side, "scale": rng.choice([8.0, 16.0]), "lights": rng.randint(1, side * side + 4),
                "ranges": rng.choice([1, 2, 3]), "threshold": rng.choice([0.1, 1.0]), "sky": rng.random() < 0.7}
    if kind == "ambient":
        return {"kind": kind, "host": rng.random() < 0.5, "samples": _log_int(rng, 7, 99991)}
    return {"kind": kind, "rows": _log_int(rng, 65, 999080) if kind == "forward" else _log_int(rng, 513, 65536)}


# ---------------------------------------------------------------- inputs

def _config(case, seed):
    c = rg.config_8x8(seed) if case.get("scale", 8.0) == 8.0 else rg.config_3x3(seed)
    return dataclasses.replace(c, side=case["side"], luxel_scale=case.get("scale", 8.0),
                               lights=case.get("lights", case["side"] ** 2), spot_fraction=0.5,
                               sky_ambient=case.get("sky", True), sun_spread=case.get("spread", 0.0),
                               sun_samples=case.get("sun_samples", 30), texlights=case.get("texlights", 0))


def _map(case, seed):
    """The case's map, lit by the seed: one geometry (every seed's lumps have
    one size, as a map does whose lights alone are edited), with the lights,
    sun and reflectivities drawn from the seed."""
    own, lit = rg.generate(_config(case, 1)), rg.generate(_config(case, seed))
    names = [f.name for f in dataclasses.fields(own) if f.name.startswith(("light_", "sun_", "ambient_"))]
    return dataclasses.replace(own, reflectivity=lit.reflectivity, **{k: getattr(lit, k) for k in names})


def _rays(world, query, n, seed):
    """(n, 7) float32 on the GPU, in the order a warp per 32 luxels emits
    them: runs of one face's luxels (of a small batch's, its first few)
    towards one target -- a light the face sees for visibility, a sky
    direction for the sky tests, the sun or a sky direction for the closest
    hits."""
    rng = np.random.default_rng([seed, 0x5241])
    dev = torch.device("cuda")
    nrm = world.face_normal.astype(np.float64)
    poly = np.stack(world.face_verts).astype(np.float64)
    if query == "visibility":
        to = world.light_origin[None, :, :] - poly.mean(1)[:, None, :]
        ok = (to * nrm[:, None, :]).sum(-1) > 1.0
        ok &= world.pvs[world.face_cluster][:, world.light_cluster]
        target = world.light_origin.astype(np.float32)
    else:
        dirs = ambient_directions().astype(np.float32)
        if query == "closest":
            # The sun as often as all of the sky's directions together.
            dirs = np.concatenate([dirs, np.repeat(world.sun_direction[None, :].astype(np.float32), len(dirs), 0)])
        ok = -(nrm @ dirs.T.astype(np.float64)) > 0.001
        target = dirs * -MAX_TRACE_LENGTH
    pf, pt = np.nonzero(ok)
    size = (world.face_extents + 1).astype(np.int64)
    count = np.minimum(size[:, 0] * size[:, 1], max(32, n // 32))
    pick, have = [], 0
    while have < n:
        k = rng.integers(0, len(pf), 1 + int((n - have) / max(1.0, float(count[pf].mean()))))
        pick.append(k)
        have += int(count[pf[k]].sum())
    pick = np.concatenate(pick)
    f, t = torch.from_numpy(pf[pick]).to(dev), torch.from_numpy(pt[pick]).to(dev)
    reps = torch.from_numpy(count).to(dev)[f]
    run = torch.repeat_interleave(torch.arange(len(f), device=dev), reps)[:n]
    first = torch.cumsum(reps, 0) - reps
    cell = torch.arange(n, device=dev) - first[run]
    face = f[run]
    wide = torch.from_numpy(size[:, 0]).to(dev)[face]
    S, Tv = world.face_s.astype(np.float64), world.face_t.astype(np.float64)
    inv = torch.linalg.inv(torch.from_numpy(np.stack([S[:, :3], Tv[:, :3], nrm], 1)).to(dev))
    off = torch.from_numpy(np.stack([world.face_mins[:, 0] + 0.5 - S[:, 3], world.face_mins[:, 1] + 0.5 - Tv[:, 3],
                                     world.face_dist.astype(np.float64)], 1)).to(dev)
    at = off[face]
    at[:, 0] += cell % wide
    at[:, 1] += cell // wide
    p = (inv[face] @ at[:, :, None])[:, :, 0]
    lo, hi = torch.from_numpy(poly.min(1)).to(dev), torch.from_numpy(poly.max(1)).to(dev)
    p = torch.minimum(torch.maximum(p, lo[face]), hi[face]) + torch.from_numpy(nrm).to(dev)[face]
    rays = torch.empty((n, 7), dtype=torch.float32, device=dev)
    rays[:, 0:3] = p.float()
    end = torch.from_numpy(target).to(dev)[t[run]]
    if query != "visibility":
        end = end + rays[:, 0:3]
    rays[:, 3:6] = end - rays[:, 0:3]
    rays[:, 6] = 1.0
    return rays


@functools.lru_cache(maxsize=1)
def _lockdown():
    """The kept geometry lumps: "VLMP", a count, then (id, version, length,
    bytes) each."""
    with open(LOCKDOWN, "rb") as fh:
        blob = fh.read()
    out, p = {}, 8
    for _ in range(int(np.frombuffer(blob, "<i4", 1, 4)[0])):
        i, ver, ln = (int(x) for x in np.frombuffer(blob, "<i4", 3, p))
        out[i] = (ver, blob[p + 12:p + 12 + ln])
        p += 12 + ln
    return out


def _ambient_lumps(seed):
    """The geometry with a seeded lighting lump, reflectivities and sky."""
    lumps = dict(_lockdown())
    rng = np.random.default_rng([seed, 0x414D])
    faces = np.frombuffer(lumps[B.LUMP_FACES][1], B.FACE)
    texinfo = np.frombuffer(lumps[B.LUMP_TEXINFO][1], B.TEXINFO)
    td = np.zeros(int(texinfo["texdata"].max()) + 1, A.TEXDATA)
    td["reflectivity"] = rng.uniform(0.05, 0.9, (len(td), 3)).astype(np.float32)
    styles = (faces["styles"] != 255).sum(1)
    size = (faces["lm_size"].astype(np.int64) + 1).prod(1) * 4 * np.maximum(styles, 1)
    end = int(np.max(np.where(faces["lightofs"] >= 0, faces["lightofs"] + 4 * size, 0)))
    light = rng.integers(0, 256, end + 64, dtype=np.uint8)
    light[3::4] = rng.integers(-9, 3, len(light[3::4])).astype(np.int8).view(np.uint8)
    wl = np.zeros(2, A.WORLDLIGHT)
    wl["type"] = (1, A.EMIT_SKYAMBIENT)
    wl["intensity"][1] = rng.uniform(0.1, 1.0, 3)
    lumps[B.LUMP_TEXDATA] = (0, td.tobytes())
    lumps[B.LUMP_LIGHTING] = (1, light.tobytes())
    lumps[A.LUMP_WORLDLIGHTS] = (0, wl.tobytes())
    return lumps


def _positions(n, seed):
    """n points in the map's open leaves."""
    ver, raw = _lockdown()[B.LUMP_LEAFS]
    leaves = np.frombuffer(raw, B.LEAF_V0 if ver == 0 else B.LEAF_V1)
    leaves = leaves[(leaves["contents"] & A.CONTENTS_SOLID) == 0]
    rng = np.random.default_rng([seed, 0x504F])
    pick = np.sort(rng.integers(0, len(leaves), n))    # leaf after leaf, as the stage plans them
    lo, hi = leaves["mins"][pick].astype(np.float64), leaves["maxs"][pick].astype(np.float64)
    return (lo + rng.uniform(0.02, 0.98, (n, 3)) * (hi - lo)).astype(np.float32)


def _network(seed):
    """The flat parameters of a network part-way through its training."""
    rng = np.random.default_rng([seed, 0x4E45])
    flat = np.zeros(N.PARAMS, np.float32)
    for name, shape in N.SHAPES.items():
        v = rng.normal(size=shape) * (np.sqrt(2.0 / shape[0]) if len(shape) == 2 else 0.05)
        flat[N.OFFSETS[name]:N.OFFSETS[name] + v.size] = v.astype(np.float32).ravel()
    return flat


def _features(rows, seed):
    """The receivers' inputs as the bounce's features lay them out (unit
    normals, logarithms scaled to about one, eleven zeros) and the log of
    their converged light."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.rand((rows, N.INPUTS), generator=g, device="cuda")
    axis = torch.randint(0, 6, (rows,), generator=g, device="cuda")
    x[:, 0:3] = torch.nn.functional.one_hot(axis % 3, 3) * torch.where(axis < 3, 1.0, -1.0)[:, None]
    x[:, 21:] = 0.0
    t = 6.0 * x[:, 10:13] + 0.5 * torch.rand((rows, 3), generator=g, device="cuda")
    return x.to(torch.bfloat16).contiguous(), t.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "trace":
        w = rg.generate(_config(case, seed))
        n = case["rays"]
        s["tracer"] = T.CudaRayTracer(T.make_triangles(w.tri_verts, w.tri_ids))
        s["options"] = T.RayTraceOptions(0.0, sky_does_not_block=case["query"] == "sky")
        rays = _rays(w, case["query"], n, seed)
        if case["host"]:
            s["rays"] = rays.cpu().numpy()
            s["out"] = np.zeros(n, T.HIT_DTYPE) if case["query"] == "closest" else np.zeros((n + 63) // 64, np.uint64)
        else:
            s["rays"] = rays
            s["out"] = (torch.zeros((n, 2), dtype=torch.int32, device="cuda") if case["query"] == "closest"
                        else torch.zeros((n + 63) // 64, dtype=torch.int64, device="cuda"))
    elif kind in ("direct", "pass", "compile"):
        w = _map(case, seed)
        inputs = L.prepare(w, hdr=case.get("ranges", 1) & L.RANGE_HDR != 0)
        st = L.LightingStage(w, inputs)
        s["stage"] = st
        if kind == "direct":
            s["out"] = torch.zeros((len(inputs.samples), 4), dtype=torch.float32, device="cuda")
        else:
            off, lst = L.pvs_lists(w)
            s["bounce"] = (L.face_reflectivity(w), off, lst)
            st.upload_bounce(*s["bounce"], bounces=100, threshold=case["threshold"])
            bufs = []
            for r in (L.RANGE_LDR, L.RANGE_HDR):
                if not case["ranges"] & r:
                    bufs.append(None)
                elif kind == "pass":
                    bufs.append(torch.zeros(st.lighting_size(), dtype=torch.uint8, device="cuda"))
                else:
                    bufs.append(torch.zeros(st.lighting_size(), dtype=torch.uint8, pin_memory=True).numpy())
            s["ldr"], s["hdr"] = bufs
            if kind == "compile":
                s["inputs"], s["tris"] = inputs, T.make_triangles(w.tri_verts, w.tri_ids)
    elif kind == "ambient":
        s["sampler"] = A.CudaAmbientSampler(_ambient_lumps(seed))
        pos = _positions(case["samples"], seed)
        s["positions"] = pos if case["host"] else torch.from_numpy(pos).cuda()
        if not case["host"]:
            s["out"] = torch.zeros((len(pos), A.SIDES, 3), dtype=torch.float32, device="cuda")
    else:
        # The network lives on the device of a tracer's context.
        s["owner"] = T.CudaRayTracer(np.array([[0, 0, 0, 1, 0, 0, 0, 1, 0]], np.float32))
        s["net"] = N.Network(s["owner"], seed=1)
        s["net"].set_params(_network(seed))
        s["x"], s["target"] = _features(case["rows"], seed)
        if kind == "forward":
            s["out"] = torch.zeros((case["rows"], N.OUTPUTS), dtype=torch.float32, device="cuda")
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "trace":
        if case["query"] == "closest":
            out = s["tracer"].trace_closest(s["rays"], s["out"], s["options"])
        else:
            out = s["tracer"].trace_visibility(s["rays"], s["out"], s["options"])
        # Hits are records (surface, fraction): their words.
        return out.view(np.int32 if out.dtype == T.HIT_DTYPE else np.int64) if case["host"] else out
    if kind == "direct":
        return s["stage"].direct_device(s["out"])
    if kind == "pass":
        s["stage"].light_pass_ranges_device(s["ldr"], s["hdr"], case["ranges"])
        return [s["ldr"], s["hdr"]]
    if kind == "compile":
        st = s["stage"]
        st.tracer.upload_scene(s["tris"])
        st.upload_world(s["inputs"])
        st.upload_bounce(*s["bounce"], bounces=100, threshold=case["threshold"])
        ldr, hdr, ofs, _, _ = st.light_pass_ranges(case["ranges"], s["ldr"], s["hdr"])
        return [ldr, hdr, ofs]
    if kind == "ambient":
        if case["host"]:
            return s["sampler"].cubes(s["positions"])
        return s["sampler"].cubes_device(s["positions"], out=s["out"])
    if kind == "forward":
        return s["net"].forward(s["x"], out=s["out"])
    grad, loss = s["net"].gradient(s["x"], s["target"])
    return [grad, loss]


# ---------------------------------------------------------------- floors

def work(case):
    kind = case["kind"]
    if kind == "trace":
        out = 8.0 if case["query"] == "closest" else 0.125
        return {"bytes": case["rays"] * (28.0 + out), "flops": 0.0}
    if kind in ("direct", "pass", "compile"):
        w = rg.generate(_config(case, 1))
        luxels, tris = float(w.luxel_counts().sum()), float(len(w.tri_ids))
        if kind == "direct":
            return {"bytes": luxels * (16.0 + 16.0) + 48.0 * tris, "flops": 0.0}
        ranges = 2 if case["ranges"] == 3 else 1
        record = 56.0 if kind == "compile" else 16.0
        return {"bytes": luxels * (record + 4.0 * ranges) + 48.0 * tris, "flops": 0.0}
    if kind == "ambient":
        return {"bytes": case["samples"] * (12.0 + 72.0), "flops": 0.0}
    macs = N.INPUTS * N.HIDDEN + N.HIDDEN * N.HIDDEN + N.HIDDEN * N.OUTPUTS
    if kind == "forward":
        return {"bytes": case["rows"] * (2.0 * N.INPUTS + 4.0 * N.OUTPUTS), "flops": 2.0 * macs * case["rows"]}
    # Forward, then per layer the weight gradient, and per layer but the
    # first the gradient of its input.
    back = macs + macs - N.INPUTS * N.HIDDEN
    return {"bytes": case["rows"] * (2.0 * N.INPUTS + 4.0 * N.OUTPUTS) + 4.0 * N.PARAMS,
            "flops": 2.0 * (macs + back) * case["rows"]}


def exact(case, seed):
    """The network's cases in 64 bits: the products of its BF16 weights and
    inputs.  Hits, bits and lumps are whole numbers; the other light values
    have no closed form."""
    if case["kind"] not in ("forward", "gradient"):
        return None
    x, target = _features(case["rows"], seed)
    flat = torch.from_numpy(_network(seed)).cuda()
    p = {k: flat[N.OFFSETS[k]:N.OFFSETS[k] + int(np.prod(v))].reshape(v) for k, v in N.SHAPES.items()}
    p = {k: (v.to(torch.bfloat16) if k[0] == "w" else v).double() for k, v in p.items()}
    x = x.double()
    h1 = torch.relu(x @ p["w1"] + p["b1"])
    h2 = torch.relu(h1 @ p["w2"] + p["b2"])
    y = h2 @ p["w3"] + p["b3"]
    if case["kind"] == "forward":
        return y
    e = y - target.double()
    dy = 2.0 * e / e.numel()
    dz2 = (dy @ p["w3"].T) * (h2 > 0)
    dz1 = (dz2 @ p["w2"].T) * (h1 > 0)
    grad = [x.T @ dz1, dz1.sum(0), h1.T @ dz2, dz2.sum(0), h2.T @ dy, dy.sum(0)]
    return [torch.cat([g.ravel() for g in grad]), float((e * e).mean())]
