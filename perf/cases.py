"""The work that the baker is timed on, through its Python entry points.

Eleven kinds of work, one or two listed cases of each.  What they stand for:

  gi         Relight's own global-illumination bake: emit and trace the photons, gather the photonmap, final-gather
             the lightmap.  gi_terrain_1024 is the benchmark's terrain (154k triangles, a million photons, 256
             samples); gi_small_97 a preview bake of a small scene into a small odd-sized map, where launches count.
  room       direct light (point, spot and area lights) and ambient occlusion of one lightmap.  room_256 is the
             benchmark's room; room_textured_48 the smallest one that the tests bake, with alpha-tested textures.
  batch      many uneven bakes (direct + AO + final gather) in one launch, as the batch benchmark and the server do.
  knn        the photonmap estimate from the k nearest photon deposits.
  radiosity  hemisphere form factors and the Jacobi solve over them (the benchmark's 16,384 patches).
  pairwise   Relight's own point-to-point form factors, CSR to the host.
  rays       rays against a scene's BVH, as the ray-query interface takes them (closest or first hit).
  denoise    the denoiser's forward pass over one lightmap's features.
  train      optimiser steps of the denoiser (forward, backward, Adam) and the updated weights.
  post       expand, blur and RGBM encoding of a finished lightmap, as saving one does.

Sizes that a case does not name are drawn from the numbers in the case, contents from the seed.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from relight_b200 import _abi, batch, denoise, scenes
from relight_b200.api import AmbientOcclusionSettings, IndirectLightSettings
from relight_b200.denoise import Denoiser
from relight_b200.device import DeviceMap, PhotonRecords, Relight

RGBM = 2  # StorageFormat of the encoded lightmap


def listed():
    return [
        # the benchmark's headline step
        {"name": "gi_terrain_1024", "kind": "gi", "verts": 256, "boxes": 2000, "width": 1024, "height": 1024,
         "photonmap": 1024, "samples": 256, "passes": 8, "bounces": 3},
        # a preview: small scene, small odd map, few samples
        {"name": "gi_small_97", "kind": "gi", "verts": 48, "boxes": 40, "width": 97, "height": 75, "photonmap": 128,
         "samples": 32, "passes": 1, "bounces": 1},
        # the benchmark's direct + AO room
        {"name": "room_256", "kind": "room", "size": 256, "boxes": 8, "textured": False, "samples": 64,
         "distance": 2.0},
        # the smallest bake, with cut-out textures in the shadow rays' way
        {"name": "room_textured_48", "kind": "room", "size": 48, "boxes": 8, "textured": True, "samples": 16,
         "distance": 2.0},
        # uneven jobs over a few scenes, the batch benchmark's recipe at a twentieth of its jobs
        {"name": "batch_24", "kind": "batch", "jobs": 24, "scenes": 4, "tris_lo": 1000, "tris_hi": 60000,
         "side_lo": 32, "side_hi": 512, "ao": 64, "samples": 128, "shape": 4},
        # the benchmark's k = 100 estimate within 2 units
        {"name": "knn_512", "kind": "knn", "side": 512, "records": 600000, "k": 100, "radius": 2.0},
        # the benchmark's radiosity step
        {"name": "radiosity_128", "kind": "radiosity", "size": 128, "rays": 512, "iters": 50},
        # Relight's own form factors over a quarter of those patches
        {"name": "pairwise_64", "kind": "pairwise", "size": 64, "threshold": 0.1},
        # a million incoherent rays, closest hit
        {"name": "rays_1m", "kind": "rays", "verts": 128, "boxes": 500, "rays": 1 << 20, "any_hit": False},
        # one full-size lightmap through the denoiser
        {"name": "denoise_1024", "kind": "denoise", "images": 1, "height": 1024, "width": 1024},
        # training steps as the trainer takes them
        {"name": "train_16x64", "kind": "train", "steps": 8, "batch": 16, "patch": 64, "patches": 64},
        # what saving a full-size lightmap does
        {"name": "post_1024", "kind": "post", "width": 1024, "height": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gi", "gi", "room", "room", "batch", "knn", "radiosity", "pairwise", "rays", "denoise", "train",
                       "post"])
    if kind == "gi":
        w, h = _log(rng, 48, 1024), _log(rng, 48, 1024)
        return {"kind": kind, "verts": _log(rng, 24, 256), "boxes": _log(rng, 10, 2000), "width": w, "height": h,
                "photonmap": _log(rng, 64, 1024), "samples": _log(rng, 16, 256), "passes": rng.randint(1, 8),
                "bounces": rng.randint(1, 3)}
    if kind == "room":
        return {"kind": kind, "size": _log(rng, 32, 384), "boxes": rng.randint(2, 16),
                "textured": rng.random() < 0.3, "samples": _log(rng, 16, 128), "distance": rng.choice([1.0, 2.0, 5.0])}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(4, 24), "scenes": rng.randint(1, 4), "tris_lo": 1000,
                "tris_hi": _log(rng, 4000, 60000), "side_lo": 32, "side_hi": _log(rng, 64, 512),
                "ao": rng.choice([16, 32, 64]), "samples": rng.choice([16, 64, 128]), "shape": rng.randrange(1 << 20)}
    if kind == "knn":
        return {"kind": kind, "side": _log(rng, 48, 512), "records": _log(rng, 20000, 600000),
                "k": rng.choice([10, 32, 50, 100, 128]), "radius": rng.choice([1.0, 2.0, 3.0])}
    if kind == "radiosity":
        return {"kind": kind, "size": rng.randint(24, 160), "rays": rng.choice([64, 100, 128, 256, 500, 512]),
                "iters": rng.randint(10, 60)}
    if kind == "pairwise":
        return {"kind": kind, "size": rng.randint(16, 128), "threshold": rng.choice([0.05, 0.1, 0.2])}
    if kind == "rays":
        return {"kind": kind, "verts": _log(rng, 24, 256), "boxes": _log(rng, 10, 1000), "rays": _log(rng, 1000, 4000000),
                "any_hit": rng.random() < 0.5}
    if kind == "denoise":
        return {"kind": kind, "images": rng.choice([1, 1, 2]), "height": _log(rng, 40, 1024), "width": _log(rng, 40, 1024)}
    if kind == "train":
        return {"kind": kind, "steps": rng.randint(2, 8), "batch": rng.choice([4, 8, 16]),
                "patch": rng.choice([32, 48, 64]), "patches": 64}
    return {"kind": kind, "width": _log(rng, 48, 1400), "height": _log(rng, 48, 1400)}


# ------------------------------------------------------------------ shared

def _stream():
    return torch.cuda.current_stream().cuda_stream


def _p(t):
    return C.c_void_p(t.data_ptr() if isinstance(t, torch.Tensor) else t.ctypes.data)


class _Lumels:
    """One lumel array of a DeviceMap for torch, which keeps this object, and through it the map, as long as the tensor."""

    def __init__(self, owner, field):
        self.owner = owner
        n, whole = owner.width * owner.height, field in ("flags", "photons")
        self.__cuda_array_interface__ = {"shape": (n,) if whole else (n, 3), "typestr": "<i4" if whole else "<f4",
                                         "data": (owner.device_arrays()[field], False), "version": 3, "strides": None}


def map_tensor(dev_map, field):
    return torch.as_tensor(_Lumels(dev_map, field), device="cuda")


def _terrain(case, seed, photonmap, **kw):
    tiles = max(1, math.ceil((case["verts"] - 1) / 255))
    return scenes.terrain_scene(seed=seed, verts=case["verts"], n_boxes=case["boxes"], size=photonmap, tiles=tiles, **kw)


def _tri_count(case):
    return 2 * (case["verts"] - 1) ** 2 + 12 * case["boxes"]


def _heights(side, seed, amplitude=5.0, extent=255.0):
    """A smooth random height field over [0, extent]^2, sampled at points (x, z) by the returned function."""
    g = np.random.default_rng(seed)
    waves = [(g.uniform(0.02, 0.3, 2), g.uniform(0, 6.28), g.uniform(0.1, 1.0)) for _ in range(12)]
    total = sum(a for _, _, a in waves)

    def at(x, z):
        y = np.zeros_like(x)
        for (kx, kz), ph, a in waves:
            y = y + a * np.sin(kx * x + kz * z + ph)
        return amplitude * y / total
    return at


# ------------------------------------------------------------------ prepare

def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


# gi: the values are averages over hundreds of millions of traced rays, more than 64-bit brute force can follow here,
# so there is no exact().

def _prepare_gi(case, seed):
    wl = _terrain(case, seed, case["photonmap"], fg_samples=case["samples"], passes=case["passes"],
                  bounces=case["bounces"])
    rl = Relight(stream=_stream(), seed=seed)
    ds = rl.device_scene(wl.scene)
    if (case["width"], case["height"]) == (case["photonmap"], case["photonmap"]):
        lm = wl.lightmap._device
    else:
        lm = DeviceMap(0, case["width"], case["height"])
        for m in range(len(wl.meshes)):
            lm.add_mesh(ds, m, rl.stream)
    pms = [m._device for m in wl.scene.flat.photonmaps]
    return {"kind": "gi", "wl": wl, "rl": rl, "ds": ds, "lm": lm, "pms": pms, "seed": seed,
            "out": [map_tensor(lm, "color"), map_tensor(pms[0], "gathered"), map_tensor(pms[0], "photons")]}


def _run_gi(s):
    wl, rl = s["wl"], s["rl"]
    for m in s["pms"]:
        m.clear(colors=True, photons=True, stream=rl.stream)
    rl.emit_photons(wl.scene, wl.settings, seed=s["seed"] * 2 + 1)
    denoise.bake_fg(rl, s["ds"], s["lm"], s["pms"], wl.settings, wl.settings.final_gather_samples, s["seed"] * 2 + 2,
                    stream=rl.stream)
    return s["out"]


def _work_gi(case):
    texels, pm, tris = case["width"] * case["height"], case["photonmap"] ** 2, _tri_count(case)
    rays = 0.8 * texels * case["samples"] + 125000 * case["passes"] * 1.5
    # lumels in, colours out, the photonmap's counts and colours out, the geometry in; per ray a direction, a walk of
    # log2(triangles) two-box nodes and two triangles
    return {"bytes": 40.0 * texels + 28.0 * pm + 48.0 * tris, "flops": rays * (60 + 24 * math.log2(tris) + 60)}


# room: a shadow ray ends on its lumel's own surface, and rounding at that end decides whether the surface stands in
# its way, so there is no exact()

def _prepare_room(case, seed):
    wl = scenes.room_scene(seed=seed, size=case["size"], n_boxes=case["boxes"], textured=case["textured"])
    rl = Relight(stream=_stream(), seed=seed)
    rl.device_scene(wl.scene)
    return {"kind": "room", "wl": wl, "rl": rl, "seed": seed, "lm": wl.lightmap._device,
            "ao": AmbientOcclusionSettings(case["samples"], 0.8, case["distance"], 1.0),
            "out": map_tensor(wl.lightmap._device, "color")}


def _run_room(s):
    wl, rl = s["wl"], s["rl"]
    s["lm"].clear(colors=True, photons=False, stream=rl.stream)
    rl.bake_direct_light(wl.scene, wl.mesh)
    rl.bake_ambient_occlusion(wl.scene, wl.mesh, None, s["ao"], seed=s["seed"])
    return s["out"]


def _work_room(case):
    texels, tris = case["size"] ** 2, 12 + 12 * case["boxes"]
    rays = 0.75 * texels * (18 + case["samples"])
    return {"bytes": 40.0 * texels + 48.0 * tris, "flops": rays * (60 + 24 * math.log2(tris) + 30)}


# batch

def _prepare_batch(case, seed):
    shapes = random.Random(case["shape"])
    wls, counts = [], []
    for k in range(case["scenes"]):
        t = _log(shapes, case["tris_lo"], case["tris_hi"])
        shape = {"verts": max(8, int(round(math.sqrt(0.45 * t))) + 1), "boxes": max(1, int(round(t / 120)))}
        wls.append(_terrain(shape, seed * 16 + k, 128, fg_samples=case["samples"], passes=1))
        counts.append(_tri_count(shape))
    jobs = [scenes.BatchJobSpec(shapes.randrange(case["scenes"]), _log(shapes, case["side_lo"], case["side_hi"]),
                                seed * 1000 + q) for q in range(case["jobs"])]
    wl = scenes.BatchWorkload(wls, counts, jobs, AmbientOcclusionSettings(case["ao"], 0.8, 2.0, 1.0))
    rb = batch.make_resident(wl, stream=_stream())
    return {"kind": "batch", "rb": rb, "batch": batch.Batch(rb.jobs), "stream": _stream(),
            "out": [map_tensor(m, "color") for m in rb.lightmaps]}


def _run_batch(s):
    s["rb"].clear(stream=s["stream"])
    s["batch"].launch(s["stream"])
    return s["out"]


def _work_batch(case):
    shapes = random.Random(case["shape"])
    tris = [_log(shapes, case["tris_lo"], case["tris_hi"]) for _ in range(case["scenes"])]
    texels = rays = 0.0
    for _ in range(case["jobs"]):
        t, side = tris[shapes.randrange(case["scenes"])], _log(shapes, case["side_lo"], case["side_hi"])
        texels += side * side
        rays += 0.8 * side * side * (5 + case["ao"] + case["samples"]) * (24 * math.log2(t) + 120)
    return {"bytes": 40.0 * texels + 48.0 * sum(tris), "flops": rays}


# knn

def _knn_inputs(case, seed):
    rng = np.random.default_rng(seed)
    side, n = case["side"], case["records"]
    ground = _heights(side, seed + 1)
    t = (np.arange(side) + 0.5) / side * 255.0
    x, z = np.meshgrid(t, t)
    pos = np.stack([x, ground(x, z), z], -1).reshape(-1, 3).astype(np.float32)
    flags = (rng.random(side * side) < 0.9).astype(np.int32)
    # deposits: most spread over the ground, some in the pools under the point lights
    px, pz = rng.uniform(0, 255, n), rng.uniform(0, 255, n)
    pool = rng.random(n) < 0.2
    px[pool] = np.clip(rng.choice([64, 191], pool.sum()) + rng.normal(0, 25, pool.sum()), 0, 255)
    pz[pool] = np.clip(rng.choice([64, 191], pool.sum()) + rng.normal(0, 25, pool.sum()), 0, 255)
    rec = np.concatenate([np.stack([px, ground(px, pz), pz], 1), rng.uniform(0.05, 1.0, (n, 3))], 1).astype(np.float32)
    return pos, flags, rec


def _prepare_knn(case, seed):
    pos, flags, rec = _knn_inputs(case, seed)
    pm = DeviceMap(1, case["side"], case["side"])
    pm.upload(stream=_stream(), flags=flags, position=pos)
    records = PhotonRecords(case["records"])
    n = case["records"]
    records.upload(rec, np.arange(n), np.zeros(n, np.int32), np.zeros(n, np.int32))
    return {"kind": "knn", "pm": pm, "records": records, "k": case["k"], "radius": case["radius"],
            "stream": _stream(), "out": map_tensor(pm, "gathered")}


def _run_knn(s):
    s["records"].gather_knn(s["pm"], 0, s["k"], s["radius"], s["stream"])
    return s["out"]


def _work_knn(case):
    texels = case["side"] ** 2
    return {"bytes": 28.0 * texels + 32.0 * case["records"], "flops": 0.9 * texels * case["k"] * 16.0}


def _exact_knn(case, seed):
    pos, flags, rec = _knn_inputs(case, seed)
    out = torch.zeros(len(pos), 3, dtype=torch.float64, device="cuda")
    rec = torch.tensor(rec.astype(np.float64), device="cuda")
    rec = rec[rec[:, 0].argsort()]
    keys = rec[:, 0].contiguous()
    valid = torch.tensor(np.nonzero(flags)[0], device="cuda")
    p = torch.tensor(pos.astype(np.float64), device="cuda")[valid]
    order = (p[:, 0] * 4).floor() * 4096 + p[:, 2] * 4  # columns a quarter unit wide, along z
    order = order.argsort()
    r = case["radius"]
    for b in range(0, len(order), 2048):
        at = order[b:b + 2048]
        q = p[at]
        lo = torch.searchsorted(keys, (q[:, 0].min() - r - 1e-3).reshape(1))
        hi = torch.searchsorted(keys, (q[:, 0].max() + r + 1e-3).reshape(1))
        near = rec[int(lo):int(hi)]
        near = near[(near[:, 2] >= q[:, 2].min() - r - 1e-3) & (near[:, 2] <= q[:, 2].max() + r + 1e-3)]
        if not len(near):
            continue
        d2 = ((q[:, None, 0] - near[None, :, 0]) ** 2 + (q[:, None, 1] - near[None, :, 1]) ** 2
              + (q[:, None, 2] - near[None, :, 2]) ** 2)
        k = min(case["k"], len(near))
        v, j = d2.topk(k, dim=1, largest=False)
        w = (v <= r * r).double()
        mean = (near[j][:, :, 3:6] * w[:, :, None]).sum(1) / w.sum(1, keepdim=True).clamp_min(1)
        out[valid[at]] = mean
    return out


# radiosity

def _patches(case, seed):
    wl = scenes.radiosity_room(size=case["size"])
    rl = Relight(stream=_stream(), seed=seed)
    ds = rl.device_scene(wl.scene)
    g = wl.radiancemap._device.download(rl.stream, fields=("flags", "position", "normal"))
    valid = np.nonzero(g["flags"] & 1)[0]
    pos, nrm = (torch.from_numpy(np.ascontiguousarray(g[f][valid])).cuda() for f in ("position", "normal"))
    return wl, rl, ds, valid, pos, nrm


def _light(n, seed):
    rng = np.random.default_rng(seed)
    rho = rng.uniform(0.3, 0.9, (n, 3)).astype(np.float32)
    E = np.zeros((n, 3), np.float32)
    E[rng.choice(n, 16, replace=False)] = 1.0
    return E, rho


def _prepare_radiosity(case, seed):
    wl, rl, ds, valid, pos, nrm = _patches(case, seed)
    n, texels = len(valid), case["size"] ** 2
    pot = np.full(texels, -1, np.int32)
    pot[valid] = np.arange(n, dtype=np.int32)
    E, rho = _light(n, seed)
    cap = n * case["rays"]
    return {"kind": "radiosity", "keep": (wl, rl), "ds": ds, "n": n, "pos": pos, "nrm": nrm, "pot": pot,
            "rays": case["rays"], "iters": case["iters"], "cap": cap, "seed": seed, "stream": _stream(),
            "mesh_map": np.array([0], np.int32), "dims": np.array([[case["size"]] * 2], np.int32),
            "base": np.array([0], np.int64), "E": torch.from_numpy(E).cuda(), "rho": torch.from_numpy(rho).cuda(),
            "row": torch.empty(n + 1, dtype=torch.int64, device="cuda"),
            "cols": torch.zeros(cap, dtype=torch.int32, device="cuda"),
            "vals": torch.zeros(cap, dtype=torch.float32, device="cuda"),
            "B": torch.empty((n, 3), dtype=torch.float32, device="cuda")}


def _run_radiosity(s):
    L, nnz = _abi.lib(), C.c_int64()
    _abi.check(L.rl_ff_hemisphere_device(s["ds"].handle, s["n"], _p(s["pos"]), _p(s["nrm"]), s["rays"], 100.0, s["seed"],
                                         _p(s["mesh_map"]), 1, _p(s["dims"]), _p(s["base"]), _p(s["pot"]),
                                         s["pot"].size, _p(s["row"]), _p(s["cols"]), _p(s["vals"]), s["cap"],
                                         C.byref(nnz), s["stream"]))
    _abi.check(L.rl_radiosity_solve(s["n"], _p(s["row"]), _p(s["cols"]), _p(s["vals"]), _p(s["E"]), _p(s["rho"]),
                                    s["iters"], _p(s["B"]), s["stream"]))
    return [s["row"], s["cols"], s["vals"], s["B"]]


def _work_radiosity(case):
    n, rays = case["size"] ** 2, case["size"] ** 2 * case["rays"]
    nnz = 0.87 * rays
    return {"bytes": 8.0 * nnz + 60.0 * n, "flops": rays * 200.0 + case["iters"] * 6.0 * nnz}


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 over int64 tensors of 32-bit words; four words of 24-bit uniforms."""
    m = 0xFFFFFFFF
    k0, k1 = seed & m, (seed >> 32) & m
    c = [c0, c1, c2, c3]

    def mulhilo(a, b):  # 32 x 32 -> 64 bits, in pieces that stay below 2^63
        lo, hi = a * (b & 0xFFFF), a * (b >> 16)
        full_lo = (lo + ((hi & 0xFFFF) << 16))
        return ((hi >> 16) + (full_lo >> 32)) & m, full_lo & m
    for _ in range(10):
        h0, l0 = mulhilo(c[0], 0xD2511F53)
        h1, l1 = mulhilo(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return [(x >> 8).double() * 2.0 ** -24 for x in c]


def _exact_radiosity(case, seed):
    """The room is an empty box: every ray ends where it first leaves it, and the radiancemap's charts are rectangles."""
    s, half = case["size"], case["size"] // 2
    q = s // 4
    if s % 4:
        return None  # charts that do not end on texel edges: which texels count is decided by rounding
    dims = torch.tensor([10.0, 5.0, 10.0], dtype=torch.float64, device="cuda")
    # face (axis, side): chart rectangle, the axis that runs along u and the one along v
    charts = {(1, 0): (0, 0, half, half, 2, 0), (1, 1): (half, 0, s, half, 2, 0),
              (0, 0): (0, half, half, half + q, 2, 1), (0, 1): (half, half, s, half + q, 2, 1),
              (2, 0): (0, half + q, half, s, 0, 1), (2, 1): (half, half + q, s, s, 0, 1)}
    pos = torch.zeros(s * s, 3, dtype=torch.float64, device="cuda")
    nrm = torch.zeros_like(pos)
    at = torch.arange(s, device="cuda")
    for (axis, side), (x0, y0, x1, y1, au, av) in charts.items():
        y, x = torch.meshgrid(at[y0:y1], at[x0:x1], indexing="ij")
        i = (y * s + x).reshape(-1)
        pos[i, axis] = side * dims[axis]
        pos[i, au] = (x.reshape(-1).double() + 0.5 - x0) / (x1 - x0) * dims[au]
        pos[i, av] = (y.reshape(-1).double() + 0.5 - y0) / (y1 - y0) * dims[av]
        nrm[i, axis] = 1.0 - 2.0 * side
    n, rays = s * s, case["rays"]
    F = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    for b in range(0, n, 1024):
        item = torch.arange(b, min(b + 1024, n), device="cuda").repeat_interleave(rays)
        sample = torch.arange(rays, device="cuda").repeat(min(b + 1024, n) - b)
        xy = torch.zeros(item.numel(), 2, dtype=torch.float64, device="cuda")
        todo = torch.arange(item.numel(), device="cuda")
        for a in range(64):
            r = _philox(item[todo], sample[todo], torch.full_like(todo, a), torch.full_like(todo, 6), seed)
            d = torch.stack(r[:2], 1) * 2 - 1
            ok = (d.float() ** 2).sum(1) <= 1
            xy[todo[ok]] = d[ok]
            todo = todo[~ok]
            if todo.numel() == 0:
                break
        z = (1 - (xy ** 2).sum(1)).clamp_min(0).sqrt()
        N = nrm[item]
        sign = torch.where(N[:, 2] >= 0, 1.0, -1.0).double()
        a = -1 / (sign + N[:, 2])
        c = N[:, 0] * N[:, 1] * a
        b1 = torch.stack([1 + sign * N[:, 0] ** 2 * a, sign * c, -sign * N[:, 0]], 1)
        b2 = torch.stack([c, sign + N[:, 1] ** 2 * a, -N[:, 1]], 1)
        d = b1 * xy[:, :1] + b2 * xy[:, 1:] + N * z[:, None]
        P = pos[item]
        t = torch.where(d > 0, (dims - P) / d, torch.where(d < 0, -P / d, torch.full_like(d, math.inf)))
        t = torch.where(N != 0, torch.where((N * d) > 0, dims / d.abs(), torch.full_like(d, math.inf)), t)
        best, axis = t.min(1)
        hit = P + d * best[:, None]
        texel = torch.full_like(item, -1)
        for (ax, side), (x0, y0, x1, y1, au, av) in charts.items():
            m = (axis == ax) & ((d.gather(1, axis[:, None])[:, 0] > 0) == bool(side)) & (best > 0.01)
            u, v = hit[m, au] / dims[au], hit[m, av] / dims[av]
            # a hit's uv takes the weights of its triangle's second and third vertices the other way round
            u, v = torch.where(u >= v, u, v - u), torch.where(u >= v, u - v, v)
            u, v = (x0 + u * (x1 - x0)) / s, (y0 + v * (y1 - y0)) / s
            texel[m] = (v * (s - 1)).long().clamp(0, s - 1) * s + (u * (s - 1)).long().clamp(0, s - 1)
        ok = texel >= 0
        F.view(-1).index_add_(0, item[ok] * n + texel[ok], torch.full((int(ok.sum()),), 1.0 / rays, dtype=torch.float64, device="cuda"))
    E, rho = (torch.tensor(v, device="cuda").double() for v in _light(n, seed))
    B = E.clone()
    for _ in range(case["iters"]):
        B = E + rho * (F @ B)
    return [None, None, None, B]


# pairwise: which segments count as open is decided by rounding at their far ends, so there is no exact()

def _prepare_pairwise(case, seed):
    wl, rl, ds, valid, pos, nrm = _patches(case, seed)
    # patch positions jittered within their texels' rows: other patches for another seed
    g = torch.Generator(device="cuda").manual_seed(seed)
    pitch = 10.0 / (case["size"] // 2)
    jitter = (torch.rand(pos.shape, generator=g, device="cuda") - 0.5) * pitch * 0.5
    pos = (pos + jitter * (nrm == 0)).contiguous()
    n = len(valid)
    return {"kind": "pairwise", "keep": (wl, rl), "ds": ds, "n": n, "pos": pos, "nrm": nrm,
            "threshold": case["threshold"], "row": np.zeros(n + 1, np.int64), "cols": np.zeros(100 * n, np.int32),
            "vals": np.zeros(100 * n, np.float32), "stream": _stream()}


def _run_pairwise(s):
    # the count call, and the fill call into arrays that have room for it
    L, count = _abi.lib(), C.c_int64()
    a = (s["ds"].handle, s["n"], _p(s["pos"]), _p(s["nrm"]), s["threshold"])
    _abi.check(L.rl_ff_pairwise(*a, None, None, None, 0, C.byref(count), s["stream"]))
    if count.value > s["cols"].size:
        raise RuntimeError("form factors: %d do not fit" % count.value)
    _abi.check(L.rl_ff_pairwise(*a, _p(s["row"]), _p(s["cols"]), _p(s["vals"]), count.value, C.byref(count),
                                s["stream"]))
    return [s["row"], s["cols"], s["vals"]]


def _work_pairwise(case):
    n = case["size"] ** 2
    return {"bytes": 24.0 * n + 8.0 * 12 * n, "flops": n * (n - 1) / 2 * 25.0}


# rays: a brute-force answer in 64 bits would take a test of every ray against every triangle, so there is no exact()

def _prepare_rays(case, seed):
    wl = _terrain(case, seed, 64)
    rl = Relight(stream=_stream(), seed=seed)
    ds = rl.device_scene(wl.scene)
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo, hi = (torch.tensor(np.asarray(v, np.float32), device="cuda") for v in (wl.scene.flat.bounds_lo, wl.scene.flat.bounds_hi))
    org = lo + (hi - lo) * torch.rand(n, 3, generator=g, device="cuda")
    org[:, 1] += 1.0
    d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
    rays = torch.cat([org, torch.full((n, 1), 0.01, device="cuda"), d, torch.full((n, 1), 400.0, device="cuda")], 1)
    return {"kind": "rays", "keep": (wl, rl), "ds": ds, "n": n, "rays": rays.contiguous(), "any": int(case["any_hit"]),
            "hit": torch.empty(n, 2, dtype=torch.int32, device="cuda"),
            "tuv": torch.empty(n, 3, dtype=torch.float32, device="cuda"), "stream": _stream()}


def _run_rays(s):
    _abi.check(_abi.lib().rl_intersect_rays(s["ds"].handle, s["n"], _p(s["rays"]), s["any"], _p(s["hit"]), _p(s["tuv"]),
                                            s["stream"]))
    # which triangle a first-hit query meets is free: only whether it meets one is an answer
    return s["hit"][:, 0] >= 0 if s["any"] else [s["hit"], s["tuv"]]


def _work_rays(case):
    tris = _tri_count(case)
    return {"bytes": 52.0 * case["rays"] + 48.0 * tris, "flops": case["rays"] * (24 * math.log2(tris) + 60)}


# denoise and train: the network of relight_b200.denoise.LAYERS

def _params(seed):
    """He-uniform weights in the denoiser's flat layout: per layer [cout][9][segments padded to 64], then the biases."""
    rng = np.random.default_rng(seed)
    out = []
    for layer, (cout, segs) in enumerate(denoise.LAYERS):
        real = [10] if layer == 0 else list(segs)
        lim = math.sqrt(6.0 / (9 * sum(real))) * (0.1 if layer == len(denoise.LAYERS) - 1 else 1.0)
        blocks = []
        for c, r in zip(segs, real):
            b = np.zeros((cout, 9, (c + 63) // 64 * 64), np.float32)
            b[:, :, :r] = rng.uniform(-lim, lim, (cout, 9, r))
            blocks.append(b)
        out += [np.concatenate(blocks, 2).reshape(-1), rng.uniform(-0.05, 0.05, cout).astype(np.float32)]
    return np.concatenate(out)


def _features(n, h, w, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.zeros(n, h, w, 16, device="cuda")
    x[..., :3] = torch.log1p(torch.rand(n, h, w, 3, generator=g, device="cuda") ** 2 * 2)
    x[..., 3:6] = torch.nn.functional.normalize(torch.randn(n, h, w, 3, generator=g, device="cuda"), dim=-1)
    x[..., 6:9] = 0.2 + 0.6 * torch.rand(n, h, w, 3, generator=g, device="cuda")
    x[..., 9] = (torch.rand(n, h, w, generator=g, device="cuda") < 0.9).float()
    return (x * x[..., 9:10]).to(torch.bfloat16).contiguous()


def _conv_flops(n, h, w):
    total = 0.0
    for (cout, segs), lv in zip(denoise.LAYERS, (0, 1, 2, 3, 2, 1, 0, 0)):
        total += 2.0 * n * math.ceil(h / 2 ** lv) * math.ceil(w / 2 ** lv) * cout * 9 * sum(segs)
    return total


def _prepare_denoise(case, seed):
    dn = Denoiser(seed=1)
    dn.set_params(_params(seed))
    dn.reserve(case["images"], case["height"], case["width"])
    return {"kind": "denoise", "dn": dn, "x": _features(case["images"], case["height"], case["width"], seed),
            "stream": _stream()}


def _run_denoise(s):
    return s["dn"].forward(s["x"], s["stream"])[..., :3]


def _work_denoise(case):
    px = case["images"] * case["height"] * case["width"]
    return {"bytes": 64.0 * px, "flops": _conv_flops(case["images"], case["height"], case["width"])}


def _net(x, flat):
    """The network in plain torch, in the type of its arguments: x [n][h][w][16] -> [n][h][w][3]."""
    F = torch.nn.functional
    layers, o = [], 0
    for cout, segs in denoise.LAYERS:
        k = sum((c + 63) // 64 * 64 for c in segs)
        w = flat[o:o + cout * 9 * k].reshape(cout, 3, 3, k).permute(0, 3, 1, 2)
        o += cout * 9 * k
        cut, at = [], 0
        for c in segs:
            cut.append(w[:, at:at + c])
            at += (c + 63) // 64 * 64
        layers.append((torch.cat(cut, 1), flat[o:o + cout]))
        o += cout

    def conv(i, t, act=True):
        w, b = layers[i]
        # rows of pixels as one matrix product per tap: 64-bit convolutions have no fast path of their own
        n, c, hh, ww = t.shape
        p = F.pad(t, (1, 1, 1, 1))
        y = b[:, None, None].expand(n, -1, hh, ww)
        for dy in range(3):
            for dx in range(3):
                y = y + torch.einsum("oc,nchw->nohw", w[:, :, dy, dx], p[:, :, dy:dy + hh, dx:dx + ww])
        return F.leaky_relu(y, 0.1) if act else y

    def pool(t):
        return F.avg_pool2d(t, 2, ceil_mode=True, count_include_pad=False)

    def up(t, like):
        return F.interpolate(t, scale_factor=2, mode="nearest")[:, :, :like.shape[2], :like.shape[3]]
    e0 = conv(0, x.permute(0, 3, 1, 2))
    e1 = conv(1, pool(e0))
    e2 = conv(2, pool(e1))
    e3 = conv(3, pool(e2))
    d2 = conv(4, torch.cat([up(e3, e2), e2], 1))
    d1 = conv(5, torch.cat([up(d2, e1), e1], 1))
    d0 = conv(6, torch.cat([up(d1, e0), e0], 1))
    return conv(7, d0, False).permute(0, 2, 3, 1)


def _exact_denoise(case, seed):
    with torch.no_grad():
        return _net(_features(case["images"], case["height"], case["width"], seed).double(),
                    torch.tensor(_params(seed), device="cuda").double())


def _pairs(case, seed):
    n, p = case["patches"], case["patch"]
    x = _features(n, p, p, seed)
    t = torch.zeros(n, p, p, 4, device="cuda")
    t[..., :3] = torch.nn.functional.avg_pool2d(x[..., :3].float().permute(0, 3, 1, 2), 5, 1, 2).permute(0, 2, 3, 1)
    t[..., 3] = x[..., 9].float()
    return x, t.contiguous()


def _prepare_train(case, seed):
    dn = Denoiser(seed=1)
    dn.set_params(_params(seed))
    dn.reserve(case["batch"], case["patch"], case["patch"], train=True)
    x, t = _pairs(case, seed)
    return {"kind": "train", "dn": dn, "x": x, "t": t, "steps": case["steps"], "batch": case["batch"],
            "stream": _stream()}


def _run_train(s):
    losses = denoise.train(s["dn"], s["x"], s["t"], s["steps"], batch=s["batch"], stream=s["stream"])
    return [losses, s["dn"].params()]


def _work_train(case):
    f = _conv_flops(case["batch"], case["patch"], case["patch"])
    px = case["batch"] * case["patch"] ** 2
    return {"bytes": case["steps"] * (48.0 * px + 24.0 * 630000), "flops": 3.0 * case["steps"] * f}


def _exact_train(case, seed):
    p = torch.tensor(_params(seed), device="cuda").double().requires_grad_(True)
    x, t = (v.double() for v in _pairs(case, seed))
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    g = torch.Generator(device="cuda").manual_seed(5)
    losses = []
    for s in range(case["steps"]):
        i = torch.randint(0, len(x), (case["batch"],), device="cuda", generator=g)
        d = _net(x[i], p) + x[i][..., :3] - t[i][..., :3]
        loss = (d.abs() * t[i][..., 3:4]).sum() / (d.numel())
        grad, = torch.autograd.grad(loss, p)
        losses.append(float(loss.detach()))
        lr = 2e-3 * 0.5 * (1 + math.cos(math.pi * s / case["steps"])) * min(1.0, (s + 1) / 200)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad * grad
            p -= lr * (m / (1 - 0.9 ** (s + 1))) / ((v / (1 - 0.999 ** (s + 1))).sqrt() + 1e-8)
    return [np.array(losses), p.detach()]


# post

def _post_inputs(case, seed):
    w, h = case["width"], case["height"]
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w]
    flags = ((x % 29 > 0) & (y % 23 > 0) & (rng.random((h, w)) < 0.97)).astype(np.int32).reshape(-1)
    color = (np.exp(rng.normal(-1.0, 1.0, (h * w, 3))) * flags[:, None]).astype(np.float32)
    return flags, color


def _prepare_post(case, seed):
    flags, color = _post_inputs(case, seed)
    lm = DeviceMap(0, case["width"], case["height"])
    lm.upload(stream=_stream(), flags=flags, color=color)
    return {"kind": "post", "lm": lm, "out": map_tensor(lm, "color"), "stream": _stream()}


def _run_post(s):
    s["lm"].expand(s["stream"])
    s["lm"].blur(s["stream"])
    return [s["out"], s["lm"].encode(RGBM, s["stream"])]


def _work_post(case):
    px = case["width"] * case["height"]
    return {"bytes": 32.0 * px, "flops": 40.0 * px}


def _exact_post(case, seed):
    w, h = case["width"], case["height"]
    flags, color = _post_inputs(case, seed)
    f = flags.reshape(h, w).astype(bool)
    c = color.astype(np.float64).reshape(h, w, 3)
    done = np.zeros((h, w), bool)
    for dy, dx in ((1, 1), (1, -1), (-1, 1), (-1, -1)):  # a texel without a lumel takes the last diagonal writer's colour
        ys, xs = np.mgrid[max(0, 1 - dy):min(h, h - 1 - dy), max(0, 1 - dx):min(w, w - 1 - dx)]
        take = ~f[ys, xs] & ~done[ys, xs] & f[ys + dy, xs + dx]
        c[ys[take], xs[take]] = c[ys[take] + dy, xs[take] + dx]
        done[ys[take], xs[take]] = True
    for t in range((w - 3) + 2 * (h - 3) + 1):  # texels of one t read only texels of smaller ones
        y = np.arange(max(1, 1 + (t - (w - 3) + 1) // 2), min(h - 2, 1 + t // 2) + 1)
        x = t - 2 * (y - 1) + 1
        total, count = np.zeros((len(y), 3)), np.zeros(len(y))
        for j in (-1, 0, 1):
            for i in (-1, 0, 1):
                on = f[y + j, x + i]
                total += np.where(on[:, None], c[y + j, x + i], 0.0)
                count += on
        on = count > 0
        c[y[on], x[on]] = total[on] / count[on, None]
    return [c.reshape(-1, 3), None]
