"""The work that users of this library have it do, as cases that can be timed.

Kinds of case:
  scan     an empty volume takes the frames of a scan one after another; then every block is exported in the
           reference record and put in the order of the keys, as a checkpoint keeps them
  walk     the next frames of a long walk into a volume that keeps growing (no reset between passes), then a
           small ray-cast preview of what has been fused
  batch    several independent scans fused together, one step per frame, each then exported as above
  mesh     marching cubes of a fused volume: the whole triangle soup, or the indexed mesh of the blocks that the
           last frame updated, into the program's buffers on the device
  raycast  the depth of the fused surface at the poses it was fused from (the denoiser's training targets)
  filter   the depth filter and the per-pixel normals of one frame on their own
  denoise  the learned depth denoiser's forward pass
  train    one training step of the denoiser

Forms: "plain" is the bit-reproducible default; "opt" is the opt-in form (truncation-band allocation, normal map,
fast math, FP16 bins).  Scenes are the library's own (orbit, object scan, room, multi-room), at any resolution.
Buffers that a call fills are the program's own, made once, of a size that any scene of the case fits.
"""
import ctypes as C
import math

import numpy as np
import torch

from voxelhashmt_gb300 import _capi, backend, denoiser, scenes

# mean depth (m) and focal length over width of each scene: the surface that a frame covers
_VIEW = {"orbit": (1.6, 0.866), "object": (2.0, 0.866), "room": (2.0, 0.82), "rooms": (3.5, 0.82)}


def listed():
    return [
        # the smallest call: one low-resolution frame filtered
        {"name": "filter_160", "kind": "filter", "form": "plain", "width": 160, "height": 120},
        # the small orbit configuration in the default form, depth from pageable host arrays
        {"name": "scan_orbit_320_plain", "kind": "scan", "scene": "orbit", "form": "plain", "width": 320,
         "height": 240, "frames": 15, "voxel_mm": 10.0, "stride": 1, "depth": "host"},
        # the room configuration in the default form
        {"name": "scan_room_640_plain", "kind": "scan", "scene": "room", "form": "plain", "width": 640,
         "height": 480, "frames": 7, "voxel_mm": 5.0, "stride": 1, "depth": "device"},
        # a low-resolution object scan in the opt-in form, page-locked host depth: frames of tens of microseconds
        {"name": "scan_object_160_opt", "kind": "scan", "scene": "object", "form": "opt", "width": 160,
         "height": 120, "frames": 47, "voxel_mm": 8.0, "stride": 1, "depth": "pinned"},
        # the room configuration in the opt-in form, from page-locked host depth as a camera driver gives it
        {"name": "scan_room_640_opt", "kind": "scan", "scene": "room", "form": "opt", "width": 640, "height": 480,
         "frames": 47, "voxel_mm": 5.0, "stride": 1, "depth": "pinned"},
        # the streaming configuration: 1280x720 at 3 mm, the next frames of the walk
        {"name": "walk_rooms_1280_opt", "kind": "walk", "scene": "rooms", "form": "opt", "width": 1280,
         "height": 720, "frames": 14, "voxel_mm": 3.0, "stride": 1, "depth": "device"},
        # object scans of mixed resolution fused as one batch
        {"name": "batch_objects_opt", "kind": "batch", "scenes": 8, "form": "opt", "width": 640, "height": 480,
         "frames": 37, "voxel_mm": 5.0, "stride": 1},
        # the final mesh of a room in the default form
        {"name": "mesh_room_plain", "kind": "mesh", "scene": "room", "form": "plain", "width": 640, "height": 480,
         "frames": 6, "voxel_mm": 5.0, "recent": False},
        # the incremental mesh of an orbit in the opt-in form, indexed, for a viewer
        {"name": "mesh_orbit_recent", "kind": "mesh", "scene": "orbit", "form": "opt", "width": 320, "height": 240,
         "frames": 9, "voxel_mm": 10.0, "recent": True},
        # training targets of the denoiser: the fused room seen again from two of its poses
        {"name": "raycast_room_640", "kind": "raycast", "scene": "room", "form": "plain", "width": 640,
         "height": 480, "frames": 6, "voxel_mm": 5.0, "views": 2},
        # the denoiser on one camera frame
        {"name": "denoise_640", "kind": "denoise", "batch": 1, "width": 640, "height": 480},
        # the denoiser's training step of the learned-filter configuration
        {"name": "train_640_b16", "kind": "train", "batch": 16, "width": 640, "height": 480},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    w = _log_int(rng, lo, hi)
    return w, max(16, int(round(w * rng.choice([0.75, 0.75, 0.5625, 0.7]))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "scan", "scan", "walk", "batch", "mesh", "mesh", "raycast", "filter",
                       "denoise", "train"])
    form = rng.choice(["plain", "opt"])
    stride = rng.choice([1, 1, 1, 2, 3])
    if kind == "scan":
        scene = rng.choice(["object", "orbit", "room"])
        w, h = _size(rng, 96, 640)
        voxel = {"object": rng.uniform(5.0, 8.0), "orbit": rng.uniform(8.0, 20.0), "room": rng.uniform(5.0, 10.0)}[scene]
        return {"kind": kind, "scene": scene, "form": form, "width": w, "height": h,
                "frames": rng.randint(2, 7) if form == "plain" else rng.randint(7, 47),
                "voxel_mm": round(voxel, 3), "stride": stride, "depth": rng.choice(["device", "host", "pinned"])}
    if kind == "walk":
        w, h = _size(rng, 320, 1280)
        return {"kind": kind, "scene": "rooms", "form": "opt", "width": w, "height": min(h, 720),
                "frames": rng.randint(2, 14), "voxel_mm": round(rng.uniform(3.0, 6.0), 3), "stride": stride,
                "depth": rng.choice(["device", "pinned"])}
    if kind == "batch":
        w, h = _size(rng, 160, 640)
        return {"kind": kind, "scenes": _log_int(rng, 2, 8), "form": "opt", "width": w, "height": h,
                "frames": rng.randint(5, 37), "voxel_mm": round(rng.uniform(5.0, 8.0), 3), "stride": 1}
    if kind in ("mesh", "raycast"):
        scene = rng.choice(["object", "orbit", "room"])
        w, h = _size(rng, 120, 480)
        case = {"kind": kind, "scene": scene, "form": form, "width": w, "height": h, "frames": rng.randint(2, 6),
                "voxel_mm": round({"object": rng.uniform(5.0, 8.0), "orbit": rng.uniform(10.0, 20.0),
                                   "room": rng.uniform(6.0, 10.0)}[scene], 3)}
        case.update({"views": rng.randint(1, 2)} if kind == "raycast" else {"recent": rng.random() < 0.4})
        return case
    if kind == "filter":
        w, h = _size(rng, 96, 1280)
        return {"kind": kind, "form": form, "width": w, "height": min(h, 720)}
    w, h = _size(rng, 96, 640)
    return {"kind": kind, "batch": _log_int(rng, 1, 16), "width": w, "height": h}


# ---- scenes ----

def _scene(name, seed, w, h, frames, voxel_mm):
    """`frames` consecutive frames of the named scene at w x h (the scene's own field of view)."""
    if name == "orbit":
        f = 277.0 * w / 320
        sc = scenes.orbit_scene(seed, frames=64, width=w, height=h, fx=f, fy=f, cx=w / 2, cy=h / 2)
        first = seed % 48
    elif name == "object":
        sc = scenes.object_scan_scene(seed, frames=120, resolution=(w, h), voxel_size=voxel_mm * 1e-3)
        first = seed % 100
    else:
        f = 525.0 * w / 640
        if name == "room":
            sc = scenes.room_scene(seed, frames=64, width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2, cy=(h - 1) / 2)
            first = seed % 16
        else:
            sc = scenes.multi_room_scene(seed, frames=6000, width=w, height=h, fx=f, fy=f, cx=(w - 1) / 2,
                                         cy=(h - 1) / 2)
            first = seed % 5900
    sc.voxel_size = voxel_mm * 1e-3
    sc.truncation = 4.0 * sc.voxel_size
    sc.poses = (sc.poses + sc.poses)[first:first + frames]
    return sc


def _volume(form, sc, max_blocks, buckets=None):
    kw = {"hash_buckets": buckets or max(sc.hash_buckets, 1 << 18), "max_blocks": max_blocks}
    if form == "opt":
        kw.update(layer_format=1, algorithm=_capi.default_algorithm(allocation_mode=1, normal_mode=1, fast_math=1))
    return backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, **kw)


def _pool(case):
    """Blocks to make room for, about twice what the frames touch."""
    scene = case.get("scene", "object")
    z, f = _VIEW[scene]
    area = (z / f) ** 2 * case["height"] / case["width"]  # m^2 seen at the mean depth, facing the camera
    per_area = 6.0 / (8e-3 * case["voxel_mm"]) ** 2  # blocks per m^2 across the band
    ample = {"orbit": 14, "object": 4, "room": 4, "rooms": 5} if case["form"] == "plain" else \
            {"orbit": 8, "object": 1.2, "room": 3, "rooms": 5}
    return int(max(8_000, ample[scene] * area * per_area))


def _depths(case, frames):
    """The frames as the program has them: device tensors, or host arrays (pageable or page-locked)."""
    if case["depth"] == "device":
        return [frames[i].view(-1) for i in range(frames.shape[0])], None
    host = frames.cpu()
    if case["depth"] == "pinned":
        host = host.pin_memory()
    return [host[i].view(-1).numpy() for i in range(host.shape[0])], host


def _ptr(t, kind=None):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(kind)) if kind else C.c_void_p(t.data_ptr())


def _import(vol, keys, voxels):
    _capi.check(_capi.lib().vh_import_blocks(vol.handle, _ptr(keys, C.c_int32), _ptr(voxels), keys.shape[0], 1, None),
                vol.handle)


def _block_buffers(rows):
    """(keys, voxel words) as the export gives them, and again for their ordered copy."""
    return [torch.zeros((rows, n), dtype=torch.int32, device="cuda") for n in (3, 512 * 6 * 3 * 4) * 2]


def _blocks(vol, buffers):
    """Every block of a volume into the buffers' ordered copy, by key; the rows beyond the block count stay 0."""
    keys, vox, okeys, ovox = buffers
    n = vol.block_count()
    _capi.check(_capi.lib().vh_export_blocks(vol.handle, 0, n, _ptr(keys, C.c_int32), _ptr(vox), 1, None), vol.handle)
    k = keys[:n].long() + (1 << 20)
    order = torch.argsort((k[:, 2] << 42) | (k[:, 1] << 21) | k[:, 0])
    torch.index_select(keys[:n], 0, order, out=okeys[:n])
    torch.index_select(vox[:n], 0, order, out=ovox[:n])
    return n, okeys, ovox


def _fused(case, seed):
    """The case's scene, its frames and a volume that they are fused in."""
    sc = _scene(case["scene"], seed, case["width"], case["height"], case["frames"], case["voxel_mm"])
    frames = denoiser.render_frames(sc, torch)
    vol = _volume(case["form"], sc, _pool(case))
    for i, pose in enumerate(sc.poses):
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, frames[i].view(-1)), pose,
                                           synchronize=False)
    vol.synchronize()
    return sc, frames, vol


def _ordered(case, sc, src):
    """A volume with the blocks of src in the order of their keys, loaded a few at a time (the order of a mesh's
    triangles follows the order of the blocks)."""
    n, keys, vox = _blocks(src, _block_buffers(src.block_count()))
    src.close()
    vol = _volume(case["form"], sc, n + 1024, buckets=1 << 22)
    for i in range(0, n, 32):
        _import(vol, keys[i:i + 32], vox[i:i + 32])
    return vol


# ---- the cases ----

def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("scan", "walk"):
        n = case["frames"] * (2 if kind == "walk" else 1)
        sc = _scene(case["scene"], seed, case["width"], case["height"], n, case["voxel_mm"])
        frames = denoiser.render_frames(sc, torch)
        st["K"], st["poses"] = sc.intrinsics, sc.poses
        st["depth"], st["keep"] = _depths(case, frames)
        st["vol"] = _volume(case["form"], sc, _pool(case))
        st["backend"] = backend.TsdfIntegrationBackend("gpu")
        if kind == "scan":
            st["buffers"] = _block_buffers(_pool(case))
        else:
            K, st["at"], st["max_depth"] = sc.intrinsics, 0, sc.max_depth
            st["preview"] = scenes.Intrinsics(max(16, K.width // 4), max(12, K.height // 4), K.fx / 4, K.fy / 4,
                                              K.cx / 4, K.cy / 4)
    elif kind == "batch":
        st.update(vols=[], K=[], poses=[], depth=[], buffers=[])
        for i in range(case["scenes"]):
            s = 4 >> (i % 3)  # full, half and quarter resolution
            w, h = max(32, case["width"] * s // 4), max(24, case["height"] * s // 4)
            sc = _scene("object", seed * 64 + i, w, h, case["frames"], case["voxel_mm"])
            st["vols"].append(_volume("opt", sc, _pool(case)))
            st["K"].append(sc.intrinsics)
            st["poses"].append(sc.poses)
            st["depth"].append(denoiser.render_frames(sc, torch))
            st["buffers"].append(_block_buffers(max(8_000, _pool(case) * 2 // 3)))
        st["batch"] = backend.VolumeBatch(st["vols"])
    elif kind == "mesh":
        sc, frames, src = _fused(case, seed)
        vol = _ordered(case, sc, src)
        # the last frame seen once more: every block it touches is there already
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, frames[-1].view(-1)), sc.poses[-1])
        rows = _pool(case) * 60
        st["vol"] = vol
        if case["recent"]:
            st["vertices"] = torch.zeros((rows, 3), dtype=torch.float32, device="cuda")
            st["faces"] = torch.zeros((rows, 3), dtype=torch.int32, device="cuda")
        else:
            st["soup"] = torch.zeros((rows, 9), dtype=torch.float32, device="cuda")
    elif kind == "raycast":
        sc, _, st["vol"] = _fused(case, seed)
        st["K"], st["poses"], st["max_depth"] = sc.intrinsics, sc.poses[-case["views"]:], sc.max_depth
    elif kind == "filter":
        sc = _scene("room", seed, case["width"], case["height"], 1, 5.0)
        st["vol"] = backend.VoxelHashTSDF(0.005, 0.02, hash_buckets=1 << 10, max_blocks=0,
                                          algorithm=_capi.default_algorithm(fast_math=int(case["form"] == "opt")))
        st["in"] = denoiser.render_frames(sc, torch)[0]
        st["out"] = torch.empty_like(st["in"])
        st["normals"] = torch.empty((*st["in"].shape, 4), dtype=torch.float32, device="cuda")
        st["K"] = _capi.intrinsics(sc.intrinsics)
    else:
        raw, target, params = _denoiser_data(case, seed)
        st["net"], st["raw"], st["target"] = denoiser.DepthDenoiser(params), raw, target
    return st


def _denoiser_data(case, seed):
    """Noisy frames of a room walk, the noise-free ones, and parameters (near identity, as training starts)."""
    sc = _scene("room", seed, case["width"], case["height"], case["batch"], 5.0)
    raw = denoiser.render_frames(sc, torch)
    sc.noise_sigma_z2, sc.dropout = 0.0, 0.0
    return raw, denoiser.render_frames(sc, torch), denoiser.init_params(seed)


def _fuse(st, first, count):
    for i in range(first, first + count):
        st["backend"].integrate(st["vol"], backend.DepthFrame(st["K"], st["depth"][i]), st["poses"][i],
                                st["case"]["stride"], synchronize=i + 1 == first + count)


def run(st):
    case = st["case"]
    kind, lib = case["kind"], _capi.lib()
    if kind == "scan":
        st["vol"].reset()
        _fuse(st, 0, case["frames"])
        return _blocks(st["vol"], st["buffers"])
    if kind == "walk":
        n, first = case["frames"], st["at"]
        _fuse(st, first, n)
        st["at"] = n - first
        return backend.raycast_depth(st["vol"], st["preview"], st["poses"][first + n - 1], 0.1, st["max_depth"],
                                     device_out="cuda")
    if kind == "batch":
        for v in st["vols"]:
            v.reset()
        for f in range(case["frames"]):
            st["batch"].integrate([d[f] for d in st["depth"]], st["K"], [p[f] for p in st["poses"]], case["stride"])
        for v in st["vols"]:
            v.synchronize()
        return [_blocks(v, b) for v, b in zip(st["vols"], st["buffers"])]
    if kind == "mesh":
        h, nt, nv, nf = st["vol"].handle, C.c_size_t(), C.c_size_t(), C.c_size_t()
        if case["recent"]:
            _capi.check(lib.vh_extract_mesh_recent(h, 0.0, 1, C.byref(nt), None), h)
            _capi.check(lib.vh_weld_mesh(h, C.byref(nv), C.byref(nf), None), h)
            rows = st["vertices"].shape[0]
            _capi.check(lib.vh_copy_welded_mesh(h, _ptr(st["vertices"]), rows, _ptr(st["faces"]), rows, 1, None), h)
            return nv.value, nf.value, st["vertices"], st["faces"]
        _capi.check(lib.vh_extract_mesh(h, 0.0, C.byref(nt), None), h)
        _capi.check(lib.vh_copy_mesh(h, _ptr(st["soup"]), st["soup"].shape[0], 1, None), h)
        return nt.value, st["soup"]
    if kind == "raycast":
        return [backend.raycast_depth(st["vol"], st["K"], p, 0.1, st["max_depth"], device_out="cuda")
                for p in st["poses"]]
    if kind == "filter":
        h, K = st["vol"].handle, C.byref(st["K"])
        _capi.check(lib.vh_filter_depth(h, _ptr(st["in"]), _ptr(st["out"]), K, None), h)
        _capi.check(lib.vh_pixel_normals(h, _ptr(st["out"]), _ptr(st["normals"]), K, None), h)
        return st["out"], st["normals"]
    if kind == "denoise":
        return st["net"].forward(st["raw"])
    rmse = st["net"].train_step(st["raw"], st["target"])
    return rmse, st["net"].grads, st["net"].params


def work(case):
    kind = case["kind"]
    px = case["width"] * case["height"]
    if kind in ("denoise", "train"):
        n = px * case["batch"]
        layers = 2 * 9 * (4 * 32 + 2 * 32 * 32 + 32)  # products and sums of a pixel
        if kind == "denoise":
            return {"bytes": 8 * n, "flops": layers * n}
        p = denoiser.init_params(0).size
        return {"bytes": 8 * n + 9 * 4 * p, "flops": 3 * layers * n}
    if kind == "filter":
        return {"bytes": px * (4 + 4 + 16), "flops": px * (25 * 40 + 500)}
    # voxels across the truncation band (8 voxels) of the surface that a frame sees
    z, f = _VIEW[case.get("scene", "object")]
    bin_bytes = 48 if case["form"] == "plain" else 32
    voxels = 8.0 * px * (z / (f * case["width"]) / (case["voxel_mm"] * 1e-3)) ** 2
    if case.get("scene", "object") == "object":
        voxels *= 0.35  # the rest of the view is empty
    blocks = voxels / 60.0  # about this many of a block's 512 voxels lie in the band
    if kind in ("scan", "walk", "batch"):
        saved = 2 * 512 * 6 * 48 * blocks  # the exported blocks, put in order
        if kind == "batch":  # a third of the scenes each at full, half and quarter resolution
            px, voxels = px * (1 + 1 / 4 + 1 / 16) / 3 * case["scenes"], voxels * case["scenes"]
            saved *= case["scenes"]
        per_voxel = 1500 if case["form"] == "plain" else 250
        return {"bytes": case["frames"] * (4 * px + 2 * bin_bytes * voxels) + (saved if kind != "walk" else px / 4),
                "flops": case["frames"] * (per_voxel * voxels + 1500 * px)}
    if kind == "raycast":  # the observed bins along the rays up to the surface, once
        return {"bytes": case["views"] * (4 * px + bin_bytes * voxels / 2), "flops": case["views"] * px * 40 * 8 * 30}
    if case["recent"]:
        return {"bytes": blocks * (2 * bin_bytes * 512 + 40 * 24), "flops": blocks * 512 * 600}
    return {"bytes": blocks * (2 * bin_bytes * 512 + 40 * 36), "flops": blocks * 512 * 600}


# ---- the same results in 64 bits ----

def exact(case, seed):
    kind = case["kind"]
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind in ("denoise", "train"):
        return _exact_net(case, seed)
    return None  # a fused volume is a long chain of decisions: no closed form


def _shift(a, dx, dy):
    """a at (x + dx, y + dy), 0 outside."""
    h, w = a.shape[:2]
    out = torch.zeros_like(a)
    ys, xs = slice(max(0, -dy), min(h, h - dy)), slice(max(0, -dx), min(w, w - dx))
    out[ys, xs] = a[max(0, dy):max(0, dy) + out[ys, xs].shape[0], max(0, dx):max(0, dx) + out[ys, xs].shape[1]]
    return out


def _unit(v):
    n = v.norm(dim=-1, keepdim=True)
    return torch.where(n > 1e-6, v / n.clamp_min(1e-300), torch.zeros_like(v))


def _facing(n, p):
    return torch.where((n * p).sum(-1, keepdim=True) > 0, -n, n)


def _exact_filter(case, seed):
    sc = _scene("room", seed, case["width"], case["height"], 1, 5.0)
    K = sc.intrinsics
    al = _capi.default_algorithm()
    d = denoiser.render_frames(sc, torch)[0].double()
    h, w = d.shape
    v, u = torch.meshgrid(torch.arange(h, device="cuda", dtype=torch.float64),
                          torch.arange(w, device="cuda", dtype=torch.float64), indexing="ij")

    def points(z):
        return torch.stack([(u - K.cx) * z / K.fx, (v - K.cy) * z / K.fy, z], -1)

    def base_normals(z):
        p = points(z)
        ok = z > 0
        for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1)):
            ok = ok & (_shift(z, dx, dy) > 0)
        n = _unit(torch.linalg.cross(_shift(p, 0, 1) - _shift(p, 0, -1), _shift(p, 1, 0) - _shift(p, -1, 0)))
        ok = ok & (n.norm(dim=-1) > 1e-6)
        return _facing(n, p) * ok[..., None], ok

    # the joint bilateral filter
    thr = (al.depth_discontinuity_relative * d.clamp_min(0)).clamp_min(al.depth_discontinuity_base)
    n, ok = base_normals(d)
    for dx, dy in ((-1, 0), (1, 0), (0, -1), (0, 1)):
        ok = ok & ((_shift(d, dx, dy) - d).abs() <= thr)
    n = n * ok[..., None]
    num, den = torch.zeros_like(d), torch.zeros_like(d)
    for dy in range(-2, 3):
        for dx in range(-2, 3):
            s, sn, sok = _shift(d, dx, dy), _shift(n, dx, dy), _shift(ok.double(), dx, dy) > 0
            cos = (n * sn).sum(-1).clamp(-1, 1)
            wt = torch.exp(-(dx * dx + dy * dy) / (2 * al.filter_sigma_spatial ** 2)
                           - (s - d) ** 2 / (2 * al.filter_sigma_range ** 2))
            wa = torch.exp(-(1 - cos) ** 2 / (2 * al.filter_sigma_angular ** 2))
            take = (s > 0) & ((s - d).abs() <= thr) & (~ok | (sok & (cos >= al.filter_min_cosine)))
            wt = torch.where(ok, wt * wa, wt) * take
            num, den = num + wt * s, den + wt
    out = torch.where(d > 0, torch.where(den > 1e-6, num / den.clamp_min(1e-300), d), torch.zeros_like(d))
    # the normal map of the filtered depth
    n, ok = base_normals(out)
    p = points(out)
    acc, ws = torch.zeros_like(n), torch.zeros_like(out)
    for dy in range(-1, 2):
        for dx in range(-1, 2):
            sn, sok = _shift(n, dx, dy), _shift(ok.double(), dx, dy) > 0
            cos = (n * sn).sum(-1).clamp(-1, 1)
            wt = torch.exp(-(dx * dx + dy * dy) / (2 * al.normal_sigma_spatial ** 2)
                           - (_shift(out, dx, dy) - out) ** 2 / (2 * al.normal_sigma_range ** 2)
                           - (1 - cos) ** 2 / (2 * al.normal_sigma_angular ** 2)) * sok
            acc, ws = acc + sn * wt[..., None], ws + wt
    m = _facing(_unit(acc / ws.clamp_min(1e-300)[..., None]), p)
    m = torch.where((ws > 1e-6)[..., None] & (m.norm(dim=-1, keepdim=True) > 1e-6), m, n) * ok[..., None]
    return out, torch.cat([m, ok.double()[..., None]], -1)


def _exact_net(case, seed):
    raw, target, params = _denoiser_data(case, seed)
    b, h, w = raw.shape
    if case["kind"] == "train" and b * h * w > 8_000_000:
        return None
    p = torch.from_numpy(params).cuda().double().requires_grad_()
    cut, at = [], 0
    for shape in ((32, 4, 3, 3), (32,), (32, 32, 3, 3), (32,), (32, 32, 3, 3), (32,), (1, 32, 3, 3), (1,)):
        size = int(np.prod(shape))
        cut.append((at, shape))
        at += size
    grads, outs = torch.zeros_like(p), []
    se, count = 0.0, 0.0
    for i in range(b):  # one image at a time: the activations are large in 64 bits
        ws = [p[a:a + int(np.prod(s))].view(s) for a, s in cut]
        d = raw[i].double()
        valid = d > 0
        pad = torch.nn.functional.pad(torch.stack([d * valid, valid.double()])[None], (1, 1, 1, 1))
        ssum, scnt = torch.nn.functional.avg_pool2d(pad, 3, 1)[0] * 9
        m = torch.where(scnt > 0.5, ssum / scnt.clamp_min(1.0), torch.zeros_like(d))
        x = torch.stack([(d - m) * 100, valid.double(), m / 4, torch.zeros_like(d)])[None] * valid
        with torch.set_grad_enabled(case["kind"] == "train"):
            for k in range(4):
                cols = torch.nn.functional.unfold(x, 3, padding=1)
                x = ((ws[2 * k].reshape(ws[2 * k].shape[0], -1) @ cols[0]) + ws[2 * k + 1][:, None]).view(1, -1, h, w)
                x = torch.relu(x) if k < 3 else x
            out = torch.where(valid, (d + x[0, 0] / 100).clamp_min(0.0), torch.zeros_like(d))
        outs.append(out.detach())
        if case["kind"] == "train":
            t = target[i].double()
            ok = valid & (t > 0) & (out > 0) & ((d - t).abs() <= (0.025 * t).clamp_min(0.012))
            loss = ((out - t) ** 2 * ok).sum()
            # the residual's gradient passes the clamp at 0 wherever the pixel counts
            (g,) = torch.autograd.grad(loss / (b * h * w), p)
            grads += g
            se, count = se + loss.item(), count + ok.sum().item()
    if case["kind"] == "denoise":
        return torch.stack(outs)
    m, v = 0.1 * grads, 0.001 * grads ** 2
    step = 1e-3 * (m / (1 - 0.9)) / ((v / (1 - 0.999)).sqrt() + 1e-8)
    return math.sqrt(se / max(count, 1.0)), grads.detach(), (p - step).detach()
