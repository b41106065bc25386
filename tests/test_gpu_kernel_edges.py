"""Kernels at the sizes where their tiles and groups can go wrong: remainders, single elements, both storage forms.
Bit-identical to the oracle's restatement (or to the general path) unless a tolerance is derived beside the test."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(product_lib, oracle_lib):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from voxelhashmt_gb300 import backend
    return backend, oracle_lib


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _fuse(backend, O, sc, frames, fp16):
    """The scene's frames in the library (exact compile) and in the oracle, with FP32 or FP16 bins."""
    from voxelhashmt_gb300 import _capi, scenes
    switches = {"alloc_mode": fp16, "normal_mode": fp16}
    vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 16, max_blocks=8192, layer_format=fp16,
                                algorithm=_capi.default_algorithm(allocation_mode=fp16, normal_mode=fp16))
    ora = O.Volume(O.config(O.FLAVOR_REF_GPU, O.EXP_OWN, threads=8, layer_format=fp16, **switches), sc.voxel_size,
                   sc.truncation)
    for f in frames:
        d = scenes.render_depth(sc, f)
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, d), sc.poses[f])
        ora.integrate(d, sc.intrinsics, sc.poses[f])
    return vol, ora


@pytest.mark.parametrize("fp16", [0, 1])
@pytest.mark.parametrize("size,step", [((1, 1), 0.5), ((7, 3), 0.5), ((33, 21), 0.25), ((70, 37), 1.7)])
def test_raycast_remainder_tiles_bit_exact(env, small_orbit, fp16, size, step):
    """Images smaller than a CTA's 8x4 pixels and with remainders in both axes, at several step lengths, from inside
    and outside the scene, against the oracle's ray-cast."""
    backend, O = env
    from voxelhashmt_gb300 import scenes
    sc = small_orbit
    vol, ora = _fuse(backend, O, sc, [0, 4, 8, 12], fp16)
    w, h = size
    K = scenes.Intrinsics(w, h, 55.4 * w / 64, 55.4 * w / 64, (w - 1) / 2.0, (h - 1) / 2.0)
    inside = scenes.look_at((0.05, 0.0, 0.4), (0.3, 0.2, 0.1))
    for pose in (sc.poses[2], sc.poses[17], inside):
        got = backend.raycast_depth(vol, K, pose, 0.0, 3.0, step)
        assert np.array_equal(_bits(got), _bits(ora.raycast_depth(K, pose, 0.0, 3.0, step)))
    vol.close()
    ora.close()


@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("fp16", [0, 1])
def test_export_to_device_equals_host(env, small_orbit, fp16, offset):
    """Blocks exported into device memory, directly (16-byte aligned) and through the staging buffer (4 bytes off), equal
    the host export word for word: the whole pool (over one staging pass), a range inside it, keys or voxels alone."""
    backend, O = env
    from voxelhashmt_gb300 import _capi
    vol, ora = _fuse(backend, O, small_orbit, [0, 5, 10, 15], fp16)
    n = vol.block_count()
    assert n > 1024 or fp16
    for first, count in ((0, n), (3, 1), (n - 77, 77)):
        hk, hv = vol.export_blocks(first, count)
        words = count * 512 * 6 * 3 * 4
        buf = torch.zeros(words + 4, dtype=torch.int32, device="cuda")
        keys = torch.zeros((count, 3), dtype=torch.int32, device="cuda")
        kp, vp = C.cast(C.c_void_p(keys.data_ptr()), C.POINTER(C.c_int32)), C.c_void_p(buf.data_ptr() + offset)
        for k, v in ((kp, vp), (kp, None), (None, vp)):
            buf.zero_()
            keys.zero_()
            _capi.check(_capi.lib().vh_export_blocks(vol.handle, first, count, k, v, 1, None), vol.handle)
            got = buf[offset // 4:offset // 4 + words].cpu().numpy().view(np.uint32)
            assert np.array_equal(got, hv.reshape(-1) if v else np.zeros_like(got))
            assert np.array_equal(keys.cpu().numpy(), hk if k else np.zeros_like(hk))
    gk, gv = O.sort_blocks(*vol.export_blocks())
    ok, ov = O.sort_blocks(*ora.blocks())
    assert np.array_equal(gk, ok)
    assert np.array_equal(gv.reshape(len(gk), -1), ov.view(np.uint32).reshape(len(ok), -1))
    vol.close()
    ora.close()


def _random_blocks(rng, keys, vs, fill):
    """Records (N, 512, 6, 3, 4) of random layers: a share `fill` of them observed, planes within 2 voxels of their
    voxel, normals in any direction."""
    n = len(keys)
    li = np.arange(512)
    local = np.stack([li & 7, (li >> 3) & 7, li >> 6], -1)
    centre = ((np.asarray(keys)[:, None, :] * 8 + local[None]) + 0.5) * vs  # (N, 512, 3)
    nrm = rng.normal(size=(n, 512, 6, 3, 3))
    nrm /= np.linalg.norm(nrm, axis=-1, keepdims=True)
    oct_ = nrm[..., :2] / np.abs(nrm).sum(-1, keepdims=True)
    sign = np.where(oct_ >= 0, 1.0, -1.0)
    oct_ = np.where(nrm[..., 2:] < 0, (1 - np.abs(oct_[..., ::-1])) * sign, oct_)
    q = np.floor((oct_ * 0.5 + 0.5) * 65535 + 0.5).astype(np.uint32)
    vox = np.zeros((n, 512, 6, 3, 4), np.float32)
    seen = rng.random((n, 512, 6, 3)) < fill
    offset = np.einsum("nvdlk,nvk->nvdl", nrm, centre) + rng.uniform(-2, 2, (n, 512, 6, 3)) * vs
    vox[..., 0] = np.where(seen, rng.uniform(0.1, 50.0, seen.shape), 0.0)
    vox[..., 1] = np.where(seen, centre[..., None, None, 0] + rng.uniform(-1, 1, seen.shape) * vs, 0.0)
    vox[..., 2] = np.where(seen, offset, 0.0)
    out = vox.view(np.uint32)
    out[..., 3] = np.where(seen, q[..., 0] | (q[..., 1] << 16), 0)
    return out


@pytest.mark.parametrize("fp16", [0, 1])
def test_export_and_reset_by_stored_directions(env, small_orbit, fp16):
    """Blocks with layers in no, one, several and all directions, and with a direction of records without weight alone (kept
    word for word by FP32 storage, empty in FP16): exported as they were imported; a reset leaves nothing of them."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    sc, vs = small_orbit, small_orbit.voxel_size
    rng = np.random.default_rng(11)
    keys = np.array([(x, y, 0) for y in range(40) for x in range(40)], np.int32)  # more than the clearing CTAs
    vox = _random_blocks(rng, keys, vs, 0.05)
    dirs = rng.integers(0, 64, len(keys))
    dirs[:3] = (0, 1, 63)
    vox[((dirs[:, None] >> np.arange(6)) & 1 == 0)[:, None, :].repeat(512, 1)] = 0
    stray = (dirs >> 3) & 1 == 0
    vox[stray, 7, 3, 1, 2] = 0x3f800000  # a plane offset without a weight
    vol, fresh = (backend.VoxelHashTSDF(vs, sc.truncation, hash_buckets=1 << 16, max_blocks=8192, layer_format=fp16)
                  for _ in range(2))
    vol.import_blocks(keys, vox)
    gk, gv = O.sort_blocks(*vol.export_blocks())
    want = vox.copy()
    if fp16:
        want[stray, 7, 3, 1, 2] = 0
    wk, wv = O.sort_blocks(keys, want)
    gv, wv = (np.ascontiguousarray(a).view(np.uint32).reshape(len(keys), 512, 6, 3, 4) for a in (gv, wv))
    assert np.array_equal(gk, wk)
    if fp16:  # rounded to binary16: the same records observed, the others empty
        seen = wv[..., 0] != 0
        assert np.array_equal(gv[..., 0] != 0, seen) and not gv[~seen].any()
    else:
        assert np.array_equal(gv, wv)
    vol.reset()
    for v in (vol, fresh):
        for f in (0, 5, 10):
            backend.integrate_depth_frame_cuda(v, backend.DepthFrame(sc.intrinsics, scenes.render_depth(sc, f)), sc.poses[f])
    (k1, v1), (k2, v2) = (O.sort_blocks(*v.export_blocks()) for v in (vol, fresh))
    assert len(k1) > 0 and np.array_equal(k1, k2) and np.array_equal(v1, v2)
    assert vol.observed_voxel_count() == fresh.observed_voxel_count() == vol.recount_observed_voxels()
    vol.close()
    fresh.close()


@pytest.mark.parametrize("fp16", [0, 1])
@pytest.mark.parametrize("fill,iso", [(0.02, 0.0), (0.35, 0.0), (0.9, 0.004)])
def test_mesh_of_random_layers(env, fp16, fill, iso):
    """Marching cubes of blocks of random planes against the oracle: from nearly empty blocks to every cell marked in
    every direction with up to 24 candidates, blocks alone and touching on faces, edges and corners, negative and large
    coordinates, an iso level off 0."""
    backend, O = env
    vs = 0.02
    keys = np.array([[x, y, z] for x in (-1, 0) for y in (-1, 0) for z in (-1, 0)] +
                    [[5, 5, 5], [6, 6, 6], [7, 6, 5], [-40, 3, 0], [300, -200, 100]], np.int32)
    vox = _random_blocks(np.random.default_rng(int(100 * fill)), keys, vs, fill)
    vol = backend.VoxelHashTSDF(vs, 4 * vs, hash_buckets=1 << 10, max_blocks=len(keys), layer_format=fp16)
    ora = O.Volume(O.config(O.FLAVOR_REF_GPU, O.EXP_OWN, threads=8, layer_format=fp16), vs, 4 * vs)
    vol.import_blocks(keys, vox)
    ora.apply_flat_blocks(keys, vox)
    tris = backend.extract_mesh_cuda(vol, iso)
    want = ora.extract_mesh(iso)
    assert tris.shape == want.shape and (fill < 0.1 or tris.shape[0] > 100)
    assert np.array_equal(_bits(O.canonical_triangles(tris)), _bits(O.canonical_triangles(want)))
    assert np.array_equal(_bits(backend.extract_mesh_cuda(vol, iso)), _bits(tris))  # the same order every time
    vol.close()
    ora.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 5, 33), (1, 17, 30), (1, 14, 61), (3, 16, 32), (1, 40, 100)])
def test_denoiser_layers_at_tile_edges(env, shape):
    """The denoiser's output and every gradient on images smaller than a tile, with remainders of the 32x16, 30x14 and
    32x8 tiles and pixels without depth, against float64 with BF16 rounding where the kernels store BF16.  Output:
    FP32 sums may round an activation to the other BF16 neighbour, 2^-8 of it, in each of the three layers; the bound
    carries that through the magnitudes of the weights (plus 1e-6 m of FP32 rounding).  Gradients: each parameter group
    within 2 % relative L2, as for the larger images of test_gpu_nn.py."""
    import torch.nn.functional as F
    from tests.test_gpu_nn import _ref_loss
    from voxelhashmt_gb300 import denoiser
    b, h, w = shape
    rng = np.random.default_rng(b * 100 + h * 10 + w)
    yy, xx = np.meshgrid(np.arange(h), np.arange(w), indexing="ij")
    clean = (1.5 + 0.01 * yy + 0.005 * xx)[None] + rng.uniform(0, 0.5, (b, 1, 1))
    raw = (clean + rng.normal(0, 0.003, (b, h, w))).astype(np.float32)
    if h * w > 1:
        raw[rng.random((b, h, w)) < 0.1] = 0.0
    p0 = denoiser.init_params(seed=5)
    p0[-289:] = rng.normal(0, 0.05, 289).astype(np.float32)
    net = denoiser.DepthDenoiser(p0)
    got, _, out = net.gradients(torch.from_numpy(raw).cuda(), torch.from_numpy(clean.astype(np.float32)).cuda())
    params = torch.from_numpy(p0.astype(np.float64)).requires_grad_(True)
    loss, want = _ref_loss(params, torch.from_numpy(raw).double(), torch.from_numpy(clean.astype(np.float32)).double())
    loss.backward()
    ref = params.grad.numpy()
    want = want.detach().numpy()
    # magnitudes of the activations and of what one rounding step per activation can move, layer by layer
    w1, b1, w2, b2, w3, b3, w4, _ = torch.split(params.detach().abs(), [1152, 32, 9216, 32, 9216, 32, 288, 1])
    d = torch.from_numpy(raw).double().unsqueeze(1)
    x = torch.cat([torch.full_like(d, 100 * 0.06), torch.ones_like(d), torch.ones_like(d), 0 * d], 1)  # bounds the channels
    mag, err = x, 0 * x
    for wt, bt, cin in ((w1, b1, 4), (w2, b2, 32), (w3, b3, 32)):
        wt = wt.view(32, cin, 3, 3)
        err = F.conv2d(err, wt, padding=1)
        mag = F.conv2d(mag, wt, bt, padding=1)
        err = err + 2.0 ** -8 * mag
    tol = (0.01 * F.conv2d(err, w4.view(1, 32, 3, 3), padding=1)).squeeze(1).numpy() + 1e-6
    assert np.all(np.abs(out.cpu().numpy().reshape(want.shape) - want) <= tol)
    off = 0
    for n in (32 * 4 * 9, 32, 32 * 32 * 9, 32, 32 * 32 * 9, 32, 32 * 9, 1):
        a, r = got[off:off + n].astype(np.float64), ref[off:off + n]
        assert np.linalg.norm(a - r) <= 2e-2 * np.linalg.norm(r) + 1e-12, (off, n)
        off += n


@pytest.mark.parametrize("form", ["plain", "chosen"])
@pytest.mark.parametrize("size", [(5, 3), (64, 48)])
def test_back_to_back_frames_equal_single_ones(env, small_orbit, form, size):
    """Frames enqueued without a wait between them, of two volumes on two streams, the one depth buffer rewritten on the
    stream between its frames and small enough that each kernel of a frame starts while the one before it runs: the same
    blocks, word for word, as with a wait after every frame."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    sc = small_orbit
    w, h = size
    K = scenes.Intrinsics(w, h, 55.4 * w / 64, 55.4 * w / 64, (w - 1) / 2.0, (h - 1) / 2.0)
    on = int(form == "chosen")
    algorithm = _capi.default_algorithm(allocation_mode=on, normal_mode=on, fast_math=on, autotune=0)
    rng = np.random.default_rng(5)
    depths = torch.from_numpy(np.stack([scenes.render_depth(sc, f)[:h, :w] for f in range(12)])).cuda()
    depths = depths + torch.from_numpy(rng.normal(0, 1e-3, tuple(depths.shape)).astype(np.float32)).cuda()

    def volume():
        return backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 16, max_blocks=8192, layer_format=on,
                                     algorithm=algorithm)

    single = volume()
    for f in range(12):
        backend.integrate_depth_frame_cuda(single, backend.DepthFrame(K, depths[f].contiguous()), sc.poses[f])
    want = O.sort_blocks(*single.export_blocks())
    torch.cuda.synchronize()
    vols, streams = [volume(), volume()], [torch.cuda.Stream(), torch.cuda.Stream()]
    bufs = [torch.zeros((h, w), device="cuda") for _ in vols]
    torch.cuda.synchronize()
    for f in range(12):
        for vol, st, buf in zip(vols, streams, bufs):
            with torch.cuda.stream(st):
                buf.copy_(depths[f])
            backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(K, buf), sc.poses[f], stream=st, synchronize=False)
    for vol, st in zip(vols, streams):
        vol.synchronize(st)
        got = O.sort_blocks(*vol.export_blocks())
        assert np.array_equal(got[0], want[0])
        assert np.array_equal(got[1], want[1])
        vol.close()
    single.close()


@pytest.mark.parametrize("radius", [0, 1, 2])
@pytest.mark.parametrize("size", [(1, 1), (3, 2), (8, 4), (9, 5), (31, 17), (729, 312), (737, 312)])
def test_filter_and_normals_of_small_and_large_tiles(env, radius, size):
    """The depth filter and the pixel normals with tiles of 8x4 pixels (up to 912 tiles of 32x8, as at 729x312: 23 by 39
    = 897) and of 32x8 (737x312: 24 by 39 = 936), with holes, steps, infinities, NaN and negative depth: word for word
    the oracle's."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    w, h = size
    rng = np.random.default_rng(w * 7 + h)
    depth = (1.0 + 0.2 * np.sin(np.arange(w) / 7.0)[None, :] + 0.01 * rng.normal(size=(h, w))).astype(np.float32)
    depth[rng.random((h, w)) < 0.05] = 0.0
    depth[rng.random((h, w)) < 0.05] += 0.3
    if w > 30:
        depth[5, 7], depth[6, 20], depth[9, 9] = np.inf, np.nan, -1.0
    K = scenes.Intrinsics(w, h, 500.0, 490.0, 20.0, 10.0)
    vol = backend.VoxelHashTSDF(0.01, 0.03, hash_buckets=1 << 10, max_blocks=64,
                                algorithm=_capi.default_algorithm(filter_radius=radius))
    finite = np.where(np.isinf(depth), np.float32(0.0), depth)  # a map's taps are pixels, the oracle's are blends of two
    src, fin = torch.from_numpy(depth).cuda(), torch.from_numpy(finite).cuda()
    out, nrm = torch.full_like(src, -7.0), torch.full((h, w, 4), -7.0, device="cuda")
    torch.cuda.synchronize()
    Ki = _capi.intrinsics(K)
    for fn, a, dst in ((_capi.lib().vh_filter_depth, src, out), (_capi.lib().vh_pixel_normals, fin, nrm)):
        _capi.check(fn(vol.handle, C.c_void_p(a.data_ptr()), C.c_void_p(dst.data_ptr()), C.byref(Ki), None), vol.handle)
    vol.synchronize()
    vol.close()
    cfg = O.config(O.FLAVOR_REF_GPU, O.EXP_OWN, threads=8, filter_radius=radius)
    assert np.array_equal(out.cpu().numpy(), O.filter_depth(cfg, depth, K), equal_nan=True)
    if radius == 2:
        want, ok = O.pixel_normals(cfg, finite, K)
        got = nrm.cpu().numpy()
        assert np.array_equal(got[..., 3], ok.astype(np.float32))
        assert np.array_equal(_bits(got[..., :3][ok != 0]), _bits(want[ok != 0]))


@pytest.mark.parametrize("form", ["plain", "chosen"])
@pytest.mark.parametrize("size,stride", [((1, 1), 1), ((7, 9), 1), ((33, 17), 2), ((300, 120), 1), ((304, 129), 1),
                                         ((97, 61), 3)])
def test_allocation_of_small_and_large_tiles(env, small_orbit, form, size, stride):
    """Frames whose filter and allocation run in tiles of 8x4 pixels (up to 152 tiles of 32x8: 300x120 is 10 by 15) and of
    32x8 (304x129 is 10 by 17): the oracle's blocks and layers, word for word, with both allocation rules; many
    blocks to a tile (a short focal length)."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    on = int(form == "chosen")
    w, h = size
    sc = scenes.orbit_scene(seed=7, frames=4, width=w, height=h, fx=0.4 * w, fy=0.4 * w, cx=w / 2.0, cy=h / 2.0)
    sc.voxel_size, sc.truncation = 0.02, 0.06
    vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 17, max_blocks=16384,
                                algorithm=_capi.default_algorithm(allocation_mode=on, normal_mode=on))
    ora = O.Volume(O.config(O.FLAVOR_REF_GPU, O.EXP_OWN, threads=8, alloc_mode=on, normal_mode=on), sc.voxel_size,
                   sc.truncation)
    for f in (0, 2):
        d = scenes.render_depth(sc, f)
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, d), sc.poses[f], stride)
        ora.integrate(d, sc.intrinsics, sc.poses[f], stride)
    gk, gv = O.sort_blocks(*vol.export_blocks())
    ok, ov = O.sort_blocks(*ora.blocks())
    assert np.array_equal(gk, ok)
    assert np.array_equal(gv.ravel(), ov.view(np.uint32).ravel())
    vol.close()
    ora.close()


@pytest.mark.parametrize("form", ["plain", "chosen"])
def test_incremental_mesh_is_every_triangle_of_its_blocks(env, small_orbit, form):
    """vh_extract_mesh_recent gives all triangles of the full extraction whose cells belong to the blocks of the last frames,
    and no others: as a volume's first extraction on a stream of its own with the default stream busy, again with
    the next epochs and two frames, and after a full extraction.  A triangle lies in its cell, so its centroid tells
    the cell unless it is within rounding of the cell's border (those may be of either)."""
    from collections import Counter
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    sc, on = small_orbit, int(form == "chosen")
    vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 16, max_blocks=8192, layer_format=on,
                                algorithm=_capi.default_algorithm(allocation_mode=on, normal_mode=on))
    stream = torch.cuda.Stream()
    visible = []

    def integrate(f):
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, scenes.render_depth(sc, f)), sc.poses[f])
        visible.append({tuple(k) for k in backend.visible_block_keys(vol)})

    def check(recent, frames):
        full = backend.extract_mesh_cuda(vol)
        listed = set().union(*visible[-frames:])
        g = full.reshape(-1, 3, 3).astype(np.float64).mean(1) / sc.voxel_size - 0.5
        near = (np.abs(g - np.round(g)) < 1e-3).any(1)
        inside = np.array([tuple(b) in listed for b in np.floor(g).astype(np.int64) >> 3])
        rows = [r.tobytes() for r in np.ascontiguousarray(full).reshape(len(g), -1)]
        got = Counter(r.tobytes() for r in np.ascontiguousarray(recent).reshape(len(recent), -1))
        must = Counter(r for r, i, n in zip(rows, inside, near) if i and not n)
        may = must + Counter(r for r, n in zip(rows, near) if n)
        assert 1000 < sum(must.values()) and sum(may.values()) < len(rows) and near.sum() < 0.05 * len(rows)
        assert not must - got and not got - may

    for f in (0, 6, 12, 18):
        integrate(f)
    vol.synchronize()
    torch.cuda._sleep(200_000_000)
    check(backend.extract_mesh_cuda(vol, recent_frames=1, stream=stream), 1)
    integrate(9)
    check(backend.extract_mesh_cuda(vol, recent_frames=1), 1)
    check(backend.extract_mesh_cuda(vol, recent_frames=2, stream=stream), 2)
    integrate(3)
    check(backend.extract_mesh_cuda(vol, recent_frames=1), 1)
    vol.close()


@pytest.mark.parametrize("zero", [("filter_sigma_spatial",), ("filter_sigma_range",), ("filter_sigma_angular",),
                                  ("normal_sigma_spatial",), ("normal_sigma_range",), ("normal_sigma_angular",),
                                  ("filter_sigma_range", "filter_sigma_angular", "normal_sigma_range", "normal_sigma_angular"), ()])
def test_sigmas_of_zero_and_infinite_depth(env, small_orbit, zero):
    """Sums that are no numbers: a sigma of 0 (its factor is infinite, and the centre's weight NaN), and an infinite depth that
    no discontinuity threshold leaves out (a weight of 0 times infinity).  The filtered depth, in small and large tiles,
    and the fused layers are the oracle's; of a layer whose normal is NaN, the weight and the surface coordinate (the bits of
    its plane offset and its packed normal depend on the machine's NaN)."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    sc = small_orbit
    ours, oras = {k: 0.0 for k in zero}, {k: 0.0 for k in zero}
    if not zero:
        ours, oras = {"depth_discontinuity_base": np.inf}, {"disc_base": np.inf}
    vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 16, max_blocks=8192,
                                algorithm=_capi.default_algorithm(**ours))
    cfg = O.config(O.FLAVOR_REF_GPU, O.EXP_OWN, threads=8, **oras)
    ora = O.Volume(cfg, sc.voxel_size, sc.truncation)
    for f in (0, 3, 6):
        d = scenes.render_depth(sc, f)
        if f == 3:
            d[10:30, 10:40] = 1.25  # neighbours of equal depth
        backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, d), sc.poses[f])
        ora.integrate(d, sc.intrinsics, sc.poses[f])
        if not zero:
            d[20, 20] = np.inf
        for w, h in ((64, 48), (1000, 480)):
            K = scenes.Intrinsics(w, h, sc.intrinsics.fx, sc.intrinsics.fy, sc.intrinsics.cx, sc.intrinsics.cy)
            Ki, img = _capi.intrinsics(K), np.zeros((h, w), np.float32)
            img[:48, :64] = d
            src, out = torch.from_numpy(img).cuda(), torch.empty((h, w), device="cuda")
            torch.cuda.synchronize()
            _capi.check(_capi.lib().vh_filter_depth(vol.handle, C.c_void_p(src.data_ptr()), C.c_void_p(out.data_ptr()),
                                                    C.byref(Ki), None), vol.handle)
            vol.synchronize()
            assert np.array_equal(out.cpu().numpy(), O.filter_depth(cfg, img, K), equal_nan=True), (f, w)
    gk, gv = O.sort_blocks(*vol.export_blocks())
    ok, ov = O.sort_blocks(*ora.blocks())
    assert np.array_equal(gk, ok)
    got, want = gv.reshape(-1, 4), ov.view(np.uint32).reshape(-1, 4)
    assert np.array_equal(got[:, :2], want[:, :2])
    nan = np.isnan(want[:, 2].copy().view(np.float32))
    assert np.array_equal(np.isnan(got[:, 2].copy().view(np.float32)), nan)
    assert np.array_equal(got[~nan, 2:], want[~nan, 2:])
    vol.close()
    ora.close()


@pytest.mark.parametrize("rows", [262140, 262141, 400001])
def test_raycast_of_a_tall_image(env, small_orbit, rows):
    """One column of more rows than a grid holds tiles along y (65,535 of 4 rows), against the oracle's ray-cast."""
    backend, O = env
    from voxelhashmt_gb300 import scenes
    sc = small_orbit
    vol, ora = _fuse(backend, O, sc, [0, 4, 8, 12], 0)
    K = scenes.Intrinsics(1, rows, 55.4, 55.4 * rows / 48, 0.0, (rows - 1) / 2.0)
    got = backend.raycast_depth(vol, K, sc.poses[2], 0.0, 3.0, 1.0)
    want = ora.raycast_depth(K, sc.poses[2], 0.0, 3.0, 1.0)
    assert (want > 0).sum() > 1000
    assert np.array_equal(_bits(got), _bits(want))
    vol.close()
    ora.close()


@pytest.mark.parametrize("alloc,normal", [(1, 1), (0, 0)])
def test_fast_math_frames_do_not_depend_on_the_tiles(env, alloc, normal):
    """The fast-math compile gives a frame the same filtered depth, blocks, layers and normal map, word for word, whether its
    image is worked on in small tiles (160x120: 75 of 32x8), its filter and allocation in large ones (320x240: 300) or its
    normal map too (960x360: 1,350).  The frame is the same one, with zeros around it."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, scenes
    w, h = 160, 120
    sc = scenes.orbit_scene(seed=7, frames=8, width=w, height=h, fx=138.5, fy=138.5, cx=w / 2.0, cy=h / 2.0)
    sc.voxel_size, sc.truncation = 0.02, 0.06
    want = None
    for W, H in ((160, 120), (320, 240), (960, 360)):
        K = scenes.Intrinsics(W, H, 138.5, 138.5, w / 2.0, h / 2.0)
        vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 16, max_blocks=16384,
                                    algorithm=_capi.default_algorithm(allocation_mode=alloc, normal_mode=normal, fast_math=1,
                                                                      autotune=0))
        Ki, nrm, maps = _capi.intrinsics(K), torch.empty((H, W, 4), device="cuda"), []
        for f in (0, 3, 6):
            d = np.zeros((H, W), np.float32)
            # a border of zeros in the small image too: beyond it a projection finds no depth in either
            d[2:h - 2, 2:w - 2] = scenes.render_depth(sc, f)[2:-2, 2:-2]
            src = torch.from_numpy(d).cuda()
            backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(K, src.view(-1)), sc.poses[f])
            _capi.check(_capi.lib().vh_pixel_normals(vol.handle, C.c_void_p(src.data_ptr()), C.c_void_p(nrm.data_ptr()),
                                                     C.byref(Ki), None), vol.handle)
            vol.synchronize()
            maps.append(_bits(nrm.cpu().numpy()[:h, :w]))
        got = (*O.sort_blocks(*vol.export_blocks()), np.stack(maps))
        vol.close()
        want = want or got
        assert len(got[0]) > 100 and all(np.array_equal(a, b) for a, b in zip(got, want)), (W, H)


@pytest.mark.parametrize("alloc,fp16", [(1, 0), (0, 0), (1, 1)])
def test_fast_math_normals_per_voxel_are_reproducible(env, alloc, fp16):
    """A scan in the fast-math compile with a normal per voxel gives the same words each time.  The room's voxels project onto the
    image's border and beside pixels without depth in every frame; an update that found no centre sample for a listed
    voxel would take its depth from what another voxel left in shared memory."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, denoiser, scenes
    sc = scenes.room_scene(1, frames=64)
    sc.voxel_size, sc.truncation, sc.poses = 0.005, 0.02, sc.poses[1:9]
    frames, want = denoiser.render_frames(sc, torch), None
    for _ in range(4):
        vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 18, max_blocks=32768, layer_format=fp16,
                                    algorithm=_capi.default_algorithm(allocation_mode=alloc, normal_mode=0, fast_math=1))
        for d, pose in zip(frames, sc.poses):
            backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, d.view(-1)), pose, synchronize=False)
        got = _device_blocks(vol)
        vol.close()
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert len(want[0]) > 10000


@pytest.mark.parametrize("scene", ["room", "object"])
def test_fast_math_records_do_not_depend_on_the_launch(env, scene):
    """With FP32 bins the fast-math compile fuses the same words in each of the update's ten launch shapes, and as a batch of one
    (one launch per kernel, one graph, one persistent launch)."""
    backend, O = env
    from voxelhashmt_gb300 import _capi, denoiser, scenes
    if scene == "room":
        sc = scenes.room_scene(1, frames=64)
        sc.voxel_size, sc.truncation, sc.poses = 0.005, 0.02, sc.poses[1:5]
    else:
        sc = scenes.object_scan_scene(3, frames=24, resolution=(160, 120), voxel_size=0.008)
        sc.truncation = 4.0 * sc.voxel_size
    frames, want = denoiser.render_frames(sc, torch), None
    for launch in [*range(10), False, True, "persistent"]:
        single = not isinstance(launch, (bool, str))
        vol = backend.VoxelHashTSDF(sc.voxel_size, sc.truncation, hash_buckets=1 << 18, max_blocks=16384,
                                    algorithm=_capi.default_algorithm(allocation_mode=1, normal_mode=1, fast_math=1, autotune=0,
                                                                      launch_variant=launch if single else 0))
        batch = None if single else backend.VolumeBatch([vol], launch)
        for d, pose in zip(frames, sc.poses):
            if single:
                backend.integrate_depth_frame_cuda(vol, backend.DepthFrame(sc.intrinsics, d.view(-1)), pose, synchronize=False)
            else:
                batch.integrate([d], [sc.intrinsics], [pose], 1)
        vol.synchronize()
        got = _device_blocks(vol)
        if batch:
            batch.close()
        vol.close()
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want)), launch
    assert len(want[0]) > 500


def _device_blocks(vol):
    """(keys, voxel words) of a volume in the order of the keys, on the device."""
    from voxelhashmt_gb300 import _capi
    n = vol.block_count()
    keys = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    words = torch.empty((n, 512 * 6 * 3 * 4), dtype=torch.int32, device="cuda")
    _capi.check(_capi.lib().vh_export_blocks(vol.handle, 0, n, C.cast(C.c_void_p(keys.data_ptr()), C.POINTER(C.c_int32)),
                                             C.c_void_p(words.data_ptr()), 1, None), vol.handle)
    k = keys.long() + (1 << 20)
    order = torch.argsort((k[:, 2] << 42) | (k[:, 1] << 21) | k[:, 0])
    return keys[order], words[order]
