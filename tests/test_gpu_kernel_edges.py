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
