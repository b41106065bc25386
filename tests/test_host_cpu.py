"""The library's host code against a CUDA runtime without a GPU (fake_cuda_runtime.c): what a call leaves behind for the
next one, the order of its work on the caller's stream, and the second device of a process."""
import ctypes as C
import os
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
STREAM = C.c_void_p(0x5000)  # a stream that does not wait for the legacy one


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    """The library linked with the fake runtime; the device code is compiled without optimisation, as none of it runs."""
    from voxelhashmt_gb300 import _capi
    from voxelhashmt_gb300 import build as pb
    out = str(tmp_path_factory.mktemp("host"))

    def compile_one(unit):
        src, name, extra = unit
        obj = os.path.join(out, name + ".o")
        pb._run([pb.nvcc(), *pb.ARCH, "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17", "-Xcompiler", "-fPIC,-O1", "-I", pb.CSRC,
                 "-I", pb.INCLUDE, *extra, "-x", "cu", "-c", os.path.join(pb.CSRC, src), "-o", obj])
        return obj

    units = [(src, os.path.splitext(src)[0], []) for src in pb.SOURCES] + pb.VARIANTS
    with ThreadPoolExecutor(max_workers=len(units)) as ex:
        objs = list(ex.map(compile_one, units))
    lib = os.path.join(out, "libhost.so")
    pb._run(["gcc", "-O1", "-fPIC", "-c", os.path.join(HERE, "fake_cuda_runtime.c"), "-o", os.path.join(out, "fake.o")])
    pb._run(["g++", "-shared", "-o", lib, *objs, os.path.join(out, "fake.o"), "-Wl,-Bsymbolic", "-Wl,-z,defs"])
    L = C.CDLL(lib)
    for name, (res, args) in _capi._SIGNATURES.items():
        getattr(L, name).restype, getattr(L, name).argtypes = res, args
    return _capi, L


@pytest.fixture
def volume(host):
    """create(algorithm options) -> handle of a small volume; closed at the end."""
    capi, L = host
    L.fake_fail(0, 0, 0)
    made = []

    def create(**algorithm):
        h = C.c_void_p()
        params = capi.default_params(voxel_size=0.02, truncation_distance=0.06, hash_buckets=1 << 10, max_blocks=64)
        assert L.vh_create(C.byref(params), C.byref(capi.default_algorithm(**algorithm)), C.byref(h)) == capi.VH_OK
        made.append(h)
        return h

    yield create
    L.fake_fail(0, 0, 0)
    for h in made:
        L.vh_destroy(h)


def _buffer(n=1 << 16):
    return C.cast((C.c_ubyte * (n + 256))(), C.c_void_p)


def _intrinsics(capi, w=16, h=12):
    from voxelhashmt_gb300 import scenes
    return C.byref(capi.intrinsics(scenes.Intrinsics(w, h, 20.0, 20.0, w / 2, h / 2)))


def test_work_on_the_legacy_stream_is_waited_for(host, volume):
    """Every clear and copy of a call that is given a stream is enqueued on that stream, or has been waited for by the time
    that the call enqueues more: a stream that does not wait for the legacy one would overtake it."""
    capi, L = host
    h = volume()
    assert L.fake_legacy_pending() == 0  # vh_create waits for its clears
    n = C.c_size_t()
    for _ in range(2):
        assert L.vh_extract_mesh_recent(h, 0.0, 1, C.byref(n), STREAM) == capi.VH_OK
        assert L.fake_legacy_pending() == 0
    assert L.vh_extract_mesh(h, 0.0, C.byref(n), STREAM) == capi.VH_OK
    assert L.vh_reset(h, STREAM) == capi.VH_OK
    assert L.fake_legacy_pending() == 0


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_a_batch_is_cleared_before_its_first_step(host, volume, mode):
    """The queue and barrier words of a batch, cleared on the legacy stream, are zero when vh_batch_create returns: a step on
    a stream that does not wait for the legacy one may follow at once."""
    capi, L = host
    vols = (C.c_void_p * 2)(volume(normal_mode=1), volume(normal_mode=1))
    b = C.c_void_p()
    assert L.vh_batch_create(vols, 2, mode, C.byref(b)) == capi.VH_OK
    assert L.fake_legacy_pending() == 0
    L.vh_batch_destroy(b)


def _failing_calls(capi, L, h):
    """name -> (copies, launches, attributes) that fail, and a call that meets them."""
    K, b, n, f = _intrinsics(capi), _buffer(), C.c_uint64(), C.c_uint32()
    pose = C.byref(capi.VhPose(R=(C.c_float * 9)(1, 0, 0, 0, 1, 0, 0, 0, 1)))
    ip = C.cast(b, C.POINTER(C.c_int32))
    up = C.cast(b, C.POINTER(C.c_uint32))
    ws = _buffer(L.vh_nn_workspace_bytes(1, 16, 12))
    return {
        "copy of a volume's call": ((1, 0, 0), lambda: L.vh_block_count(h, C.byref(n))),
        "blocks into a buffer": ((1, 0, 0), lambda: L.vh_export_blocks(h, 0, 0, ip, b, 1, STREAM)),
        "dependent launch": ((0, 1, 0), lambda: L.vh_filter_depth(h, b, b, K, STREAM)),
        "frame": ((0, 2, 0), lambda: L.vh_integrate(h, b, 1, K, pose, 1, STREAM)),
        "kernel attribute": ((0, 0, 1), lambda: L.vh_nn_conv32(b, b, None, None, b, 1, 16, 12, 0, 0, up, STREAM)),
        "tensor-core launch": ((0, 1, 0), lambda: L.vh_nn_conv32(b, b, None, None, b, 1, 16, 12, 0, 0, up, STREAM)),
        "denoiser": ((0, 2, 0), lambda: L.vh_nn_forward(b, b, b, b, 1, 16, 12, ws, up, STREAM)),
        "denoiser parameters": ((1, 0, 0), lambda: L.vh_set_depth_denoiser(h, C.cast(b, C.POINTER(C.c_float)))),
        "exponential check": ((1, 0, 0), lambda: L.vh_expf_check(0, 16, C.byref(n), C.byref(f), STREAM)),
    }


@pytest.mark.parametrize("name", ["copy of a volume's call", "blocks into a buffer", "dependent launch", "frame",
                                  "kernel attribute", "tensor-core launch", "denoiser", "denoiser parameters",
                                  "exponential check"])
def test_a_failed_call_does_not_fail_the_next(host, volume, name):
    """The error of a call that fails is that call's alone: the next one, on the same volume or on another, succeeds."""
    capi, L = host
    h, other = volume(), volume()
    n = C.c_uint64()
    fails, call = _failing_calls(capi, L, h)[name]
    L.fake_fail(*fails)
    status = call()
    L.fake_fail(0, 0, 0)
    assert status == capi.VH_ERR_CUDA
    for v in (other, h):
        assert L.vh_recount_observed_voxels(v, C.byref(n), STREAM) == capi.VH_OK


def test_denoiser_on_every_device(host, volume):
    """The kernels that need more than 48 KB of shared memory are allowed it on each device that runs them, and a refusal is not
    kept: forward and backward pass and both entry points of a single layer, on the first device, on the second,
    and after a call that failed."""
    capi, L = host
    K, b = (1, 16, 12), _buffer(1 << 20)
    up, fp = C.cast(b, C.POINTER(C.c_uint32)), b
    ws = _buffer(L.vh_nn_workspace_bytes(*K))
    calls = {
        "forward": lambda: L.vh_nn_forward(fp, b, fp, fp, *K, ws, up, STREAM),
        "backward": lambda: L.vh_nn_backward(fp, b, fp, fp, fp, *K, ws, fp, fp, up, STREAM),
        "conv32": lambda: L.vh_nn_conv32(b, b, None, None, b, *K, 0, 0, up, STREAM),
        "wgrad32": lambda: L.vh_nn_wgrad32(b, b, fp, fp, *K, up, STREAM),
    }
    for device in (1, 0, 1):
        L.cudaSetDevice(device)
        for name, call in calls.items():
            L.fake_fail(0, 0, 1)
            assert call() == capi.VH_ERR_CUDA, (device, name)
            L.fake_fail(0, 0, 0)
            before = L.fake_launches()
            assert call() == capi.VH_OK, (device, name)
            assert L.fake_launches() > before
    L.cudaSetDevice(0)
