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
    """create(device) -> handle of a small volume; closed at the end."""
    capi, L = host
    L.fake_fail(0, 0, 0)
    made = []

    def create(device=0):
        h = C.c_void_p()
        params = capi.default_params(voxel_size=0.02, truncation_distance=0.06, hash_buckets=1 << 10, max_blocks=64)
        params.device = device
        assert L.vh_create(C.byref(params), None, C.byref(h)) == capi.VH_OK
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
