"""Host code of the library against a fake CUDA runtime (no GPU): whichever CUDA
call fails, a call returns with no copy of the caller's buffers still pending.
And the order of the copies that a small call waits for."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpu-compressor_b200", "csrc")
FAKE = os.path.join(ROOT, "tests", "fake_cuda", "fake_cuda.cpp")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake_cuda")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    out = str(d / "libgcz_host.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++17", "-cudart", "none",
                    "-shared", "-Xlinker", "-Bsymbolic", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"),
                    "-I", CSRC, os.path.join(CSRC, "gcz_api.cu"), FAKE, "-o", out, "-lpthread"], check=True)
    L = ctypes.CDLL(out)
    vp, sz = ctypes.c_void_p, ctypes.c_size_t
    L.gcz_create.argtypes = [ctypes.c_int, ctypes.POINTER(vp)]
    L.gcz_destroy.argtypes = [vp]
    for f in (L.gcz_zstd_match_find, L.gcz_zstd_match_find_packed):
        f.argtypes = [vp, vp, sz, ctypes.c_uint32, vp, sz, vp]
    L.gcz_lzma2_match_find.argtypes = [vp, vp, sz, ctypes.c_uint32, vp, vp]
    L.gcz_zstd_compress_frames_gpu.argtypes = [vp, vp, sz, ctypes.c_uint32, vp, sz, vp, vp]
    L.gcz_set_option.argtypes = [vp, ctypes.c_char_p, ctypes.c_long]
    L.gcz_last_error.argtypes, L.gcz_last_error.restype = [vp], ctypes.c_char_p
    L.fake_last_to.argtypes = [vp]
    L.fake_fail_at.argtypes = [ctypes.c_long]
    L.fake_calls.restype = ctypes.c_long
    L.fake_pending.argtypes, L.fake_pending.restype = [vp, sz], ctypes.c_long
    return L


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("n", [1, 4096, 200_003, 262_144])
def test_small_call_leaves_nothing_pending(lib, n, packed):
    src = np.zeros(n, np.uint8)
    seqs = np.zeros(n * 4 + 16, np.uint32)
    offsets = np.zeros(8, np.uint64)
    call = lib.gcz_zstd_match_find_packed if packed else lib.gcz_zstd_match_find

    def run(fail_at):
        h = ctypes.c_void_p()
        lib.fake_fail_at(0)
        assert lib.gcz_create(0, ctypes.byref(h)) == 0
        lib.fake_fail_at(fail_at)
        rc = call(h, src.ctypes.data, n, 16, seqs.ctypes.data, n, offsets.ctypes.data)
        calls = lib.fake_calls()
        lib.fake_fail_at(0)
        left = [lib.fake_pending(a.ctypes.data, a.nbytes) for a in (src, seqs, offsets)]
        lib.gcz_destroy(h)
        return rc, calls, left

    rc, calls, left = run(0)
    assert rc == 0 and left == [0, 0, 0] and calls > 5
    for k in range(1, calls + 1):
        rc, _, left = run(k)
        assert rc != 0, k
        assert left == [0, 0, 0], k


@pytest.mark.parametrize("n", [1, 4096, 200_003])
def test_lzma_results_leave_last(lib, n):
    """A copy to pageable memory holds the host up: nothing may be queued behind it."""
    src, packed, has = np.zeros(n, np.uint8), np.zeros(n, np.uint32), np.zeros(4, np.uint8)
    h = ctypes.c_void_p()
    lib.fake_fail_at(0)
    assert lib.gcz_create(0, ctypes.byref(h)) == 0
    assert lib.gcz_lzma2_match_find(h, src.ctypes.data, n, 32, packed.ctypes.data, has.ctypes.data) == 0
    last = lib.fake_last_to(packed.ctypes.data)
    lib.gcz_destroy(h)
    assert last


@pytest.mark.parametrize("kind", ["sequences", "packed", "lzma", "triage", "frames"])
@pytest.mark.parametrize("n", [65536, 9 * 65536 + 1])
def test_sliced_call_leaves_nothing_pending(lib, n, kind):
    nb = (n + 65535) // 65536
    src, out = np.zeros(n, np.uint8), np.zeros(n * 4 + 1024 * nb, np.uint32)
    small, size = np.zeros(nb + 1, np.uint64), np.zeros(1, np.uint64)
    s, o, m = src.ctypes.data, out.ctypes.data, small.ctypes.data
    call = {
        "sequences": lambda h: lib.gcz_zstd_match_find(h, s, n, 16, o, n, m),
        "packed": lambda h: lib.gcz_zstd_match_find_packed(h, s, n, 16, o, n, m),
        "lzma": lambda h: lib.gcz_lzma2_match_find(h, s, n, 32, o, m),
        "triage": lambda h: lib.gcz_lzma2_match_find(h, s, n, 32, None, m),
        "frames": lambda h: lib.gcz_zstd_compress_frames_gpu(h, s, n, 1, o, out.nbytes, m, size.ctypes.data),
    }[kind]

    def run(fail_at):
        h = ctypes.c_void_p()
        lib.fake_fail_at(0)
        assert lib.gcz_create(0, ctypes.byref(h)) == 0
        for key in (b"slice_windows", b"frames_slice_windows"):
            assert lib.gcz_set_option(h, key, 2) == 0
        lib.fake_fail_at(fail_at)
        rc = call(h)
        calls = lib.fake_calls()
        lib.fake_fail_at(0)
        left = [lib.fake_pending(a.ctypes.data, a.nbytes) for a in (src, out, small)]
        why = lib.gcz_last_error(h)
        lib.gcz_destroy(h)
        return rc, calls, left, why

    rc, calls, left, _ = run(0)
    assert rc == 0 and left == [0, 0, 0] and calls > 5
    for k in range(1, calls + 1):
        rc, _, left, why = run(k)
        assert rc != 0 and why, k
        assert left == [0, 0, 0], k
