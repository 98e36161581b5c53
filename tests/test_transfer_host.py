"""The transfers through pinned buffers (csrc/transfer.cpp) against a CUDA runtime that is a fake on the host: what they pin,
what they do when nothing more can be pinned, and that every value arrives whatever the sizes.  The fake's device memory
is host memory, its copies are done when issued, and it can be told to refuse pinned memory or a copy."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lionbolt_b200", "csrc")

FAKE = r"""
#include "lb_internal.h"
#include <cstdlib>
#include <cstring>
static long long g_pinned = 0, g_pin_limit = -1, g_copies = 0, g_fail_at = -1;
extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) {
    if (g_pin_limit >= 0 && g_pinned + (long long)n > g_pin_limit) return cudaErrorMemoryAllocation;
    g_pinned += n;
    size_t* q = (size_t*)std::malloc(n + 64);
    *q = n;
    *p = (char*)q + 64;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    size_t* q = (size_t*)((char*)p - 64);
    g_pinned -= *q;
    std::free(q);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free((void*)e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (g_copies++ == g_fail_at) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
}
namespace lb {
int cuda_fail(Handle*, cudaError_t, const char*) { return LB_ERR_CUDA; }
int fail(Handle*, int code, const std::string&) { return code; }
}
extern "C" {
void* t_new() {
    lb::Handle* h = new lb::Handle();
    h->h_red = (double*)std::malloc(sizeof(double) * lb::kRedHost + 2 * lb::kPipeSmall);
    return h;
}
void t_free(void* p) {
    lb::Handle* h = (lb::Handle*)p;
    lb::pipe_free(h);
    std::free(h->h_red);
    delete h;
}
long long t_pinned() { return g_pinned; }
void t_pin_limit(long long n) { g_pin_limit = n; }
void t_fail_after(long long n) { g_fail_at = n < 0 ? -1 : g_copies + n; }
int t_up_f32(void* h, float* d, const double* s, size_t n) { return lb::pipe_up_f32((lb::Handle*)h, d, s, n, ""); }
int t_down_f32(void* h, double* d, const float* s, size_t n, int sub) { return lb::pipe_down_f32((lb::Handle*)h, d, s, n, sub, ""); }
int t_up(void* h, void* d, const void* s, size_t n) { return lb::pipe_up((lb::Handle*)h, d, s, n, ""); }
int t_down(void* h, void* d, const void* s, size_t n) { return lb::pipe_down((lb::Handle*)h, d, s, n, ""); }
}
"""

MB = 1 << 20
# around the small buffers (95 KB), the step to the large ones (4 MB), their chunks (512 KB) and the threads' parts
BYTES = [1, 95 * 1024, 95 * 1024 + 1, 190 * 1024 + 1, 4 * MB, 4 * MB + 1, 5 * MB - 3, 9 * MB + 17]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("transfer")
    (d / "fake.cpp").write_text(FAKE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    cxx = "/usr/bin/g++" if os.access("/usr/bin/g++", os.X_OK) else "g++"      # as the Makefile
    subprocess.check_call([cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-fopenmp", f"-I{CSRC}",
                           f"-I{cuda}/include", str(d / "fake.cpp"), os.path.join(CSRC, "transfer.cpp"), "-o",
                           str(d / "libfake.so")])
    lib = ctypes.CDLL(str(d / "libfake.so"))
    v, n = ctypes.c_void_p, ctypes.c_size_t
    lib.t_new.restype, lib.t_pinned.restype = v, ctypes.c_longlong
    lib.t_free.argtypes = [v]
    lib.t_pin_limit.argtypes = lib.t_fail_after.argtypes = [ctypes.c_longlong]
    lib.t_up_f32.argtypes = lib.t_up.argtypes = lib.t_down.argtypes = [v, v, v, n]
    lib.t_down_f32.argtypes = [v, v, v, n, ctypes.c_int]
    return lib


@pytest.fixture
def handle(lib):
    h = lib.t_new()
    yield h
    lib.t_pin_limit(-1)
    lib.t_fail_after(-1)
    lib.t_free(h)


def _p(a):
    return a.ctypes.data


def _round_trip(lib, h, nbytes, seed=0):
    r = np.random.default_rng(seed)
    src = r.integers(0, 256, nbytes, dtype=np.uint8)
    dev, back = np.zeros_like(src), np.zeros_like(src)
    assert lib.t_up(h, _p(dev), _p(src), nbytes) == 0 and np.array_equal(dev, src)
    assert lib.t_down(h, _p(back), _p(dev), nbytes) == 0 and np.array_equal(back, src)
    n = max(1, nbytes // 4)
    x = r.normal(size=n)
    f, y = np.zeros(n, np.float32), np.zeros(n)
    assert lib.t_up_f32(h, _p(f), _p(x), n) == 0 and np.array_equal(f, x.astype(np.float32))
    assert lib.t_down_f32(h, _p(y), _p(f), n, 0) == 0 and np.array_equal(y, f.astype(np.float64))
    assert lib.t_down_f32(h, _p(x), _p(f), n, 1) == 0 and np.abs(x).max() < 1e-6


@pytest.mark.parametrize("nbytes", BYTES)
def test_every_value_arrives(lib, handle, nbytes):
    _round_trip(lib, handle, nbytes)
    _round_trip(lib, handle, 300 * 1024, seed=1)     # through whichever pair the handle has by now
    lib.t_pin_limit(lib.t_pinned())
    _round_trip(lib, handle, nbytes, seed=2)


@pytest.mark.parametrize("allowed", [0, MB // 2])
def test_without_pinned_memory_the_small_buffers_do(lib, handle, allowed):
    before = lib.t_pinned()
    lib.t_pin_limit(before + allowed)               # none, or one buffer of the pair
    _round_trip(lib, handle, 9 * MB + 17)
    assert lib.t_pinned() == before


def test_a_first_large_transfer_pins_little(lib, handle):
    """Pinning takes 0.5 ms per MB: a pair that costs more than the one call it is for makes that call slower."""
    before = lib.t_pinned()
    _round_trip(lib, handle, 4 * MB)
    assert lib.t_pinned() == before
    _round_trip(lib, handle, 6 * MB)
    assert 0 < lib.t_pinned() - before <= MB


@pytest.mark.parametrize("refused", [False, True])
def test_a_handle_that_moves_much_gets_larger_buffers(lib, handle, refused):
    before = lib.t_pinned()
    src, dev = np.ones(16 * MB, np.uint8), np.zeros(16 * MB, np.uint8)
    for k in range(9):
        if k == 8 and refused:
            lib.t_pin_limit(lib.t_pinned())
        assert lib.t_up(handle, _p(dev), _p(src), src.size) == 0
        assert lib.t_pinned() - before == (8 * MB if k == 8 and not refused else MB)
    _round_trip(lib, handle, 9 * MB + 17)


@pytest.mark.parametrize("nbytes", BYTES)
def test_a_difference_is_taken_whole_or_not_at_all(lib, handle, nbytes):
    """The subtracted-from vector is the caller's operand: a copy that fails, whichever it is, leaves it as it was."""
    n = max(1, nbytes // 4)
    r = np.random.default_rng(3)
    x, y = r.normal(size=n), r.normal(size=n).astype(np.float32)
    failed = 0
    for k in range(64):
        lib.t_fail_after(k)
        out = x.copy()
        rc = lib.t_down_f32(handle, _p(out), _p(y), n, 1)
        assert np.array_equal(out, x if rc else x - y)
        failed += rc != 0
        if rc == 0:
            break
    assert failed >= 1
