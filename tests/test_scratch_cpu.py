"""The runtime's scratch (csrc/capi.cu) over a stand-in for the CUDA runtime.

capi.cu is compiled as it is and linked with a small allocator in host memory:
the lowest free place that is large enough, contents left as they were, a
limit on the bytes in use.  A buffer that grows may thus come back at its old
address with another allocation's contents, as cudaFree and cudaMalloc may
give it.
"""
import ctypes
import subprocess

import pytest

from clustkit_gb300 import build

RUNTIME = r"""
#include <cstdint>
#include <cstring>
#include <map>
#include <vector>
#include <cuda_runtime_api.h>

static std::vector<char> heap((size_t)64 << 20, (char)0x5a);
static std::map<size_t, size_t> used;  // offset -> bytes
static size_t limit = 0;               // bytes that may be in use; 0: the heap
static size_t in_use() { size_t n = 0; for (auto &u : used) n += u.second; return n; }
static size_t most() { return limit ? limit : heap.size(); }

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    n = (n + 255) & ~(size_t)255;
    *p = nullptr;
    if (in_use() + n > most()) return cudaErrorMemoryAllocation;
    size_t at = 0;
    for (auto &u : used) {
        if (u.first - at >= n) break;
        at = u.first + u.second;
    }
    if (at + n > heap.size()) return cudaErrorMemoryAllocation;
    used[at] = n;
    *p = heap.data() + at;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { if (p) used.erase((char *)p - heap.data()); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *t = most(); *f = most() - in_use(); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) { memset(p, 0, sizeof *p); p->multiProcessorCount = 4; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { *t = 0; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
int64_t t_in_use() { return (int64_t)in_use(); }
void t_limit(int64_t n) { limit = (size_t)n; }
void *t_malloc(int64_t n) { void *p; return cudaMalloc(&p, (size_t)n) == cudaSuccess ? p : nullptr; }
void t_free(void *p) { cudaFree(p); }
}
"""

REST = r"""
#include <new>
#include "ck_common.cuh"
namespace ck {
int32_t sw_plain_launch(const SwIn &, const SwOut &, int64_t, const int32_t *, const int32_t *, int32_t *, cudaStream_t, SwCounters *) { return 0; }
int32_t sw_batched_launch(const SwIn &, const SwOut &, int64_t, const int8_t *, int32_t *, cudaStream_t, SwCounters *, bool) { return 0; }
int32_t sketch_launch(const uint8_t *, int64_t, const int64_t *, const int32_t *, int64_t, int32_t, int32_t, int32_t, uint64_t, uint64_t *, int32_t *, cudaStream_t) { return 0; }
int32_t jaccard_launch(const int32_t *, int64_t, const uint64_t *, int64_t, int32_t, float, float *, uint8_t *, int32_t *, cudaStream_t) { return 0; }
int32_t sw_set_rows_per_strip(int32_t) { return 0; }
int32_t sw_rows_per_strip() { return 0; }
int32_t sw_set_strip_threads(int32_t) { return 0; }
int32_t sw_strip_threads() { return 0; }
int32_t sw_set_wide_key(int32_t) { return 0; }
int32_t sw_wide_key() { return 0; }
int32_t sw_set_variant(int32_t) { return 0; }
int32_t sw_variant() { return 0; }
int32_t sw_set_wave(int32_t, int32_t) { return 0; }
int32_t sw_wave(int32_t) { return 0; }
}

struct Ask { int32_t slot; size_t bytes; bool zeroed; char *p; };
static int32_t ask(void *pv) {
    Ask &a = *(Ask *)pv;
    int32_t status = CK_OK;
    a.p = (char *)(a.zeroed ? ck::scratch_zeroed(a.slot, a.bytes, nullptr, &status) : ck::scratch(a.slot, a.bytes, &status));
    return status;
}
static int32_t no_memory(void *) { throw std::bad_alloc(); }
extern "C" {
int32_t t_no_memory(int32_t ctx) { return ck::run_in_context(ctx, no_memory, nullptr); }
// The buffer of a context's slot, or null; *nonzero the bytes of it that are not zero.
void *t_scratch(int32_t ctx, int32_t slot, int64_t bytes, int32_t zeroed, int64_t *nonzero) {
    Ask a{slot, (size_t)bytes, zeroed != 0, nullptr};
    if (ck::run_in_context(ctx, ask, &a) != CK_OK) return nullptr;
    *nonzero = 0;
    for (int64_t i = 0; i < bytes; ++i) *nonzero += a.p[i] != 0;
    return a.p;
}
int32_t t_bins() { return ck::SLOT_SEARCH_BINS; }
}
"""


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    at = tmp_path_factory.mktemp("runtime")
    (at / "runtime.cpp").write_text(RUNTIME)
    (at / "rest.cu").write_text(REST)
    objects = []
    for src in (build.CSRC / "capi.cu", at / "runtime.cpp", at / "rest.cu"):
        objects.append(str(at / (src.stem + ".o")))
        subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-c", str(src), "-o", objects[-1]], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", str(at / "runtime.so"), *objects, "-lpthread"],
                   check=True)
    return at / "runtime.so"


@pytest.fixture
def rt(library, tmp_path):
    """A copy of the library with state of its own."""
    own = tmp_path / "runtime.so"
    own.write_bytes(library.read_bytes())
    lib = ctypes.CDLL(str(own))
    for name in ("t_scratch", "t_malloc"):
        getattr(lib, name).restype = ctypes.c_void_p
    lib.t_scratch.argtypes = [ctypes.c_int32, ctypes.c_int32, ctypes.c_int64, ctypes.c_int32, ctypes.c_void_p]
    lib.t_malloc.argtypes, lib.t_limit.argtypes = [ctypes.c_int64], [ctypes.c_int64]
    lib.t_free.argtypes = [ctypes.c_void_p]
    lib.t_in_use.restype = ctypes.c_int64
    return lib


def _create(rt):
    h = ctypes.c_int32()
    assert rt.ck_ctx_create(ctypes.byref(h)) == 0
    return h.value


def _scratch(rt, ctx, slot, nbytes, zeroed=False):
    n = ctypes.c_int64()
    p = rt.t_scratch(ctx, slot, nbytes, int(zeroed), ctypes.byref(n))
    return p, n.value


@pytest.mark.parametrize("handed_on", [False, True])
def test_kept_zero_buffer_that_grows_in_place(rt, handed_on):
    """The kept-zero bins are all zero at every size they grow to, at the same
    address or another, in a context that lives on and in the one that takes
    over its scratch."""
    ctx, bins, places = _create(rt), rt.t_bins(), []
    for nbytes in (1000, 1001, 5000, 5000, 200_000, 3_000_000):
        p, nonzero = _scratch(rt, ctx, bins, nbytes, zeroed=True)
        assert p and nonzero == 0, nbytes
        places.append(p)
        if handed_on:
            assert rt.ck_ctx_destroy(ctx) == 0
            ctx = _create(rt)
    assert len(set(places)) == 1  # it did come back where it was


def test_kept_scratch_is_given_back(rt):
    """A destroyed context's scratch is kept for the next one only while it is a
    small part of the memory left, and is freed by ck_ctx_trim, by the next set
    kept, and when an allocation fails without it."""
    MB = 1 << 20
    base, ctx = rt.t_in_use(), _create(rt)  # the device's own words stay allocated
    one = rt.t_in_use()
    base += 0 if base else one - 256  # (made by the first call)
    p, _ = _scratch(rt, ctx, 0, 4 * MB)
    assert rt.ck_ctx_destroy(ctx) == 0 and rt.t_in_use() >= base + 4 * MB  # kept
    ctx = _create(rt)
    assert _scratch(rt, ctx, 0, 3 * MB)[0] == p  # handed on
    assert rt.ck_ctx_destroy(ctx) == 0
    assert rt.ck_ctx_trim() == 0 and rt.t_in_use() == base
    assert rt.ck_ctx_trim() == 0 and rt.t_in_use() == base

    # 4 MB of scratch with less than 32 MB left is freed at once
    other = rt.t_malloc(30 * MB)
    ctx = _create(rt)
    _scratch(rt, ctx, 0, 4 * MB)
    assert rt.ck_ctx_destroy(ctx) == 0 and rt.t_in_use() == base + 30 * MB
    rt.t_free(other)

    # kept, and in the way of the library's own next allocation
    ctx, second = _create(rt), _create(rt)
    _scratch(rt, ctx, 0, 4 * MB)
    assert rt.ck_ctx_destroy(ctx) == 0 and rt.t_in_use() >= base + 4 * MB
    assert _scratch(rt, second, 0, 62 * MB)[0]
    assert rt.ck_ctx_destroy(second) == 0 and rt.t_in_use() == base


def test_host_allocation_that_fails_is_a_status(rt):
    """An exception of a host container ends as a status of the call, whose
    context is no longer the thread's."""
    ctx = _create(rt)
    p, _ = _scratch(rt, ctx, 0, 1000)
    assert rt.t_no_memory(ctx) == 4  # CK_ERR_OUT_OF_MEMORY
    rt.ck_last_error.restype = ctypes.c_char_p
    assert b"host memory" in rt.ck_last_error()
    assert _scratch(rt, 0, 0, 1000)[0] != p  # the default context's own
    assert _scratch(rt, ctx, 0, 1000)[0] == p
