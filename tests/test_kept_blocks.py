"""The kept device blocks (csrc/resources.cuh) on the CPU, over a fake of the
CUDA calls that they use: what is kept stays within its limits, a block is
reused only where its last use is over, nothing is freed into a stream that is
being captured, and an allocation that fails gets everything that can be given
back.  The fake knows which blocks are out, which streams are captured, and how
much memory there is.
"""
import ctypes as C
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KEPT_BYTES, KEPT_BLOCKS = 2 << 30, 512
SHIM = r"""
#include "resources.cuh"
#include <set>
using namespace uaamg;
namespace {
std::unordered_map<void*, size_t> out;      // blocks the pool has given
std::set<cudaStream_t> captured;            // as cudaStreamIsCapturing sees it
size_t used = 0, total = ~size_t(0), next = 4096, streams = 256;
int bad_frees = 0, device_syncs = 0;
std::unordered_map<void*, cudaStream_t> freed;  // where each block last went back
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)++streams; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = captured.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { ++device_syncs; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMallocHost(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
    if (n > total - used) return cudaErrorMemoryAllocation;
    *p = (void*)(next += 4096);
    out[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
    bad_frees += captured.count(s) || !out.count(p);
    used -= out[p];
    out.erase(p);
    freed[p] = s;
    return cudaSuccess;
}
static DeviceCtx* ctx() { cudaError_t e; return device_ctx(&e); }
long k_stream() { cudaStream_t s; ctx_stream_acquire(ctx(), &s); return (long)s; }
long k_alloc(size_t n, long s) { void* p = nullptr; return ctx_dev_alloc(ctx(), &p, n, (cudaStream_t)s) == cudaSuccess ? (long)p : 0; }
int k_free(long p, long s, int idle) { return (int)ctx_dev_free(ctx(), (void*)p, (cudaStream_t)s, idle != 0); }
void k_captured(long s, int on) { if (on) captured.insert((cudaStream_t)s); else captured.erase((cudaStream_t)s); }
#ifndef NO_MARK
void* k_mark(long s) { return new CaptureMark(ctx(), (cudaStream_t)s); }
void k_unmark(void* m) { delete (CaptureMark*)m; }
#endif
void k_total(size_t n) { total = n; }
size_t k_used() { return used; }
size_t k_kept() { return ctx()->blocks_bytes; }
size_t k_blocks() { return ctx()->blocks.size(); }
long k_freed(long p) { return freed.count((void*)p) ? (long)freed[(void*)p] : -1; }
long k_free_stream() { return (long)ctx()->free_stream; }
int k_bad() { return bad_frees; }
int k_device_syncs() { return device_syncs; }
}
"""


@pytest.fixture
def k(tmp_path):
    src, lib = tmp_path / "shim.cpp", tmp_path / "shim.so"
    src.write_text(SHIM)
    nvcc = shutil.which(os.environ.get("NVCC", "nvcc")) or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fno-gnu-unique", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", cuda, "-I",
                    os.path.join(ROOT, "uaamg_b200", "csrc"), "-o", str(lib), str(src)], check=True)
    f = C.CDLL(str(lib))
    for name in ("k_stream", "k_alloc", "k_used", "k_kept", "k_blocks", "k_freed", "k_free_stream"):
        getattr(f, name).restype = C.c_size_t
    f.k_alloc.argtypes = [C.c_size_t, C.c_long]
    f.k_free.argtypes = [C.c_long, C.c_long, C.c_int]
    f.k_freed.argtypes = [C.c_long]
    f.k_captured.argtypes = [C.c_long, C.c_int]
    f.k_mark.argtypes, f.k_mark.restype, f.k_unmark.argtypes = [C.c_long], C.c_void_p, [C.c_void_p]
    f.k_total.argtypes = [C.c_size_t]
    yield f
    assert f.k_bad() == 0 and f.k_device_syncs() == 0


CALLER = 77  # a stream that the library did not make


def test_reuse_where_the_last_use_is_over(k):
    a, b = k.k_stream(), k.k_stream()
    p = k.k_alloc(1 << 20, a)
    k.k_free(p, a, 0)
    assert k.k_alloc(1 << 20, b) != p and k.k_alloc(1 << 20, CALLER) != p
    assert k.k_alloc((1 << 20) - 4096, a) == p  # in the order of the stream it was freed on
    k.k_free(p, a, 1)
    assert k.k_alloc(1 << 20, b) == p  # idle: anywhere
    kept = k.k_blocks()
    k.k_free(p, CALLER, 0)
    assert k.k_blocks() == kept  # a caller's stream: to the pool
    p = k.k_alloc(1 << 20, CALLER)
    k.k_free(p, CALLER, 1)
    assert k.k_blocks() == kept + 1 and k.k_alloc(1 << 20, a) == p


@pytest.mark.parametrize("seed,top", [(0, 1 << 16), (1, 1 << 27), (2, 1 << 30)])
def test_what_is_kept_is_bounded(k, seed, top):
    rng = random.Random(seed)
    streams = [k.k_stream() for _ in range(4)] + [0, CALLER]
    live = {}
    full = 0.0
    for _ in range(4000):
        if live and rng.random() < 0.5:
            p, n = rng.choice(list(live.items()))
            del live[p]
            k.k_free(p, rng.choice(streams), rng.random() < 0.5)
        else:
            n = int(2 ** rng.uniform(8, top.bit_length() - 1))
            p = k.k_alloc(n, rng.choice(streams))
            assert p and p not in live
            live[p] = n
        assert k.k_kept() <= KEPT_BYTES and k.k_blocks() <= KEPT_BLOCKS
        assert k.k_used() <= k.k_kept() + sum(max(1024, n + n // 4 + (2 << 20)) for n in live.values())
        full = max(full, k.k_kept() / KEPT_BYTES, k.k_blocks() / KEPT_BLOCKS)
    for p in list(live):
        k.k_free(p, streams[0], 1)
    assert k.k_kept() <= KEPT_BYTES and k.k_used() == k.k_kept()
    assert full > 0.1


@pytest.mark.parametrize("how", ["status", "mark"])
@pytest.mark.parametrize("idle", [0, 1])
def test_nothing_is_freed_into_a_capture(k, how, idle):
    """A stream freed blocks, went to another handle and is captured there while
    this thread's frees push the old blocks out."""
    a, b = k.k_stream(), k.k_stream()
    for p in [k.k_alloc(1 << 20, a) for _ in range(8)]:
        k.k_free(p, a, idle)
    mark = k.k_mark(a) if how == "mark" else None
    k.k_captured(a, 1 if how == "status" else 0)
    before = k.k_used()
    more = [k.k_alloc(n << 20, b) for n in (400, 401, 402, 403, 404, 405, 406)]
    for p in more:
        k.k_free(p, b, 0)
    assert k.k_bad() == 0 and k.k_kept() <= KEPT_BYTES
    if not idle:  # still there (the mark holds before the stream's status shows it)
        for _ in range(600):
            k.k_free(k.k_alloc(1 << 30, b), b, 0)
        assert k.k_used() >= before
    if mark:
        k.k_unmark(mark)
    k.k_captured(a, 0)
    for p in [k.k_alloc(n << 20, b) for n in (300, 301, 302, 303, 304, 305, 306)]:
        k.k_free(p, b, 0)
    assert k.k_kept() <= KEPT_BYTES


def test_an_allocation_that_fails_gets_what_is_kept(k):
    a, b, c = k.k_stream(), k.k_stream(), k.k_stream()
    blocks = [k.k_alloc(n << 20, s) for n, s in ((100, a), (101, b), (102, c), (103, CALLER))]
    for p, s, idle in zip(blocks, (a, b, c, CALLER), (0, 0, 1, 1)):
        k.k_free(p, s, idle)
    k.k_total(512 << 20)
    k.k_captured(b, 1)
    assert k.k_alloc(420 << 20, a) == 0  # b's block cannot go back now
    assert k.k_blocks() == 1
    k.k_captured(b, 0)
    assert k.k_alloc(420 << 20, a) != 0
    assert k.k_blocks() == 0


@pytest.mark.parametrize("idle", [0, 1])
@pytest.mark.parametrize("captured", [0, 1])
def test_where_blocks_go_back(k, captured, idle):
    """On the stream they were freed on, whose later allocations the pool can
    serve from them at once; an idle block of a captured stream or of a caller's
    on the stream kept for that."""
    a, b = k.k_stream(), k.k_stream()
    p, q = k.k_alloc(300 << 20, a), k.k_alloc(301 << 20, CALLER)
    k.k_free(p, a, idle)
    k.k_free(q, CALLER, 1)
    k.k_captured(a, captured)
    for r in [k.k_alloc((400 + i) << 20, b) for i in range(6)]:
        k.k_free(r, b, 0)
    assert k.k_freed(q) == k.k_free_stream()
    if not captured:
        assert k.k_freed(p) == a
    elif idle:
        assert k.k_freed(p) == k.k_free_stream()
    else:
        assert k.k_freed(p) == C.c_size_t(-1).value  # kept
