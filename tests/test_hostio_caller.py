"""Staged host copies on the CPU, over a stand-in for the CUDA runtime: hostio.cu
is compiled as C++ against functions that carry a DMA out as late as its event
allows and note which thread made each call.

A stream handle may mean another stream in another thread (cudaStreamPerThread,
handle 2, does), and a caller's context need not be the one a helper thread would
get: every CUDA call of a copy has to be the calling thread's."""
from __future__ import annotations

import ctypes
import subprocess
import threading

import numpy as np
import pytest

from conftest import PKG, ROOT

MB = 1 << 20
FAKE = r'''
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
namespace gpupr {
struct Error;
void host_to_device(void*, const void*, size_t, cudaStream_t);
void device_to_host(void*, const void*, size_t, cudaStream_t);
void upload_topology(int32_t*, const void*, uint64_t, int64_t, int64_t, int, cudaStream_t);
}
namespace {
struct Op { void* dst; const void* src; size_t n; cudaEvent_t ev; };
std::mutex mu;
std::map<cudaStream_t, std::deque<Op>> queues;   // copies and events not carried out yet
std::map<cudaEvent_t, cudaStream_t> waiting;     // the queue an event is in
std::atomic<long> foreign{0}, calls{0}, dmas{0}, fail_at{-1};
thread_local bool caller = false;
cudaError_t note()
{
    if (!caller) ++foreign;
    return ++calls == fail_at ? cudaErrorUnknown : cudaSuccess;
}
void drain(cudaStream_t s, cudaEvent_t until)   // mu held
{
    auto& q = queues[s];
    while (!q.empty()) {
        Op o = q.front();
        q.pop_front();
        if (o.dst) std::memcpy(o.dst, o.src, o.n);
        if (o.ev) {
            auto w = waiting.find(o.ev);
            if (w != waiting.end()) waiting.erase(w);
            if (o.ev == until) return;
        }
    }
}
template <class F> int guarded(F f)
{
    caller = true;
    int rc = 0;
    try { f(); } catch (...) { rc = 1; }
    caller = false;
    return rc;
}
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return note(); }
cudaError_t cudaSetDevice(int) { return note(); }
cudaError_t cudaGetLastError() { note(); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::aligned_alloc(4096, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::aligned_alloc(4096, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*)
{
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s)
{
    const cudaError_t e = note();
    ++dmas;
    std::lock_guard<std::mutex> l(mu);
    if (e == cudaSuccess) queues[s].push_back({dst, src, n, nullptr});
    return e;
}
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t s)
{
    const cudaError_t e = note();
    std::lock_guard<std::mutex> l(mu);
    if (e == cudaSuccess) { queues[s].push_back({nullptr, nullptr, 0, ev}); waiting[ev] = s; }
    return e;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev)
{
    const cudaError_t e = note();
    std::lock_guard<std::mutex> l(mu);
    auto w = waiting.find(ev);
    if (w != waiting.end()) drain(w->second, ev);
    return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    const cudaError_t e = note();
    std::lock_guard<std::mutex> l(mu);
    drain(s, nullptr);
    return e;
}
long fake_foreign() { return foreign.exchange(0); }
long fake_calls() { return calls.exchange(0); }
long fake_dmas() { return dmas.exchange(0); }
void fake_fail_at(long n) { calls = 0; fail_at = n; }
int fake_h2d(void* d, const void* h, size_t n, void* s)
{ return guarded([&] { gpupr::host_to_device(d, h, n, (cudaStream_t)s); }); }
int fake_d2h(void* h, const void* d, size_t n, void* s)
{ return guarded([&] { gpupr::device_to_host(h, d, n, (cudaStream_t)s); }); }
int fake_topology(void* d, const void* h, uint64_t rows, int64_t rs, int64_t cs, int eb, void* s)
{ return guarded([&] { gpupr::upload_topology((int32_t*)d, h, rows, rs, cs, eb, (cudaStream_t)s); }); }
int fake_sync(void* s) { return guarded([&] { cudaStreamSynchronize((cudaStream_t)s); }); }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("hostio")
    (d / "fake.cpp").write_text(FAKE)
    out = d / "libhostio.so"
    inc = [f"-I{x}" for x in ("/usr/local/cuda/include", ROOT / "include", PKG / "csrc")]
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-Wno-attributes", *inc, "-x", "c++",
                           str(d / "fake.cpp"), str(PKG / "csrc" / "hostio.cu"), "-o", str(out), "-lpthread"])
    x = ctypes.CDLL(str(out))
    p, n, i = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int64
    for f in (x.fake_h2d, x.fake_d2h):
        f.argtypes = [p, p, n, p]
    x.fake_topology.argtypes = [p, p, ctypes.c_uint64, i, i, ctypes.c_int, p]
    x.fake_sync.argtypes = [p]
    x.fake_fail_at.argtypes = [ctypes.c_long]
    for f in (x.fake_foreign, x.fake_calls, x.fake_dmas):
        f.restype = ctypes.c_long
    return x


def data(n, seed):
    return np.random.default_rng(seed).integers(0, 256, n, dtype=np.uint8)


SIZES = [MB, 4 * MB - 1, 4 * MB, 11 * MB + 5, 32 * MB, 33 * MB + 7, 70 * MB + 48, 150 * MB + 3]


@pytest.mark.parametrize("nbytes", SIZES)
@pytest.mark.parametrize("stream", [0, 2, 77])
def test_copies_by_the_caller(lib, nbytes, stream):
    src = data(nbytes, nbytes)
    dev, back = np.zeros_like(src), np.zeros_like(src)
    lib.fake_foreign()
    assert lib.fake_h2d(dev.ctypes.data, src.ctypes.data, nbytes, stream) == 0
    want = src.copy()
    src[:] = 0   # the array has been read when the call returns
    lib.fake_sync(stream)
    assert np.array_equal(dev, want)
    assert lib.fake_d2h(back.ctypes.data, dev.ctypes.data, nbytes, stream) == 0
    assert np.array_equal(back, want)
    assert lib.fake_foreign() == 0


def layouts(rows, seed):
    rng = np.random.default_rng(seed)
    for bits in (4, 8):
        t = np.int32 if bits == 4 else np.int64
        a = rng.integers(-2**31 if bits == 4 else -2**62, 2**31 if bits == 4 else 2**62, (rows, 4), dtype=np.int64)
        a = a.astype(t)
        yield "C", a
        yield "F", np.asfortranarray(a)
        yield "reversed rows", a[::-1]
        yield "reversed columns", a[:, ::-1]
        yield "F reversed", np.asfortranarray(a)[::-1, ::-1]
        yield "wide rows", np.concatenate([a, a], 1)[:, 2:6]
        yield "every other column", np.repeat(a, 2, 1)[:, ::2]
        yield "F rows of a taller matrix", np.asfortranarray(np.concatenate([a, a, a, a]))[3:rows + 3]
        yield "broadcast row", np.broadcast_to(a[:1], (rows, 4))
        yield "broadcast column", np.broadcast_to(a[:, :1], (rows, 4))
        raw = np.zeros(a.nbytes + 3, np.uint8)
        raw[3:] = np.frombuffer(a.tobytes(), np.uint8)
        yield "unaligned", np.frombuffer(raw.data, t, rows * 4, 3).reshape(rows, 4)
        yield "unaligned F", np.frombuffer(raw.data, t, rows * 4, 3).reshape(4, rows).T


@pytest.mark.parametrize("rows", [1, 7, MB // 16, MB // 16 + 1, 5 * MB // 16 + 3, 40 * MB // 16 + 9])
def test_topology_by_the_caller(lib, rows):
    lib.fake_foreign()
    for name, a in layouts(rows, rows):
        out = np.full((rows, 4), -7, np.int32)
        assert lib.fake_topology(out.ctypes.data, a.ctypes.data, rows, a.strides[0], a.strides[1], a.itemsize, 2) == 0
        lib.fake_sync(2)
        assert np.array_equal(out, a.astype(np.int32)), (name, a.dtype)
    assert lib.fake_foreign() == 0


def test_threads(lib):
    """Copies of several threads at once, more of them than staging sets."""
    ok = []

    def one(k):
        src = data(45 * MB + k, k)
        dev, back = np.zeros_like(src), np.zeros_like(src)
        for _ in range(3):
            rc = lib.fake_h2d(dev.ctypes.data, src.ctypes.data, src.size, 100 + k)
            lib.fake_sync(100 + k)
            rc |= lib.fake_d2h(back.ctypes.data, dev.ctypes.data, src.size, 100 + k)
            ok.append(rc == 0 and np.array_equal(back, src))
            back[:] = 0

    t = [threading.Thread(target=one, args=(k,)) for k in range(6)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert ok == [True] * 18


def test_errors(lib):
    """A CUDA error anywhere in a copy comes back as the call's error, no helper
    works on after it, and the next copy is whole."""
    src = data(70 * MB + 48, 1)
    dev = np.zeros_like(src)
    for f, d, s in ((lib.fake_h2d, dev, src), (lib.fake_d2h, dev, src)):
        assert f(d.ctypes.data, s.ctypes.data, s.size, 5) == 0
        lib.fake_sync(5)
        lib.fake_calls()
        assert f(d.ctypes.data, s.ctypes.data, s.size, 5) == 0
        calls = lib.fake_calls()   # give or take which pieces share a DMA
        lib.fake_sync(5)
        for at in [2, 3, 4, 5, 6] + [calls * k // 10 for k in range(1, 9)]:
            lib.fake_fail_at(at)
            rc = f(d.ctypes.data, s.ctypes.data, s.size, 5)
            lib.fake_fail_at(-1)
            lib.fake_sync(5)
            assert rc == 1, at
            d[:] = 0
            assert f(d.ctypes.data, s.ctypes.data, s.size, 5) == 0
            lib.fake_sync(5)
            assert np.array_equal(d, s)
            d[:] = 0


def test_pieces_share_a_dma(lib):
    """Past its ends a large copy takes several pieces to a DMA."""
    src = data(150 * MB + 3, 2)
    dev = np.zeros_like(src)
    lib.fake_dmas()
    assert lib.fake_h2d(dev.ctypes.data, src.ctypes.data, src.size, 3) == 0
    lib.fake_sync(3)
    assert np.array_equal(dev, src) and lib.fake_dmas() < 151 // 2
    assert lib.fake_d2h(src.ctypes.data, dev.ctypes.data, src.size, 3) == 0
    assert np.array_equal(dev, src) and lib.fake_dmas() < 151 // 2
