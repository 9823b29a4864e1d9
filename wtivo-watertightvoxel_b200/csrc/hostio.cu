// hostio.cu -- copies between PAGEABLE host arrays and the device.
//
// The drop-in boundary takes numpy arrays (vertices, labels in; labels out),
// and the serving loop takes whole graphs from host memory.  A plain
// cudaMemcpyAsync from pageable memory goes through the driver's own staging
// at the speed of one host thread.  Here a copy is cut into 1 MiB pieces that
// rotate through a ring of pinned buffers: the calling thread and a small pool
// of host threads each take the next piece and copy it between the caller's
// array and its buffer, and the calling thread issues the DMAs between its own
// pieces, so host copies and DMA overlap and the copy runs near the PCIe rate.
// The threads are woken once per copy, one waking the next, and the caller starts
// at once: waking all of them for every 8 MiB chunk, and waiting for the slowest of
// them at its end, cost more than the copy itself up to tens of MB (that way ->
// now, in brackets the driver's own: 4 MB 0.6 -> 0.3 ms (0.25), 13 MB 1.5 -> 0.8
// (0.7), 34 MB 2.0 -> 1.6 (2.9), 102 MB 3.7 -> 3.7 (9.0), 400 MB 9.3 -> 9.2 (35);
// samples and labels of 5M tets to the host 1.6 -> 1.4, of 80M 31 -> 23).  Pinned
// source/destination arrays skip the staging.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "gpupr_internal.cuh"

namespace gpupr {
namespace {

constexpr size_t kPiece = 1u << 20;     // bytes per staging buffer
constexpr int kSlots = 32;              // staging buffers per set, side by side
constexpr int kGroup = 4;               // pieces one DMA takes in the middle of a copy
constexpr size_t kDirect = 1u << 20;    // below this, the driver's own path

// A copy's pieces, shared by its caller and the host threads that help it.  A
// helper works on host memory only: it takes the next piece, waits until its
// buffer is open, copies between the buffer and the caller's array and marks
// the piece done.  It makes no CUDA call: a stream handle may mean another
// stream in another thread (cudaStreamPerThread does), and the context current
// in the caller need not be the one a helper would get.
struct CopyJob {
    const std::function<void(char*, size_t, size_t)>* fill = nullptr;   // alive while a piece is taken
    char* pin = nullptr;
    int64_t parts = 0;
    size_t bytes = 0;
    std::atomic<int64_t> next{0};       // the next piece to take
    std::atomic<int64_t> open{0};       // pieces below it may be worked on
    std::atomic<int64_t> finished{0};   // pieces taken and worked on (or skipped)
    std::atomic<bool> stop{false};      // after an error: nothing more is copied
    std::atomic<int64_t> done[kSlots];  // p + 1 of the last piece done in a buffer

    CopyJob()
    {
        for (auto& d : done) d.store(0, std::memory_order_relaxed);
    }
    char* buffer(int64_t p) const { return pin + (size_t)(p % kSlots) * kPiece; }
    size_t offset(int64_t p) const { return (size_t)p * kPiece; }
    size_t length(int64_t p) const { return std::min(kPiece, bytes - offset(p)); }
    void finish(int64_t p)
    {
        done[p % kSlots].store(p + 1, std::memory_order_release);
        finished.fetch_add(1, std::memory_order_release);
    }
    void help()
    {
        for (;;) {
            const int64_t p = next.fetch_add(1);
            if (p >= parts) return;
            while (open.load(std::memory_order_acquire) <= p && !stop.load(std::memory_order_relaxed))
                std::this_thread::yield();
            if (!stop.load(std::memory_order_relaxed)) (*fill)(buffer(p), offset(p), length(p));
            finish(p);
        }
    }
};

// A fixed set of host worker threads that help the callers of copies.  Each
// job is its own object that workers pick up under the pool mutex, so a worker
// can never take a piece of a later job by mistake.
class CopyPool {
public:
    CopyPool()
    {
        int n = 8;
        if (const char* e = std::getenv("GPUPR_COPY_THREADS")) n = std::atoi(e);
        const unsigned hw = std::thread::hardware_concurrency();
        if (hw) n = std::min<int>(n, (int)hw / 2);
        n = std::max(0, std::min(n, 32));
        for (int i = 0; i < n; ++i) workers_.emplace_back([this] { work(); });
    }
    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();
    }

    // Sends up to `helpers` workers to the job; returns how many.
    int64_t enlist(const std::shared_ptr<CopyJob>& job, int64_t helpers)
    {
        const int64_t want = std::min(std::min((int64_t)workers_.size(), helpers), job->parts - 1);
        if (want <= 0) return 0;
        int64_t sent = 0;
        try {
            std::lock_guard<std::mutex> lk(mu_);
            for (; sent < want; ++sent) calls_.push_back(job);
        } catch (const std::bad_alloc&) {
            // fewer helpers: the caller does what they do not
        }
        cv_.notify_one();   // that thread wakes the next
        return sent;
    }

private:
    void work()
    {
        for (;;) {
            std::shared_ptr<CopyJob> job;
            bool more;
            {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [&] { return stop_ || !calls_.empty(); });
                if (stop_) return;
                job = std::move(calls_.front());
                calls_.pop_front();
                more = !calls_.empty();
            }
            if (more) cv_.notify_one();
            job->help();
        }
    }

    std::vector<std::thread> workers_;
    std::mutex mu_;
    std::condition_variable cv_;
    std::deque<std::shared_ptr<CopyJob>> calls_;   // one entry per thread a job may use
    bool stop_ = false;
};

CopyPool& copy_pool()
{
    static CopyPool* p = new CopyPool();   // lives for the process
    return *p;
}

struct Staging {
    std::mutex mu;
    char* pin = nullptr;
    cudaEvent_t ev[kSlots] = {};
    bool pending[kSlots] = {};   // a DMA of the buffer was issued ...
    int last[kSlots] = {};       // ... together with the next ones up to this, whose event it has
};

// Staging sets per device and direction (0 = to device, 1 = to host) that
// host threads can hold at the same time, so that copies issued by
// different threads (the server's two lanes, each uploading its own batch)
// run side by side instead of queueing on one set; each set is kSlots x
// kPiece pinned bytes, made on first use with its device current.
constexpr int kSets = 3;

// A staging set held by one copy until the lease goes out of scope.
struct StagingLease {
    Staging* st;
    std::unique_lock<std::mutex> lk;
};

// Takes a staging set of the current device for direction dir that no other
// copy holds; makes one while there are fewer than kSets, else waits for the
// first set.
StagingLease staging(int dir)
{
    static std::mutex mu;
    static std::map<std::pair<int, int>, std::vector<std::unique_ptr<Staging>>> all;
    int dev = 0;
    GPUPR_CUDA(cudaGetDevice(&dev));
    Staging* first = nullptr;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto& sets = all[{dev, dir}];
        for (auto& s : sets) {
            std::unique_lock<std::mutex> l(s->mu, std::try_to_lock);
            if (l.owns_lock()) return {s.get(), std::move(l)};
        }
        if ((int)sets.size() < kSets) {
            auto s = std::make_unique<Staging>();
            GPUPR_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&s->pin), kPiece * kSlots, cudaHostAllocPortable));
            for (int i = 0; i < kSlots; ++i)
                GPUPR_CUDA(cudaEventCreateWithFlags(&s->ev[i], cudaEventDisableTiming));
            std::unique_lock<std::mutex> l(s->mu);
            Staging* p = s.get();
            sets.push_back(std::move(s));
            return {p, std::move(l)};
        }
        first = sets.front().get();
    }
    return {first, std::unique_lock<std::mutex>(first->mu)};
}

// Waits for the copies a previous call left in flight (after an error, or
// the last chunks of a host-to-device copy) before the buffers are reused.
void settle(Staging& st)
{
    for (int k = 0; k < kSlots; ++k)
        if (st.pending[k]) {
            GPUPR_CUDA(cudaEventSynchronize(st.ev[st.last[k]]));
            st.pending[k] = false;
        }
}

bool is_pinned(const void* p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

// Host threads that help the caller with a memcpy through the staging: waking a
// sleeping thread costs about what copying 1 MiB does, so each has to bring
// several pieces' worth.  To the device, with 0 / 1 / 2 / 3 / 8 helpers at most: 34 MB
// 2.8 / 2.7 / 1.4 / 1.5 / 1.5 ms, 102 MB 8.3 / 7.9 / 3.3 / 3.0 / 3.8, 400 MB 33 / 18 /
// 11.5 / 9.1 / 9.2 (four: 2.9-3.4 and 8.5-11, by host).  A larger copy to the host
// meets pages of the caller's array that were never touched, which its threads
// fault in side by side: with a helper for 10 / 3 MB of it, samples and labels of 13M
// tets (52 + 13 MB) took 5.4 / 3.7 ms, of 5M 1.8 / 1.35, but of 3M 1.1 / 1.4 and of 2M
// 0.9 / 1.0.
int64_t copy_helpers(size_t bytes, bool to_host)
{
    const size_t each = to_host && bytes >= (16u << 20) ? 3u << 20 : 10u << 20;
    return bytes < (4u << 20) ? 0 : std::max<int64_t>(1, (int64_t)(bytes / each));
}

// Issues one DMA for the n pieces from p on, whose buffers lie side by side.
cudaError_t transfer(Staging& st, int64_t p, int64_t n, char* dev, size_t bytes, cudaMemcpyKind kind, cudaStream_t s)
{
    const int k = (int)(p % kSlots), last = k + (int)n - 1;
    const size_t off = (size_t)p * kPiece, len = std::min((size_t)n * kPiece, bytes - off);
    char* pin = st.pin + (size_t)k * kPiece;
    const cudaError_t e = kind == cudaMemcpyHostToDevice ? cudaMemcpyAsync(dev + off, pin, len, kind, s)
                                                         : cudaMemcpyAsync(pin, dev + off, len, kind, s);
    if (e != cudaSuccess) return e;
    for (int i = k; i <= last; ++i) {
        st.pending[i] = true;
        st.last[i] = last;
    }
    return cudaEventRecord(st.ev[last], s);
}

// Pieces that the next DMA, from piece p on, should wait for: single ones at the
// ends of a copy, where the link or the caller waits for each; groups between,
// because each DMA with its event costs the link time of its own (400 MB in
// single ones 10.2-10.6 ms, in groups of four 9.1-9.5, of eight 9.2-9.5).
int64_t group_at(int64_t p, int64_t parts)
{
    if (p < 2 * kGroup || parts - p <= 2 * kGroup) return 1;
    return std::min<int64_t>(kGroup, kSlots - p % kSlots);
}

// The caller works on a piece in this many bytes at a time, so that pieces its
// helpers have done wait for their DMA no longer than that.
constexpr size_t kCallerStep = 256u << 10;

// Runs a copy of `bytes` bytes, in pieces of kPiece,
// through a staging set: fill(pin, offset, length) copies between a buffer and
// the caller's array, on this thread or a helper's, once the buffer's last DMA is
// through; after(p, n) issues the DMA that follows the n pieces from p on, in order.
// All CUDA calls are this thread's.  After an error nothing more is copied and,
// once no helper works on the job, the error is thrown.
template <class After>
void run_pieces(Staging& st, size_t bytes, int64_t helpers,
                const std::function<void(char*, size_t, size_t)>& fill, const After& after)
{
    auto job = std::make_shared<CopyJob>();
    job->fill = &fill;
    job->pin = st.pin;
    job->bytes = bytes;
    const int64_t parts = job->parts = (int64_t)((bytes + kPiece - 1) / kPiece);
    cudaError_t err = cudaSuccess;
    int64_t passed = 0;   // pieces whose after() ran
    int64_t open = 0;     // job->open
    const int64_t ahead = 1 + copy_pool().enlist(job, helpers);   // pieces asked for at once
    auto pass = [&] {
        while (err == cudaSuccess && passed < parts) {
            const int64_t most = std::min(std::min<int64_t>(kGroup, kSlots - passed % kSlots), parts - passed);
            int64_t n = 0;
            while (n < most && job->done[(passed + n) % kSlots].load(std::memory_order_acquire) == passed + n + 1) ++n;
            if (n < group_at(passed, parts)) return;
            err = after(passed, n);
            passed += n;
        }
    };
    // a buffer opens when its last DMA is through: waited for only when a piece
    // in it is asked for, or may be next
    auto admit = [&] {
        const int64_t want = std::min(std::min(parts, passed + kSlots), job->next.load() + ahead);
        while (err == cudaSuccess && open < want) {
            const int k = (int)(open % kSlots);
            if (st.pending[k]) {
                err = cudaEventSynchronize(st.ev[st.last[k]]);
                if (err != cudaSuccess) return;
                st.pending[k] = false;
            }
            job->open.store(++open, std::memory_order_release);
        }
    };
    int64_t mine = -1;   // this thread's piece
    while (err == cudaSuccess && passed < parts) {
        pass();
        admit();
        if (mine < 0) mine = job->next.fetch_add(1);
        if (mine >= open || mine >= parts) {   // taken by others, or its buffer is not open yet
            std::this_thread::yield();
            continue;
        }
        const size_t off = job->offset(mine), len = job->length(mine);
        for (size_t b = 0; b < len && err == cudaSuccess; b += kCallerStep) {
            fill(job->buffer(mine) + b, off + b, std::min(kCallerStep, len - b));
            pass();
        }
        job->finish(mine);
        mine = -1;
    }
    if (err == cudaSuccess) return;
    // no helper may touch the caller's array or the buffers once this returns
    job->stop.store(true);
    const int64_t taken = std::min(parts, job->next.exchange(parts)) - (mine >= 0 && mine < parts ? 1 : 0);
    while (job->finished.load(std::memory_order_acquire) < taken) std::this_thread::yield();
    GPUPR_CUDA(err);
}

// Rows [row, row + n) of an Nx4 matrix of E (4- or 8-byte integers) at any byte
// strides, low 32 bits, as contiguous int32 rows.  Bound by the host's memory
// where several threads gather, by instructions where one does: the two orders that
// matrices come in have loops of their own that the compiler can vectorise (one
// loop with an element size and strides at run time -> now, on one thread: 30k
// rows of 64 bits 0.13 -> 0.06 ms, 60k 0.24 -> 0.12; on nine: 300k 0.75 -> 0.63,
// 3.2M 2.5 -> 1.9-2.3, row-major 3.0 -> 2.0-2.4; in 8 MiB chunks with the former loop
// 0.10, 0.11, 0.9, 1.9-2.2 and 2.3-2.9; one call after another: 3.2M 1.4-1.7, in
// chunks 2.1-2.3).
template <class E>
void gather_rows(int32_t* __restrict__ out, const char* base, int64_t row, int64_t n, int64_t row_stride,
                 int64_t col_stride)
{
    struct __attribute__((packed, may_alias)) Elem {   // numpy arrays may be unaligned
        E v;
    };
    const char* first = base + row * row_stride;
    if (row_stride == (int64_t)(4 * sizeof(E)) && col_stride == (int64_t)sizeof(E)) {   // row-major
        const Elem* in = reinterpret_cast<const Elem*>(first);
        for (int64_t i = 0; i < 4 * n; ++i) out[i] = (int32_t)(uint32_t)in[i].v;
        return;
    }
    if (row_stride == (int64_t)sizeof(E)) {   // column-major
        const Elem* a = reinterpret_cast<const Elem*>(first);
        const Elem* b = reinterpret_cast<const Elem*>(first + col_stride);
        const Elem* c = reinterpret_cast<const Elem*>(first + 2 * col_stride);
        const Elem* d = reinterpret_cast<const Elem*>(first + 3 * col_stride);
        for (int64_t r = 0; r < n; ++r) {
            out[4 * r] = (int32_t)(uint32_t)a[r].v;
            out[4 * r + 1] = (int32_t)(uint32_t)b[r].v;
            out[4 * r + 2] = (int32_t)(uint32_t)c[r].v;
            out[4 * r + 3] = (int32_t)(uint32_t)d[r].v;
        }
        return;
    }
    for (int64_t r = 0; r < n; ++r)
        for (int j = 0; j < 4; ++j)
            out[4 * r + j] = (int32_t)(uint32_t)reinterpret_cast<const Elem*>(first + r * row_stride + j * col_stride)->v;
}

}  // namespace

void host_to_device(void* d_dst, const void* h_src, size_t bytes, cudaStream_t s)
{
    if (!bytes) return;
    if (bytes < kDirect || is_pinned(h_src)) {
        GPUPR_CUDA(cudaMemcpyAsync(d_dst, h_src, bytes, cudaMemcpyHostToDevice, s));
        return;
    }
    StagingLease lease = staging(0);
    Staging& st = *lease.st;
    const char* src = static_cast<const char*>(h_src);
    char* dst = static_cast<char*>(d_dst);
    run_pieces(
        st, bytes, copy_helpers(bytes, false),
        [&](char* pin, size_t off, size_t len) { std::memcpy(pin, src + off, len); },
        [&](int64_t p, int64_t n) { return transfer(st, p, n, dst, bytes, cudaMemcpyHostToDevice, s); });
}

void device_to_host(void* h_dst, const void* d_src, size_t bytes, cudaStream_t s)
{
    if (!bytes) return;
    if (bytes < kDirect || is_pinned(h_dst)) {
        GPUPR_CUDA(cudaMemcpyAsync(h_dst, d_src, bytes, cudaMemcpyDeviceToHost, s));
        GPUPR_CUDA(cudaStreamSynchronize(s));
        return;
    }
    StagingLease lease = staging(1);
    Staging& st = *lease.st;
    settle(st);
    char* src = static_cast<char*>(const_cast<void*>(d_src));
    char* dst = static_cast<char*>(h_dst);
    const int64_t parts = (int64_t)((bytes + kPiece - 1) / kPiece);
    auto issue = [&](int64_t p, int64_t n) { return transfer(st, p, n, src, bytes, cudaMemcpyDeviceToHost, s); };
    // a ring of DMAs ahead; once pieces are copied out, those that follow in
    // their buffers are issued
    for (int64_t p = 0, n; p < std::min<int64_t>(parts, kSlots); p += n) {
        n = group_at(p, parts);
        GPUPR_CUDA(issue(p, n));
    }
    run_pieces(
        st, bytes, copy_helpers(bytes, true),
        [&](char* pin, size_t off, size_t len) { std::memcpy(dst + off, pin, len); },
        [&](int64_t p, int64_t n) {
            const int64_t q = p + kSlots;
            return q < parts ? issue(q, std::min(n, parts - q)) : cudaSuccess;
        });
}

// Nx4 integer topology (int32 or int64 elements, any byte strides, e.g. a
// Fortran-ordered matrix) -> contiguous int32 Nx4 on the device.  Rows are
// gathered piece by piece into the pinned staging by the host threads while
// earlier pieces are in flight; int64 values are narrowed the way numpy's
// astype(int32) narrows them (low 32 bits).
void upload_topology(int32_t* d_out, const void* host, uint64_t rows, int64_t row_stride,
                     int64_t col_stride, int elem_bytes, cudaStream_t s)
{
    if (!rows) return;
    if (elem_bytes == 4 && row_stride == 16 && col_stride == 4) {
        host_to_device(d_out, host, rows * 16u, s);
        return;
    }
    const char* base = static_cast<const char*>(host);
    StagingLease lease = staging(0);
    Staging& st = *lease.st;
    char* dst = reinterpret_cast<char*>(d_out);
    const size_t bytes = rows * 16u;
    // a strided gather costs several times a memcpy: a helper per piece
    run_pieces(
        st, bytes, (int64_t)((bytes + kPiece - 1) / kPiece),
        [&](char* pin, size_t off, size_t len) {   // multiples of a row's 16 bytes
            int32_t* out = reinterpret_cast<int32_t*>(pin);
            const int64_t row = (int64_t)(off / 16u), n = (int64_t)(len / 16u);
            if (elem_bytes == 8) gather_rows<uint64_t>(out, base, row, n, row_stride, col_stride);
            else gather_rows<uint32_t>(out, base, row, n, row_stride, col_stride);
        },
        [&](int64_t p, int64_t n) { return transfer(st, p, n, dst, bytes, cudaMemcpyHostToDevice, s); });
}

namespace {

struct ThreadRes {
    int device = -1;
    Ctl* ctl = nullptr;
    cudaEvent_t ev[8] = {};
    ~ThreadRes()
    {
        if (ctl) cudaFreeHost(ctl);
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
    }
};

ThreadRes& thread_res()
{
    thread_local std::vector<std::unique_ptr<ThreadRes>> all;
    int dev = 0;
    GPUPR_CUDA(cudaGetDevice(&dev));
    for (auto& r : all)
        if (r->device == dev) return *r;
    auto r = std::make_unique<ThreadRes>();
    r->device = dev;
    GPUPR_CUDA(cudaMallocHost(reinterpret_cast<void**>(&r->ctl), sizeof(Ctl)));
    for (cudaEvent_t& e : r->ev) GPUPR_CUDA(cudaEventCreate(&e));
    all.push_back(std::move(r));
    return *all.back();
}

}  // namespace

Ctl* pinned_ctl() { return thread_res().ctl; }

cudaEvent_t timing_event(int slot) { return thread_res().ev[slot & 7]; }

}  // namespace gpupr
