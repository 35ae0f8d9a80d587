/*
 * Copies between a caller's pageable arrays and the device.
 *
 * CUDA moves pageable memory through one thread: 11 GB/s up, and down into pages the
 * caller has just allocated (every result array of the Python package) 4-5 GB/s, most of it
 * the kernel clearing pages.  Here kThreads threads move parts of the copy, each through two
 * pinned chunks of its own, so that pages are cleared and chunks copied side by side while the
 * next ones cross the bus.  96 MB up 8.3 -> 3.3 ms, down into fresh pages 20 -> 5 ms; 14 MB 1.2
 * -> 0.6 and 3.0 -> 0.9; 2 MB down 0.9 -> 0.4 (16 host cores).
 *
 * A context of at least kContextBytes of state owns the pinned chunks, streams and events (2 ms
 * to allocate).  Its copies of kThreadedBytes or more go through the threads; smaller ones (3 MB
 * up 0.26 ms by plain copies, 0.33 by threads) only down into pages not yet there, from
 * kFreshBytes on (2 MB 0.9 -> 0.4 ms; into resident pages 0.14 by a plain copy).  Pinned arrays
 * are at the bus's speed already and take plain copies, as do smaller contexts.  On one CPU or
 * two the threads wait for one another, and only copies into absent pages gain: 14 MB up 0.87 ms
 * plain, by threads 1.25 on one CPU, 1.00 on two, 0.86 on three, 0.75 on four; 4 MB into absent
 * pages 2.2 plain, 1.4 on one CPU, 1.1 on two, 0.85 on three, 0.70 on four.
 */
#include <algorithm>
#include <cstring>
#include <new>
#include <thread>

#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include "dgr_internal.cuh"

namespace dgr {

namespace {
constexpr int kThreads = 4, kSlots = 2 * kThreads;
constexpr size_t kChunk = 512 << 10, kContextBytes = 4 << 20, kThreadedBytes = 6 << 20, kFreshBytes = 1 << 20;
}  // namespace

struct Stager {
    char *pinned; /* [kSlots][kChunk] */
    cudaStream_t stream[kThreads];
    cudaEvent_t done[kSlots], ready;
};

namespace {

/* chunk j of the copies: every copy is cut into chunks of its own */
struct Cut {
    const HostCopy *copy;
    size_t off, bytes;
};

size_t chunks_of(const HostCopy &p) { return (p.bytes + kChunk - 1) / kChunk; }

Cut cut_at(const HostCopy *p, size_t j)
{
    while (j >= chunks_of(*p)) j -= chunks_of(*p++);
    return {p, j * kChunk, std::min(kChunk, p->bytes - j * kChunk)};
}

/* chunks lo..hi-1 through thread t's slots; returns with all of them at their destination */
cudaError_t move_chunks(const Stager *st, int device, int t, const HostCopy *p, size_t lo, size_t hi, bool down)
{
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st->stream[t], st->ready, 0);
    const auto slot = [st, t](size_t j) { return st->pinned + (2 * t + (j & 1)) * kChunk; };
    const auto done = [st, t](size_t j) { return st->done[2 * t + (j & 1)]; };
    const auto land = [&](size_t j) { /* a chunk that has come down to its place in the caller's array */
        const Cut c = cut_at(p, j);
        const cudaError_t w = cudaEventSynchronize(done(j));
        if (w == cudaSuccess) memcpy((char *)c.copy->host + c.off, slot(j), c.bytes);
        return w;
    };
    for (size_t j = lo; j < hi && e == cudaSuccess; ++j) {
        const Cut c = cut_at(p, j);
        char *dev = (char *)c.copy->dev + c.off, *host = (char *)c.copy->host + c.off;
        if (down) {
            e = cudaMemcpyAsync(slot(j), dev, c.bytes, cudaMemcpyDeviceToHost, st->stream[t]);
            if (e == cudaSuccess) e = cudaEventRecord(done(j), st->stream[t]);
            if (e == cudaSuccess && j > lo) e = land(j - 1);
        } else {
            if (j >= lo + 2) e = cudaEventSynchronize(done(j)); /* the slot's previous chunk is up */
            if (e == cudaSuccess) memcpy(slot(j), host, c.bytes);
            if (e == cudaSuccess) e = cudaMemcpyAsync(dev, slot(j), c.bytes, cudaMemcpyHostToDevice, st->stream[t]);
            if (e == cudaSuccess) e = cudaEventRecord(done(j), st->stream[t]);
        }
    }
    if (down && hi > lo && e == cudaSuccess) e = land(hi - 1);
    const cudaError_t w = cudaStreamSynchronize(st->stream[t]);
    return e == cudaSuccess ? w : e;
}

bool is_pinned(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type != cudaMemoryTypeUnregistered;
}

/* whether more than an eighth of the arrays' pages (by eight looked at in each) are still to be
 * provided by the kernel: with a fifth of them absent threads gain already (4.5 MB down 0.75 ms
 * plain, 0.51 by threads, 0.63 on one CPU; a third absent 0.95, 0.63, 0.75), with none they do not */
bool are_fresh(const HostCopy *p, int n)
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    size_t absent = 0, total = 0;
    for (const HostCopy *q = p; q < p + n; ++q) {
        total += q->bytes;
        for (int i = 0; i < 8; ++i) {
            unsigned char in = 1;
            void *at = (void *)(((size_t)q->host + q->bytes / 8 * i + q->bytes / 16) / page * page);
            if (mincore(at, page, &in) == 0 && !(in & 1)) absent += q->bytes / 8;
        }
    }
    return absent > total / 8;
}

/* whether the calling thread, and so the threads it starts, may use enough CPUs for threads to
 * gain where no pages are cleared */
bool enough_cpus()
{
    cpu_set_t set;
    return sched_getaffinity(0, sizeof set, &set) != 0 || CPU_COUNT(&set) > kThreads / 2;
}

/* whether two copies have host bytes in common: copies down must then land in their order */
bool overlap(const HostCopy *p, int n)
{
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < i; ++j)
            if ((char *)p[i].host < (char *)p[j].host + p[j].bytes && (char *)p[j].host < (char *)p[i].host + p[i].bytes)
                return true;
    return false;
}

}  // namespace

void stager_release(dgr_ctx *c)
{
    Stager *st = c->stager;
    if (!st) return;
    for (cudaStream_t s : st->stream)
        if (s) cudaStreamDestroy(s);
    for (cudaEvent_t e : st->done)
        if (e) cudaEventDestroy(e);
    if (st->ready) cudaEventDestroy(st->ready);
    if (st->pinned) cudaFreeHost(st->pinned);
    delete st;
    c->stager = nullptr;
}

/* without one (no memory for it, or a small context) copies are plain */
void stager_create(dgr_ctx *c)
{
    const size_t state = (size_t)3 * c->nm * c->ne * sizeof(double);
    if (state < kContextBytes) return;
    Stager *st = new (std::nothrow) Stager();
    if (!st) return;
    c->stager = st;
    cudaError_t e = cudaHostAlloc((void **)&st->pinned, kSlots * kChunk, cudaHostAllocDefault);
    for (cudaStream_t &s : st->stream)
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
    for (cudaEvent_t &d : st->done)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&st->ready, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        cudaGetLastError();
        stager_release(c);
    }
}

cudaError_t host_copies(dgr_ctx *c, const HostCopy *p, int n, bool down)
{
    const Stager *st = c->stager;
    HostCopy threaded[kMaxHostCopies];
    int k = 0;
    size_t bytes = 0;
    const bool apart = st && !(down && overlap(p, n));
    for (int i = 0; i < n; ++i) {
        if (!p[i].bytes) continue;
        if (apart && p[i].bytes >= kFreshBytes / 8 && !is_pinned(p[i].host)) {
            threaded[k++] = p[i];
            bytes += p[i].bytes;
        }
    }
    const bool threads = (bytes >= kThreadedBytes && enough_cpus()) ||
                         (down && bytes >= kFreshBytes && are_fresh(threaded, k));
    for (int i = 0, j = 0; i < n; ++i) {
        if (!p[i].bytes) continue;
        if (j < k && threaded[j].host == p[i].host && threaded[j].dev == p[i].dev) {
            ++j;
            if (threads) continue;
        }
        const cudaError_t e = down ? cudaMemcpyAsync(p[i].host, p[i].dev, p[i].bytes, cudaMemcpyDeviceToHost, c->stream)
                                   : cudaMemcpyAsync(p[i].dev, p[i].host, p[i].bytes, cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return e;
    }
    if (!threads) return cudaSuccess;
    /* the threads' streams come after what this stream has been given so far */
    cudaError_t e = cudaEventRecord(st->ready, c->stream);
    if (e != cudaSuccess) return e;
    size_t total = 0;
    for (int i = 0; i < k; ++i) total += chunks_of(threaded[i]);
    const int T = (int)std::min<size_t>(kThreads, (total + 1) / 2);
    cudaError_t result[kThreads];
    std::thread th[kThreads];
    for (int t = 1; t < T; ++t) {
        const size_t lo = total * t / T, hi = total * (t + 1) / T;
        const auto part = [st, c, t, &threaded, lo, hi, down, &result] {
            result[t] = move_chunks(st, c->device, t, threaded, lo, hi, down);
        };
        try {
            th[t] = std::thread(part);
        } catch (...) { /* no thread to be had: its part is done here */
            part();
        }
    }
    result[0] = move_chunks(st, c->device, 0, threaded, 0, total / T, down);
    e = cudaSuccess;
    for (int t = 0; t < T; ++t) {
        if (th[t].joinable()) th[t].join();
        if (e == cudaSuccess) e = result[t];
    }
    return e;
}

}  // namespace dgr
