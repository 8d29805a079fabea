// capi.cu -- the C ABI of include/uegccd.h: contexts, batches and the solve drivers.
//
// A context is a batch of one system.  The drivers follow DrvMBPT (MP2.f90:11-157),
// DrvCCD (CCD.f90:18-183) and DrvdRPA (dRPA.f90:23-174): MP2 guess, then
// residual -> update -> convergence -> energy per iteration until max|dT| < TolMax
// or MaxIter, then one final residual for MaxRes.  All amplitudes, index maps,
// intermediates and the iteration's control stay on the device for the whole solve;
// the host reads a flag in its own memory, and (E, max|dT|, max|R|) of every solve at the end.
#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <deque>
#include <condition_variable>
#include <atomic>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/uegccd.h"
#include "kernels.h"
#include "plan.h"
#include "two_channel.h"
#include "uegccd_internal.h"

using namespace uegccd;

namespace {

thread_local std::string g_last_error;

// A persistent pool of host threads (one per core) for the parallel parts of batch creation
// and downloads: starting threads per call cost more than the work of a small batch.  Several
// callers (the creator threads of a pipelined host) share it.
class HostPool {
public:
    explicit HostPool(int n)
    {
        for (int k = 0; k < n; k++)
            th_.emplace_back([this]() {
                for (;;) {
                    std::function<void()> job;
                    {
                        std::unique_lock<std::mutex> lock(mu_);
                        cv_.wait(lock, [this]() { return stop_ || !q_.empty(); });
                        if (stop_ && q_.empty()) return;
                        job = std::move(q_.front());
                        q_.pop_front();
                    }
                    job();
                }
            });
    }
    ~HostPool()
    {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto &t : th_) t.join();
    }
    void post(std::function<void()> job)
    {
        {
            std::lock_guard<std::mutex> lock(mu_);
            q_.push_back(std::move(job));
        }
        cv_.notify_one();
    }

private:
    std::mutex mu_;
    std::condition_variable cv_;
    std::deque<std::function<void()>> q_;
    std::vector<std::thread> th_;
    bool stop_ = false;
};

HostPool &host_pool()
{
    static HostPool pool(std::max(1, (int)std::thread::hardware_concurrency()));
    return pool;
}

// Runs f(0..n-1) on the calling thread and up to nthreads - 1 pool threads; items are taken
// in turn from a shared counter, and each f(i) writes only its own outputs.
template <class F>
void parallel_for(int n, int nthreads, F f)
{
    if (nthreads <= 1 || n <= 1) {
        for (int i = 0; i < n; i++) f(i);
        return;
    }
    struct Shared {
        std::atomic<int> next{0};
        std::mutex mu;
        std::condition_variable cv;
        int finished = 0;
    } sh;
    const int helpers = std::min(nthreads, n) - 1;
    auto body = [&]() {
        for (int i; (i = sh.next.fetch_add(1)) < n;) f(i);
    };
    for (int k = 0; k < helpers; k++)
        host_pool().post([&]() {
            body();
            std::lock_guard<std::mutex> lock(sh.mu);
            if (++sh.finished == helpers) sh.cv.notify_one();
        });
    body();
    std::unique_lock<std::mutex> lock(sh.mu);
    sh.cv.wait(lock, [&]() { return sh.finished == helpers; });
}

int fail(int code, const std::string &msg)
{
    g_last_error = msg;
    return code;
}

#define CU(call)                                                                                       \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess)                                                                         \
            return fail(UEGCCD_ERR_CUDA, std::string(#call ": ") + cudaGetErrorString(e_));            \
    } while (0)

int check_device()
{
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0)
        return fail(UEGCCD_ERR_CUDA, std::string("no CUDA device: ") + cudaGetErrorString(e));
    int dev = 0;
    CU(cudaGetDevice(&dev));
    // one attribute query (cudaGetDeviceProperties reads every property: tens of ms per call)
    int major = 0;
    CU(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) {
        cudaDeviceProp p;
        CU(cudaGetDeviceProperties(&p, dev));
        return fail(UEGCCD_ERR_CUDA, std::string("the library is built for sm_100a (B200); device is ") + p.name);
    }
    return 0;
}

}  // namespace

// ----------------------------------------------------------------------------
// Batch: plans + device buffers of n systems
// ----------------------------------------------------------------------------
// Device memory of a batch: carved from chunks of at least kArenaChunk bytes. Chunks
// freed by a destroyed batch are kept in a small per-process cache (up to kPoolCap
// bytes) for the next batch; uegccd_trim_cache returns them to the driver.
namespace {
constexpr size_t kArenaChunk = 64ull << 20;
constexpr size_t kPoolCap = 32ull << 30;   // a 100-twist N=54 batch takes ~3 GB; pipelines keep 3-4 alive
struct DevChunk {
    char *p;
    size_t size;
    int dev;
};
// Page-locked host memory (portable: page-locked for every device's context).  Downloads take
// buffers that outlive the calls: any number of threads theirs, given back for the next call, until
// uegccd_trim_cache.  At most kPinnedCap bytes are locked at a time, idle or in use; past that a
// call goes on without one.  A buffer of more than about twice the size asked for stays where it
// is: a large one would be out of reach of the downloads it was made for.
constexpr size_t kPinnedCap = 512ull << 20;
constexpr size_t kPinnedMin = 64ull << 10;
struct PinnedBuf {
    char *p = nullptr;
    size_t bytes = 0;
};
std::mutex g_pinned_mu;
std::vector<PinnedBuf> g_pinned;   // idle, the longest idle first
size_t g_pinned_bytes = 0;         // locked, idle or in use

char *lock_host(size_t bytes)
{
    void *p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) == cudaSuccess) return (char *)p;
    cudaGetLastError();
    return nullptr;
}

// At least `bytes` > 0 (p = nullptr: past the cap, or the host has no more to lock).
PinnedBuf pinned_get(size_t bytes)
{
    PinnedBuf b;
    b.bytes = (bytes + kPinnedMin - 1) / kPinnedMin * kPinnedMin;
    std::vector<PinnedBuf> drop;
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        int best = -1;
        for (size_t k = 0; k < g_pinned.size(); k++)
            if (g_pinned[k].bytes >= bytes && g_pinned[k].bytes <= 2 * b.bytes &&
                (best < 0 || g_pinned[k].bytes < g_pinned[best].bytes))
                best = (int)k;
        if (best >= 0) {
            b = g_pinned[best];
            g_pinned.erase(g_pinned.begin() + best);
            return b;
        }
        while (g_pinned_bytes + b.bytes > kPinnedCap && !g_pinned.empty()) {   // idle ones make room
            drop.push_back(g_pinned.front());
            g_pinned_bytes -= g_pinned.front().bytes;
            g_pinned.erase(g_pinned.begin());
        }
        if (g_pinned_bytes + b.bytes > kPinnedCap) b.bytes = 0;
        g_pinned_bytes += b.bytes;
    }
    for (auto &x : drop) cudaFreeHost(x.p);
    if (b.bytes == 0 || (b.p = lock_host(b.bytes))) return b;
    std::lock_guard<std::mutex> lock(g_pinned_mu);
    g_pinned_bytes -= b.bytes;
    return PinnedBuf{};
}

void pinned_put(const PinnedBuf &b)
{
    if (!b.p) return;
    std::lock_guard<std::mutex> lock(g_pinned_mu);
    g_pinned.push_back(b);
}

// A buffer of one call, none for 0 bytes.  A call that returns early with copies in flight waits
// for them before another may have it.
struct PinnedScope {
    PinnedBuf b;
    cudaStream_t st;
    bool settled = false;   // no copy in flight
    PinnedScope(size_t bytes, cudaStream_t stream) : st(stream)
    {
        if (bytes > 0) b = pinned_get(bytes);
    }
    ~PinnedScope()
    {
        if (b.p && !settled) cudaStreamSynchronize(st);
        pinned_put(b);
    }
    PinnedScope(const PinnedScope &) = delete;
    PinnedScope &operator=(const PinnedScope &) = delete;
};

// Page-locked words an object keeps for its life (the flag of an iteration, small reads): kWords
// bytes each, cut from slabs of their own.
constexpr size_t kWords = 4096, kSlab = 64ull << 10;
constexpr size_t kFlagBytes = 64;   // of a batch's words: CtlBuffers::done, then the two-channel results
constexpr size_t kReadAt = kFlagBytes + kTcWords * sizeof(double);   // then small reads
std::vector<char *> g_slabs, g_words;   // slabs, and their free pieces (under g_pinned_mu)

char *words_get()
{
    std::lock_guard<std::mutex> lock(g_pinned_mu);
    if (g_words.empty()) {
        char *s = lock_host(kSlab);
        if (!s) return nullptr;
        g_slabs.push_back(s);
        for (size_t k = kSlab; k > 0; k -= kWords) g_words.push_back(s + k - kWords);
    }
    char *p = g_words.back();
    g_words.pop_back();
    return p;
}

void words_put(char *p)
{
    if (!p) return;
    std::lock_guard<std::mutex> lock(g_pinned_mu);
    g_words.push_back(p);
}

// The idle buffers and the slabs nothing uses, back to the host.
void pinned_trim()
{
    std::vector<char *> drop;
    {
        std::lock_guard<std::mutex> lock(g_pinned_mu);
        for (auto &b : g_pinned) {
            drop.push_back(b.p);
            g_pinned_bytes -= b.bytes;
        }
        g_pinned.clear();
        for (size_t k = 0; k < g_slabs.size();) {
            char *s = g_slabs[k];
            auto in = [s](char *w) { return w >= s && w < s + kSlab; };
            if (std::count_if(g_words.begin(), g_words.end(), in) < (int)(kSlab / kWords)) {
                k++;
                continue;
            }
            g_words.erase(std::remove_if(g_words.begin(), g_words.end(), in), g_words.end());
            g_slabs.erase(g_slabs.begin() + k);
            drop.push_back(s);
        }
    }
    for (char *p : drop) cudaFreeHost(p);
}

// Side streams and untimed events of destroyed batches, kept for the next batch of their device (at
// most kIdleForks sets and kIdleEvents events a process, until uegccd_trim_cache).  Making and destroying a set
// with each batch took 0.3-0.5 ms, as long as the rest of a small batch's making: 3 twists of N=14 made,
// solved and released, 1.42 -> 1.80 ms.
constexpr size_t kIdleForks = 32, kIdleEvents = 256;
template <class T>
struct Idle {
    int dev;
    T x;
};
std::mutex g_idle_mu;
std::vector<Idle<Fork>> g_forks;
std::vector<Idle<cudaEvent_t>> g_events;

template <class T>
bool idle_get(std::vector<Idle<T>> &v, int dev, T &x)
{
    std::lock_guard<std::mutex> lock(g_idle_mu);
    for (size_t k = v.size(); k-- > 0;)
        if (v[k].dev == dev) {
            x = v[k].x;
            v.erase(v.begin() + k);
            return true;
        }
    return false;
}
template <class T>
bool idle_put(std::vector<Idle<T>> &v, size_t most, int dev, const T &x)
{
    std::lock_guard<std::mutex> lock(g_idle_mu);
    if (v.size() >= most) return false;
    v.push_back(Idle<T>{dev, x});
    return true;
}

void fork_destroy(Fork &f)
{
    for (cudaEvent_t e : {f.start, f.staged})
        if (e) cudaEventDestroy(e);
    for (auto &e : f.done)
        if (e) cudaEventDestroy(e);
    for (auto &x : f.s)
        if (x) cudaStreamDestroy(x);
    f = Fork{};
}

// The side streams of a batch on device dev (current): a whole set, or none.
bool fork_get(Fork &f, int dev)
{
    if (idle_get(g_forks, dev, f)) return true;
    bool ok = cudaEventCreateWithFlags(&f.start, cudaEventDisableTiming) == cudaSuccess &&
              cudaEventCreateWithFlags(&f.staged, cudaEventDisableTiming) == cudaSuccess;
    for (int k = 0; k < kSideStreams; k++)
        ok = ok && cudaStreamCreateWithFlags(&f.s[k], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&f.done[k], cudaEventDisableTiming) == cudaSuccess;
    if (ok) return true;
    cudaGetLastError();
    fork_destroy(f);
    return false;
}

// Back for another batch; a set with work left on a stream, or one that a failed capture still
// holds, is destroyed.
void fork_put(Fork &f, int dev)
{
    if (!f.s[0]) return;
    bool ok = true;
    for (auto &x : f.s) {
        cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
        ok = ok && cudaStreamIsCapturing(x, &c) == cudaSuccess && c == cudaStreamCaptureStatusNone &&
             cudaStreamQuery(x) == cudaSuccess;
    }
    if (!ok) cudaGetLastError();
    if (!ok || !idle_put(g_forks, kIdleForks, dev, f)) fork_destroy(f);
}

cudaError_t event_get(cudaEvent_t &e, int dev)
{
    return idle_get(g_events, dev, e) ? cudaSuccess : cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
}

void event_put(cudaEvent_t e, int dev)
{
    if (e && !idle_put(g_events, kIdleEvents, dev, e)) cudaEventDestroy(e);
}

// The idle sets and events back to their devices.
void idle_trim()
{
    std::vector<Idle<Fork>> f;
    std::vector<Idle<cudaEvent_t>> e;
    {
        std::lock_guard<std::mutex> lock(g_idle_mu);
        f.swap(g_forks);
        e.swap(g_events);
    }
    for (auto &k : f) {
        DeviceScope scope(k.dev);
        fork_destroy(k.x);
    }
    for (auto &k : e) {
        DeviceScope scope(k.dev);
        cudaEventDestroy(k.x);
    }
}

bool is_pinned(const void *p)
{
    cudaPointerAttributes pa;
    const bool yes = cudaPointerGetAttributes(&pa, p) == cudaSuccess && pa.type == cudaMemoryTypeHost;
    if (!yes) cudaGetLastError();   // clear the query's status on older drivers
    return yes;
}

// memcpy, on the host's cores from kCoresMin bytes on, each a range of its own.  The destination's
// pages are often touched first here, and threads that fault pages in contend: three arrays of
// 2.7 MB take 0.35 ms by one thread and 0.9 ms by 16, of 28 MB 12 and 5 ms.
constexpr size_t kCoresMin = 8ull << 20;
void host_copy(char *dst, const char *src, size_t bytes, bool cores)
{
    if (!cores) {
        std::memcpy(dst, src, bytes);
        return;
    }
    const int nth = std::max(1, std::min(16, (int)std::thread::hardware_concurrency()));
    const size_t piece = (bytes + nth - 1) / nth;
    parallel_for(nth, nth, [&](int k) {
        const size_t a = (size_t)k * piece, e = std::min(bytes, a + piece);
        if (a < e) std::memcpy(dst + a, src + a, e - a);
    });
}
// g_pool_mu guards the cache, the per-device byte counts and the limit
std::mutex g_pool_mu;
std::vector<DevChunk> g_pool;
size_t g_pool_bytes = 0;
int64_t g_dev_bytes[kMaxDevices] = {};   // bytes the library holds from cudaMalloc per device (live + cached)
int64_t g_mem_limit = 0;                 // uegccd_set_memory_limit; 0: none

// Returns the cache of device dev to the driver (the caller holds no lock; dev is current).
void drop_cached(int dev)
{
    std::vector<DevChunk> drop;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        for (size_t k = 0; k < g_pool.size();)
            if (g_pool[k].dev == dev) {
                drop.push_back(g_pool[k]);
                g_pool_bytes -= g_pool[k].size;
                g_dev_bytes[dev % kMaxDevices] -= (int64_t)g_pool[k].size;
                g_pool.erase(g_pool.begin() + k);
            } else {
                k++;
            }
    }
    for (auto &c : drop) cudaFree(c.p);
}

// Device memory that makes a call faster and that it can do without, of one holder: kept between its
// calls, and given up then to an allocation that finds no room (under g_pool_mu).
struct SpareChunk {
    DevChunk c{nullptr, 0, -1};
    bool busy = false;
    size_t refused = 0;          // bytes there was no room for, at g_released
    uint64_t refused_at = 0;
};
uint64_t g_released = 0;              // how often memory was given back or the limit moved
std::vector<SpareChunk *> g_spares;   // those with a chunk

// Returns the idle spare chunks of device dev (-1: of all) to the driver, as drop_cached.
bool drop_spares(int dev)
{
    std::vector<DevChunk> drop;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        for (size_t k = 0; k < g_spares.size();) {
            SpareChunk &s = *g_spares[k];
            if (s.busy || (dev >= 0 && s.c.dev != dev)) {
                k++;
                continue;
            }
            drop.push_back(s.c);
            g_dev_bytes[s.c.dev % kMaxDevices] -= (int64_t)s.c.size;
            s.c = DevChunk{nullptr, 0, -1};
            g_released++;
            g_spares.erase(g_spares.begin() + k);
        }
    }
    for (auto &c : drop) {
        DeviceScope scope(c.dev);
        cudaFree(c.p);
    }
    return !drop.empty();
}

// True when `need` more bytes on dev stay within the limit (under g_pool_mu).
bool within_limit(int dev, size_t need)
{
    return g_mem_limit <= 0 || g_dev_bytes[dev % kMaxDevices] + (int64_t)need <= g_mem_limit;
}

// A chunk of at least `need` bytes on device dev (current): from the cache, else cudaMalloc.
// Past the memory limit, or when cudaMalloc fails, the device's cache goes back to the driver
// and the request is tried once more; then, unless it is for a spare chunk itself, with the idle spare
// chunks back too; then cudaErrorMemoryAllocation.
cudaError_t chunk_get(size_t need, int dev, DevChunk &out, bool spare = false)
{
    bool fits = true;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        int best = -1;
        for (size_t k = 0; k < g_pool.size(); k++)
            if (g_pool[k].dev == dev && g_pool[k].size >= need && g_pool[k].size <= 2 * need + kArenaChunk &&
                (best < 0 || g_pool[k].size < g_pool[best].size))
                best = (int)k;
        if (best >= 0) {
            out = g_pool[best];
            g_pool_bytes -= out.size;
            g_pool.erase(g_pool.begin() + best);
            return cudaSuccess;
        }
        fits = within_limit(dev, need);
    }
    if (!fits) {
        auto room = [&]() {
            std::lock_guard<std::mutex> lock(g_pool_mu);
            return within_limit(dev, need);
        };
        drop_cached(dev);
        if (!room() && (spare || !drop_spares(dev) || !room())) return cudaErrorMemoryAllocation;
    }
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, need);
    for (int k = 0; k < 2 && e != cudaSuccess; k++) {
        cudaGetLastError();
        if (k == 0) drop_cached(dev);
        else if (spare || !drop_spares(dev)) break;
        e = cudaMalloc(&p, need);
    }
    if (e == cudaSuccess) {
        out = DevChunk{(char *)p, need, dev};
        std::lock_guard<std::mutex> lock(g_pool_mu);
        g_dev_bytes[dev % kMaxDevices] += (int64_t)need;
    }
    return e;
}

// Straight back to the driver; c.dev is current.
void chunk_free(const DevChunk &c)
{
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        g_dev_bytes[c.dev % kMaxDevices] -= (int64_t)c.size;
        g_released++;
    }
    cudaFree(c.p);
}

// Back to the cache, or (past its cap) to the driver; c.dev is current.
void chunk_put(const DevChunk &c)
{
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        g_released++;
        if (g_pool_bytes + c.size <= kPoolCap) {
            g_pool.push_back(c);
            g_pool_bytes += c.size;
            return;
        }
        g_dev_bytes[c.dev % kMaxDevices] -= (int64_t)c.size;
    }
    cudaFree(c.p);
}

// The chunk of s for one call, at least `need` bytes on device dev (current): the one it has kept, else
// another (fresh = true), else none.
char *spare_hold(SpareChunk &s, size_t need, int dev, bool &fresh)
{
    DevChunk old{nullptr, 0, -1};
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        if (s.c.p && s.c.size >= need) {
            s.busy = true;
            fresh = false;
            return s.c.p;
        }
        if (s.refused > 0 && need >= s.refused && s.refused_at == g_released) return nullptr;
        if (s.c.p) {
            old = s.c;
            s.c = DevChunk{nullptr, 0, -1};
            g_spares.erase(std::find(g_spares.begin(), g_spares.end(), &s));
        }
    }
    if (old.p) chunk_put(old);
    DevChunk c;
    const bool found = chunk_get(need, dev, c, true) == cudaSuccess;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    s.refused = found ? 0 : need;   // not asked for again before memory was given back somewhere
    s.refused_at = g_released;
    if (!found) return nullptr;
    s.c = c;
    s.busy = true;
    g_spares.push_back(&s);
    fresh = true;
    return c.p;
}

void spare_rest(SpareChunk &s)
{
    std::lock_guard<std::mutex> lock(g_pool_mu);
    s.busy = false;
}

void spare_free(SpareChunk &s)
{
    DevChunk c{nullptr, 0, -1};
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        if (!s.c.p) return;
        c = s.c;
        s.c = DevChunk{nullptr, 0, -1};
        g_spares.erase(std::find(g_spares.begin(), g_spares.end(), &s));
    }
    chunk_put(c);
}
}  // namespace

struct UegccdBatch {
    int dev = -1;                    // the CUDA device the batch lives on (current at creation)
    bool broken = false;             // restoring the plain integral tables failed: calls are refused
    std::vector<SystemHost> sys;
    std::vector<SolvePlan> plans;
    std::vector<SolveDev> hsolves;
    DevBatch d;
    std::vector<DevChunk> chunks;    // device memory of the batch (see chunk_get): arena chunks
    size_t chunk_used = 0;           // bytes used in the last arena chunk
    std::vector<DevChunk> big;       // chunks of one large array each
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev_solve0 = nullptr, ev_solve1 = nullptr;
    char *words = nullptr;           // page-locked words (on first use; kFlagBytes, kReadAt)
    PinnedBuf pin;                   // where small reads land that the words do not hold
    cudaEvent_t ev_iter[2] = {nullptr, nullptr};            // the two latest iterations
    cudaEvent_t ev_copy[3] = {nullptr, nullptr, nullptr};   // arrays of a download (on first use)
    Fork fork;                       // side streams of a small batch's residual (on first use)
    bool fork_made = false;
    std::vector<double> red;         // host copy: 3 per solve
    std::vector<uint8_t> active;     // host copy
    double *dense = nullptr;         // reference-layout scratch: three arrays of the largest solve
    size_t dense_n = 0;
    double *dense_all = nullptr;     // reference layout of every solve, back to back (on first use)
    int64_t *dense_off = nullptr;
    size_t dense_all_n = 0;
    int launches = 0;
    int64_t h2d_bytes = 0, d2h_bytes = 0;   // host<->device traffic of the calls so far
    KernelTimer kt;
    bool kt_events = false;
    // device-side iteration control (allocated on first solve; DIIS history grows on demand)
    CtlBuffers ctl;
    int diis_cap = 0;
    std::vector<int> last_niter;     // iterations of each solve in the last solve call
    // an incremental solve (uegccd_batch_start / _advance): its options and which solves have
    // had their result released
    struct Session {
        bool on = false;
        UegccdOptions opt{};
        int drpa = 0, ndiis = 0, max_rec = 0;
        TermFlags f;
        std::vector<uint8_t> released;
    } ses;
    // CUDA graphs of one iteration, in FP64 and with the mixed-precision ladder (a mixed solve runs
    // both), each kept until other options or buffers are asked for
    struct GraphKey {
        int do_ring, do_xring, do_ladder, do_mosaic, drpa, ndiis, max_iter, mixed;
        double tol;
        bool operator==(const GraphKey &o) const
        {
            return do_ring == o.do_ring && do_xring == o.do_xring && do_ladder == o.do_ladder &&
                   do_mosaic == o.do_mosaic && drpa == o.drpa && ndiis == o.ndiis && max_iter == o.max_iter &&
                   mixed == o.mixed && tol == o.tol;
        }
    };
    struct IterGraph {
        GraphKey key{};
        cudaGraphExec_t exec = nullptr;
        bool valid = false;
        int launches = 0;            // kernels per iteration
    } graphs[2];
    void drop_graphs() { graphs[0].valid = graphs[1].valid = false; }
    bool tuned = false;              // launch shape picked (before the first graph capture)
    // structure factors (on first use): every solve's particle-hole groups {first row, rows},
    // solve s at [sf_g0[s], sf_g0[s+1]); one grid of the largest solve
    int2 *sf_groups = nullptr;
    std::vector<int> sf_g0;
    // integral options (CoreN, GapII) in force, and the unfiltered |q|^2 tables of all solves
    int core_n = 0;
    double gapii = 0.0;
    std::vector<double> vtab_base;
    // range-separated integrals with one flag for every CCD term (uegccd_*_set_range)
    int range_flag = 0;
    double screening = 0.0;
    // batch solves in the two-channel form (do_ring != do_xring): one two_channel.cu state per
    // system, made on first use; each solve's iteration table; two_channel_amps: the batch's
    // amplitudes hold T2abab of such a solve (the spin relation does not give T2abba)
    std::vector<std::unique_ptr<uegccd::TwoChannel>> tcs;
    std::vector<std::vector<double>> tc_en, tc_dt;
    SpareChunk tc_work;              // the workspace their matrix-product form shares
    const void *tc_work_user = nullptr;   // the state that used it last
    bool two_channel_amps = false;
    double *sf_grid = nullptr;
    int *sf_err = nullptr;

    ~UegccdBatch()
    {
        for (auto &g : graphs)
            if (g.exec) cudaGraphExecDestroy(g.exec);
        if (kt_events)
            for (auto &e : kt.ev) cudaEventDestroy(e);
        if (stream) cudaStreamSynchronize(stream);
        spare_free(tc_work);
        for (auto &c : chunks) chunk_put(c);
        for (auto &c : big) chunk_put(c);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (ev_solve0) cudaEventDestroy(ev_solve0);
        if (ev_solve1) cudaEventDestroy(ev_solve1);
        pinned_put(pin);
        words_put(words);
        for (auto &e : ev_iter) event_put(e, dev);
        for (auto &e : ev_copy) event_put(e, dev);
        fork_put(fork, dev);
        if (stream) cudaStreamDestroy(stream);
    }

    template <class T>
    int alloc(T *&p, size_t n)
    {
        p = nullptr;
        if (n == 0) n = 1;
        const size_t bytes = (n * sizeof(T) + 255) & ~(size_t)255;
        if (bytes >= kArenaChunk / 2) {
            // large arrays get a chunk of their own, of exactly the size they need
            DevChunk c;
            cudaError_t e = chunk_get(bytes, dev, c);
            if (e != cudaSuccess)
                return fail(UEGCCD_ERR_ALLOC, std::string("device allocation of ") + std::to_string(bytes) +
                                                  " bytes: " + cudaGetErrorString(e));
            big.push_back(c);
            p = reinterpret_cast<T *>(c.p);
            return 0;
        }
        if (chunks.empty() || chunk_used + bytes > chunks.back().size) {
            DevChunk c;
            cudaError_t e = chunk_get(kArenaChunk, dev, c);
            if (e != cudaSuccess)
                return fail(UEGCCD_ERR_ALLOC, std::string("device allocation of ") + std::to_string(kArenaChunk) +
                                                  " bytes: " + cudaGetErrorString(e));
            chunks.push_back(c);
            chunk_used = 0;
        }
        p = reinterpret_cast<T *>(chunks.back().p + chunk_used);
        chunk_used += bytes;
        return 0;
    }
    // Allocation marks: rollback(mark()) returns every chunk taken since the mark to the driver
    // (not to the cache: a failed group of allocations means memory is short) and the arena
    // space carved since -- the batch is left as it was (arena chunks are only ever appended,
    // so the mark's last one is the last one again).
    struct Mark {
        size_t nchunks, nbig, used;
    };
    Mark mark() const { return Mark{chunks.size(), big.size(), chunk_used}; }
    void rollback(const Mark &m)
    {
        while (big.size() > m.nbig) {
            chunk_free(big.back());
            big.pop_back();
        }
        while (chunks.size() > m.nchunks) {
            chunk_free(chunks.back());
            chunks.pop_back();
        }
        chunk_used = m.used;
    }
    template <class T>
    int upload(T *&p, const std::vector<T> &h)
    {
        int rc = alloc(p, h.size());
        if (rc) return rc;
        if (!h.empty()) CU(cudaMemcpyAsync(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, stream));
        h2d_bytes += (int64_t)(h.size() * sizeof(T));
        return 0;
    }
};

struct UegccdCtx {
    std::unique_ptr<UegccdBatch> batch;
    // the two-channel form (two_channel.cu), made on first use, and the integral selection of
    // uegccd_ctx_set_eri
    std::unique_ptr<uegccd::TwoChannel> tc;
    bool eri_set = false;
    UegccdRangeTerms flags{};
    int safe_eri = 0;
    double screening = 0.0;
};

namespace {

int read_system(const UegccdSystem *s, SystemHost &h)
{
    if (!s || !s->eigen || !s->nvec) return fail(UEGCCD_ERR_ARG, "null system or array");
    if (s->nocc <= 0 || s->nao <= s->nocc) return fail(UEGCCD_ERR_ARG, "need 0 < NOcc < NAO");
    if (!(s->L > 0)) return fail(UEGCCD_ERR_ARG, "L must be positive");
    h.O = s->nocc;
    h.M = s->nao;
    h.L = s->L;
    h.madelung = s->madelung;
    h.eigen.assign(s->eigen, s->eigen + s->nao);
    h.n.resize(s->nao);
    for (int p = 0; p < s->nao; p++)
        for (int d = 0; d < 3; d++) h.n[p][d] = s->nvec[p + (size_t)s->nao * d];
    return 0;
}

// UEGCCD_TRACE=1 in the environment: batch creation prints its phase times to stderr.
struct PhaseTrace {
    bool on = false;
    std::chrono::steady_clock::time_point t0, last;
    std::string line;
    PhaseTrace()
    {
        const char *e = std::getenv("UEGCCD_TRACE");
        on = e && e[0] == '1';
        t0 = last = std::chrono::steady_clock::now();
    }
    void mark(const char *what)
    {
        if (!on) return;
        const auto now = std::chrono::steady_clock::now();
        char buf[96];
        std::snprintf(buf, sizeof buf, " %s %.2f", what, std::chrono::duration<double, std::milli>(now - last).count());
        line += buf;
        last = now;
    }
    ~PhaseTrace()
    {
        if (on)
            std::fprintf(stderr, "uegccd batch create (ms):%s total %.2f\n", line.c_str(),
                         std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
    }
};

// The FP64 ladder's tiles (ladder.cu), form by form, those of one row count together (they run the
// same code: CTAs of different ones evict each other's instructions) and the longest first, so
// that the last wave is short.  A block of up to 4 rows is one tile (or one per 256 columns); a larger one is cut into
// row tiles of at most 16, and those into column tiles of so many passes that the batch makes at
// least about four tiles per SM -- every column tile forms the block's H again, so a large batch
// keeps a row tile whole.
std::vector<LadderTile64> ladder_tiles(const std::vector<BlockDev> &blocks, const std::vector<SolveDev> &solves,
                                       int (&count)[2], int &max_rows)
{
    constexpr int kSms = 148;
    int64_t passes = 0;
    auto row_tiles = [](int rows) { return (rows + kLadderMmaRows - 1) / kLadderMmaRows; };
    for (const auto &B : blocks) {
        const int rows = B.nd + B.dg, h = B.nvd + B.sd;
        max_rows = std::max(max_rows, rows);
        if (rows <= kLadderFmaRows) continue;
        const int nt = row_tiles(rows), pc = ladder_pass_cols((rows + nt - 1) / nt);
        passes += (int64_t)nt * ((h + rows + pc - 1) / pc);
    }
    const int per_tile = (int)std::max<int64_t>(1, std::min<int64_t>(passes / (4 * kSms), 1 << 16));
    std::vector<LadderTile64> tiles[2];
    std::vector<std::pair<float, int>> cost[2];
    for (const BlockDev &B : blocks) {
        const int rows = B.nd + B.dg, h = B.nvd + B.sd;
        const SolveDev &S = solves[B.solve];
        const int f = rows <= kLadderFmaRows ? 0 : 1, nt = f ? row_tiles(rows) : 1, np = (rows + nt - 1) / nt;
        const int w = (f ? per_tile * ladder_pass_cols(np) : kLadderFmaCols) - rows;
        for (int p0 = 0; p0 < rows; p0 += np)
            for (int a0 = 0; a0 < h; a0 += w) {
                const int a1 = std::min(h, a0 + w), n = std::min(np, rows - p0);
                cost[f].emplace_back((f ? (n <= 8 ? 0 : 1) : rows) * 1e7f + (float)h * ((rows + a1 - a0 + 31) / 32),
                                     (int)tiles[f].size());
                tiles[f].push_back(LadderTile64{(int)B.t0, B.vir0, B.pair0, S.vtab0, B.solve, S.q2max, a0, a1, B.v,
                                                B.nvd, B.sd, B.nd, B.dg, p0, n, 0});
            }
    }
    std::vector<LadderTile64> out;
    out.reserve(tiles[0].size() + tiles[1].size());
    for (int f = 0; f < 2; f++) {
        std::sort(cost[f].begin(), cost[f].end(), [](const auto &x, const auto &y) {
            return x.first != y.first ? x.first > y.first : x.second < y.second;
        });
        for (const auto &c : cost[f]) out.push_back(tiles[f][c.second]);
        count[f] = (int)tiles[f].size();
    }
    return out;
}

int build_batch(const UegccdSystem *systems, int n, std::unique_ptr<UegccdBatch> &out)
{
    PhaseTrace trace;
    int rc = check_device();
    if (rc) return rc;
    if (n <= 0) return fail(UEGCCD_ERR_ARG, "empty batch");
    auto b = std::make_unique<UegccdBatch>();
    CU(cudaGetDevice(&b->dev));   // the batch lives on the device current now
    b->sys.resize(n);
    b->plans.resize(n);
    for (int s = 0; s < n; s++) {
        rc = read_system(&systems[s], b->sys[s]);
        if (rc) return rc;
    }
    // plans of different systems are independent: build them on parallel host threads
    const int nthreads = std::max(1, std::min(n, (int)std::thread::hardware_concurrency()));
    std::vector<std::string> msgs(n);
    parallel_for(n, nthreads, [&](int s) { msgs[s] = build_solve_plan(b->sys[s], b->plans[s]); });
    for (int s = 0; s < n; s++) {
        if (!msgs[s].empty()) return fail(UEGCCD_ERR_ARG, "system " + std::to_string(s) + ": " + msgs[s]);
        if (b->plans[s].O > 64) return fail(UEGCCD_ERR_UNSUPPORTED, "NOcc > 64 is outside the hole-hole ladder tiling");
        for (const auto &v : b->sys[s].n)
            if (std::abs(v[0]) > 63 || std::abs(v[1]) > 63 || std::abs(v[2]) > 63)
                return fail(UEGCCD_ERR_UNSUPPORTED, "system " + std::to_string(s) +
                                                        ": a plane-wave component beyond +-63 (the kernels take "
                                                        "momentum differences as signed bytes)");
    }
    trace.mark("plans");
    CU(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    CU(cudaEventCreate(&b->ev0));
    CU(cudaEventCreate(&b->ev1));
    CU(cudaEventCreate(&b->ev_solve0));
    CU(cudaEventCreate(&b->ev_solve1));
    trace.mark("stream");

    std::vector<SolveDev> solves(n);
    std::vector<BlockDev> blocks;
    std::vector<LadderTile> tc16, tc32, tc64;
    std::vector<TcTileDev> tcx16, tcx32, tcx64;   // beside tc16/32/64: FP16 operand offsets
    std::vector<WSlabDev> wslabs;
    std::vector<DTileDev> dtiles;
    int64_t w16_n = 0, d16_n = 0;
    int nscale = 0;
    // the large host tables live in vectors kept per creating thread between creates: a
    // fresh allocation would page-fault on first touch, which cost more than filling them
    struct HostTables {
        std::vector<ChunkDev> chunks, rchunks;
        std::vector<int2> targets;
        std::vector<int16_t> pair_i, pair_j, vir, pcol, ph_i, ph_x;
        std::vector<int4> nv4;
        std::vector<int> nvp;
        std::vector<double> eigen;
    };
    static thread_local HostTables ht;
    auto &chunks = ht.chunks, &rchunks = ht.rchunks;
    auto &targets = ht.targets;
    auto &pair_i = ht.pair_i, &pair_j = ht.pair_j, &vir = ht.vir;
    auto &pcol = ht.pcol;   // beside vir: the partner's column in the same block
    auto &nv4 = ht.nv4;
    auto &nvp = ht.nvp;     // beside nv4: packed a component per byte
    auto &eigen = ht.eigen;
    auto &ph_i = ht.ph_i, &ph_x = ht.ph_x;
    for (auto *v : {&chunks, &rchunks}) v->clear();
    targets.clear();
    for (auto *v : {&pair_i, &pair_j, &vir, &pcol, &ph_i, &ph_x}) v->clear();
    nv4.clear();
    nvp.clear();
    eigen.clear();
    std::vector<double> vtab;
    std::vector<RingPairDev> rpairs, spairs;
    int64_t amp0 = 0, pos0 = 0, ph0 = 0, phr0 = 0, mrows = 0, mcols = 0;
    std::vector<int> s_t0(n);   // first mosaic target of each solve
    int orb0 = 0, vtab0 = 0, jvv0 = 0, joo0 = 0, max_o = 0, max_v = 0, max_occ = 0;
    // offsets of each solve in the large concatenated arrays (filled in parallel below)
    std::vector<int64_t> s_phr0(n);
    for (int s = 0; s < n; s++) {
        const SolvePlan &P = b->plans[s];
        const SystemHost &H = b->sys[s];
        SolveDev &S = solves[s];
        S.O = P.O; S.V = P.V; S.M = P.M;
        S.nblk = (int)P.blocks.size();
        S.blk0 = (int)blocks.size();
        S.orb0 = orb0;
        S.vtab0 = vtab0;
        S.q2max = P.q2max;
        S.amp0 = amp0;
        S.namp = (int32_t)P.namp;
        S.core_n = 0;
        S.pos0 = pos0;
        S.ph0 = ph0;
        S.jvv0 = jvv0;
        S.joo0 = joo0;
        S.denom_factor = 2.0;
        S.phr0 = phr0;
        max_occ = std::max(max_occ, P.O);
        s_phr0[s] = phr0;
        for (size_t gi = 0; gi < P.groups.size(); gi++) {
            const auto &G = P.groups[gi];
            if (G.partner < 0 || G.partner < (int)gi) continue;  // each {Q, -Q} once
            const auto &H2 = P.groups[G.partner];
            // the smaller group first: k_rings gathers and multiplies from its side
            if (G.n <= H2.n) rpairs.push_back(RingPairDev{s, G.r0, G.n, H2.r0, H2.n, 0});
            else rpairs.push_back(RingPairDev{s, H2.r0, H2.n, G.r0, G.n, 0});
        }
        for (const auto &B : P.blocks) {
            BlockDev bd;
            bd.solve = s; bd.o = B.o; bd.v = B.v;
            bd.pair0 = (int)pair_i.size() + B.pair0;
            bd.vir0 = (int)vir.size() + B.vir0;
            bd.t0 = amp0 + B.t0;
            bd.nd = B.nd;
            bd.dg = B.dg;
            bd.nvd = B.nvd;
            bd.sd = B.sd;
            bd.row0 = mrows;
            bd.col0 = mcols;   // shifted past all rows below
            mrows += B.o;
            mcols += B.v;
            int bi = (int)blocks.size();
            blocks.push_back(bd);
            max_o = std::max(max_o, B.o);
            max_v = std::max(max_v, B.v);
            const int oc = B.nd + B.dg;
            // tensor-core tiles: 128 virtuals x (16, 32 or 64) rows over the rows i <= j (the
            // update reads G there only); their FP16 operands: one Coulomb slab per 128
            // virtuals, one d tile per row tile, each over all K chunks
            const int ntc = oc <= 16 ? 16 : oc <= 32 ? 32 : 64;
            auto &tl = ntc == 16 ? tc16 : ntc == 32 ? tc32 : tc64;
            auto &tx = ntc == 16 ? tcx16 : ntc == 32 ? tcx32 : tcx64;
            const int64_t nch = (B.v + 31) / 32;
            const int64_t w0 = w16_n, d0 = d16_n;
            const int s0 = nscale;
            for (int a0 = 0; a0 < B.v; a0 += 128) {
                wslabs.push_back(WSlabDev{bi, a0, w16_n});
                w16_n += nch * 128 * 32;
            }
            for (int p0 = 0; p0 < oc; p0 += ntc) {
                dtiles.push_back(DTileDev{bi, p0, ntc, nscale, d16_n});
                d16_n += nch * ntc * 32;
                nscale += ntc;
            }
            for (int a0 = 0; a0 < B.v; a0 += 128)
                for (int p0 = 0; p0 < oc; p0 += ntc) {
                    tl.push_back(LadderTile{bi, a0, p0, ntc});
                    const int it = p0 / ntc;
                    tx.push_back(TcTileDev{w0 + (a0 / 128) * nch * 128 * 32, d0 + it * nch * ntc * 32, s0 + it * ntc, 0});
                }
        }
        pair_i.insert(pair_i.end(), P.pair_i.begin(), P.pair_i.end());
        pair_j.insert(pair_j.end(), P.pair_j.begin(), P.pair_j.end());
        vir.insert(vir.end(), P.vir.begin(), P.vir.end());
        pcol.insert(pcol.end(), P.pcol.begin(), P.pcol.end());
        for (int p = 0; p < P.M; p++) {
            nv4.push_back(make_int4(H.n[p][0], H.n[p][1], H.n[p][2], 0));
            nvp.push_back((H.n[p][0] & 0xff) | ((H.n[p][1] & 0xff) << 8) | ((H.n[p][2] & 0xff) << 16));
        }
        eigen.insert(eigen.end(), H.eigen.begin(), H.eigen.end());
        vtab.insert(vtab.end(), P.vtab.begin(), P.vtab.end());
        for (int64_t st = 0; st < P.namp; st += kChunk) chunks.push_back(ChunkDev{s, (int32_t)st});
        for (int64_t st = 0; st < P.ring_entries; st += kChunk) rchunks.push_back(ChunkDev{s, (int32_t)st});
        s_t0[s] = (int)targets.size();
        for (int x = 0; x < P.V + P.O; x++) targets.push_back(make_int2(s, x));
        amp0 += P.namp;
        pos0 += (int64_t)P.O * P.O * P.V;
        ph0 += P.ring_entries;
        orb0 += P.M;
        vtab0 += P.q2max + 1;
        jvv0 += P.V;
        joo0 += P.O;
        phr0 += (int64_t)P.O * P.V;
        if (amp0 >= ((int64_t)1 << 31)) return fail(UEGCCD_ERR_ARG, "batch too large for 32-bit packed indices");
    }
    // tiles of the amplitudes i <= j: each block's rows up to its diagonal pair
    std::vector<UTileDev> utiles;
    std::vector<int> utile_begin(n + 1, 0);
    for (const auto &bd : blocks) {
        const SolveDev &S = solves[bd.solve];
        struct Emit {
            std::vector<UTileDev> *out;
            UTileDev base;
        } em{&utiles, UTileDev{(int)bd.t0, bd.vir0, bd.pair0, bd.solve, S.orb0, S.vtab0, S.jvv0, S.joo0, (int)S.phr0,
                               S.q2max, bd.v, bd.nvd, (int16_t)bd.sd, (int16_t)bd.dg, (int16_t)bd.nd, 0, 0, 0, 0,
                               (int16_t)S.O, S.V, {0, 0, 0}}};
        update_tiles(bd.nd + bd.dg, bd.nvd + bd.sd,
                     [](void *to, int c0, int nc, int r0, int nr) {
                         auto *e = static_cast<Emit *>(to);
                         UTileDev t = e->base;
                         t.c0 = (int16_t)c0;
                         t.nc = (int16_t)nc;
                         t.r0 = (int16_t)r0;
                         t.nr = (int16_t)nr;
                         e->out->push_back(t);
                     },
                     &em);
        utile_begin[bd.solve + 1] = (int)utiles.size();
    }
    for (int s = 0; s < n; s++) utile_begin[s + 1] = std::max(utile_begin[s + 1], utile_begin[s]);
    trace.mark("solve-loop");
    ph_i.resize(phr0);
    ph_x.resize(phr0);
    parallel_for(n, nthreads, [&](int s) {
        const SolvePlan &P = b->plans[s];
        std::copy(P.ph_i.begin(), P.ph_i.end(), ph_i.begin() + s_phr0[s]);
        std::copy(P.ph_x.begin(), P.ph_x.end(), ph_x.begin() + s_phr0[s]);
    });

    // mosaic targets: Jvv(c) adds the column sums of c over the blocks holding it, Joo(k)
    // the row sums of the pairs (k, l); both in block order
    for (auto &bd : blocks) bd.col0 += mrows;
    // the lists themselves are built on the device (k_mosaic_targets); here only each solve's
    // first target and first list entry
    std::vector<int64_t> mt_lbase(n + 1, 0);
    int max_vo = 0;
    for (int s = 0; s < n; s++) {
        int64_t e = 0;
        for (const auto &B : b->plans[s].blocks) e += (int64_t)B.o + B.v;
        mt_lbase[s + 1] = mt_lbase[s] + e;
        max_vo = std::max(max_vo, b->plans[s].V + b->plans[s].O);
    }
    if (mt_lbase[n] >= ((int64_t)1 << 31)) return fail(UEGCCD_ERR_ARG, "batch too large for 32-bit mosaic lists");
    if ((size_t)max_vo * sizeof(int) > 200 * 1024) return fail(UEGCCD_ERR_UNSUPPORTED, "NAO too large for the mosaic lists");
    if (mrows + mcols >= ((int64_t)1 << 31)) return fail(UEGCCD_ERR_ARG, "batch too large for 32-bit mosaic indices");
    trace.mark("ph+mosaic");

    DevBatch &d = b->d;
    d.nsolves = n;
    d.nblocks = (int)blocks.size();
    int q2m = 0, n2m = 0;
    for (const auto &P : b->plans) q2m = std::max(q2m, P.q2max);
    for (const auto &v : nv4) n2m = std::max(n2m, v.x * v.x + v.y * v.y + v.z * v.z);
    d.q2max = q2m;
    d.n2max = n2m;
    int max_rows = 0;
    const std::vector<LadderTile64> ltiles = ladder_tiles(blocks, solves, d.nltiles, max_rows);
    d.ntc16 = (int)tc16.size();
    d.ntc32 = (int)tc32.size();
    d.ntc64 = (int)tc64.size();
    std::vector<LadderTile> tct;
    tct.insert(tct.end(), tc16.begin(), tc16.end());
    tct.insert(tct.end(), tc32.begin(), tc32.end());
    tct.insert(tct.end(), tc64.begin(), tc64.end());
    std::vector<TcTileDev> tcx;
    tcx.insert(tcx.end(), tcx16.begin(), tcx16.end());
    tcx.insert(tcx.end(), tcx32.begin(), tcx32.end());
    tcx.insert(tcx.end(), tcx64.begin(), tcx64.end());
    d.nwslabs = (int)wslabs.size();
    d.ndtiles = (int)dtiles.size();
    d.w16_n = w16_n;
    d.d16_n = d16_n;
    d.nscale = nscale;
    d.nchunks = (int)chunks.size();
    d.nutiles = (int)utiles.size();
    d.nrchunks = (int)rchunks.size();
    d.ntargets = (int)targets.size();
    d.max_v = max_v;
    for (int f = 0; f < 2; f++) {
        d.ladder_smem[f] = ladder_smem_bytes(q2m, n2m, max_rows, f, d.nltiles[f]);
        set_ladder_smem_limit(d.ladder_smem[f]);
    }
    // K blocks of more than some 9000 virtuals are outside what the kernels are checked for
    if (24 * (size_t)max_v + 40 * (size_t)max_o + 8 * (size_t)std::min(q2m + 1, kVtabSmemEntries) > 227 * 1024)
        return fail(UEGCCD_ERR_UNSUPPORTED, "momentum block too large");
    d.max_occ = max_occ;
    d.namp = amp0;
    // ring pairs by class, then by solve (the class sort is stable), and k_rings' CTAs: runs of one
    // solve's pairs, so long that a CTA's table serves up to four passes while the batch still
    // makes eight CTAs an SM
    std::vector<RingItemDev> ritems;
    {
        std::vector<int> cls(rpairs.size());
        std::vector<size_t> start(kRingClasses + 1, 0);
        for (size_t k = 0; k < rpairs.size(); k++) {
            if ((cls[k] = ring_class(rpairs[k].n1)) < 0) return fail(UEGCCD_ERR_UNSUPPORTED, "ring group of more than 64 rows");
            start[cls[k] + 1]++;
        }
        for (int c = 0; c < kRingClasses; c++) start[c + 1] += start[c];
        std::vector<size_t> at(start.begin(), start.end() - 1);
        std::vector<RingPairDev> sorted(rpairs.size());
        for (size_t k = 0; k < rpairs.size(); k++) sorted[at[cls[k]]++] = rpairs[k];
        rpairs.swap(sorted);
        // each pair's rows in the particle-hole arrays, in launch order: group-1 row a holds
        // 2 round8(n2) doubles (a multiple of 16: every row starts 128-byte aligned)
        int64_t xy_n = 0;
        for (auto &r : rpairs) {
            r.xy0 = (int32_t)xy_n;
            xy_n += (int64_t)r.n1 * 2 * ((r.n2 + 7) & ~7);
            if (xy_n >= ((int64_t)1 << 31)) return fail(UEGCCD_ERR_ARG, "batch too large for 32-bit ring offsets");
        }
        d.xy_n = xy_n;
        // the staging kernel walks the pairs solve by solve (a stable sort restores that order)
        spairs.assign(rpairs.begin(), rpairs.end());
        std::stable_sort(spairs.begin(), spairs.end(),
                         [](const RingPairDev &x, const RingPairDev &y) { return x.solve < y.solve; });
        int64_t passes = 0;
        for (int c = 0; c < kRingClasses; c++)
            passes += ((int64_t)(start[c + 1] - start[c]) + ring_pairs_per_pass(c) - 1) / ring_pairs_per_pass(c);
        const int per_cta = (int)std::max<int64_t>(1, std::min<int64_t>(passes / (8 * 148), 4));
        for (int c = 0; c < kRingClasses; c++) {
            const int run = ring_pairs_per_pass(c) * per_cta;
            int max_n2 = 0;
            for (size_t k = start[c]; k < start[c + 1];) {
                RingItemDev it{(int)k, 0, rpairs[k].solve, 0};
                for (; k < start[c + 1] && it.count < run && rpairs[k].solve == it.solve; k++, it.count++)
                    max_n2 = std::max(max_n2, rpairs[k].n2);
                ritems.push_back(it);
                d.nritems[c]++;
            }
            if (d.nritems[c] == 0) continue;
            d.ring_doubles[c] = ring_doubles(c, max_n2);
            d.ring_smem[c] = ring_smem_bytes(d, c, max_n2);
            if (d.ring_smem[c] > 227 * 1024) return fail(UEGCCD_ERR_UNSUPPORTED, "ring group pair exceeds shared memory");
            set_rings_smem_limit(d.ring_smem[c]);
        }
    }
    trace.mark("classes");
    d.nrpairs = (int)rpairs.size();
    trace.mark("host-tables");
    if ((rc = b->upload(d.solves, solves))) return rc;
    if ((rc = b->upload(d.blocks, blocks))) return rc;
    if ((rc = b->upload(d.ltiles, ltiles))) return rc;
    if ((rc = b->upload(d.tctiles, tct))) return rc;
    if ((rc = b->upload(d.tcx, tcx))) return rc;
    if ((rc = b->upload(d.wslabs, wslabs))) return rc;
    if ((rc = b->upload(d.dtiles, dtiles))) return rc;
    if ((rc = b->upload(d.chunks, chunks))) return rc;
    if ((rc = b->upload(d.rchunks, rchunks))) return rc;
    if ((rc = b->upload(d.utiles, utiles))) return rc;
    if ((rc = b->upload(d.utile_begin, utile_begin))) return rc;
    if ((rc = b->upload(d.targets, targets))) return rc;
    if ((rc = b->upload(d.pcol, pcol))) return rc;
    int *d_tbase = nullptr;
    int64_t *d_lbase = nullptr;
    if ((rc = b->upload(d_tbase, s_t0))) return rc;
    if ((rc = b->upload(d_lbase, mt_lbase))) return rc;
    if ((rc = b->alloc(d.mt_start, targets.size() + 1))) return rc;
    if ((rc = b->alloc(d.mt_list, (size_t)mt_lbase[n]))) return rc;
    if ((rc = b->alloc(d.mpart, mrows + mcols))) return rc;
    if ((rc = b->upload(d.pair_i, pair_i))) return rc;
    if ((rc = b->upload(d.pair_j, pair_j))) return rc;
    if ((rc = b->upload(d.vir, vir))) return rc;
    if ((rc = b->alloc(d.vpk, vir.size()))) return rc;
    if ((rc = b->alloc(d.ppk, pair_i.size()))) return rc;
    if ((rc = b->alloc(d.rowpk, pair_i.size()))) return rc;
    if ((rc = b->alloc(d.pos, pos0))) return rc;
    if ((rc = b->alloc(d.partner, amp0))) return rc;
    if ((rc = b->alloc(d.amps, amp0))) return rc;
    if ((rc = b->upload(d.nv4, nv4))) return rc;
    if ((rc = b->upload(d.nvp, nvp))) return rc;
    if ((rc = b->upload(d.eigen, eigen))) return rc;
    if ((rc = b->upload(d.vtab, vtab))) return rc;
    b->vtab_base = vtab;
    if ((rc = b->upload(d.rpairs, rpairs))) return rc;
    if ((rc = b->upload(d.spairs, spairs))) return rc;
    if ((rc = b->upload(d.ritems, ritems))) return rc;
    std::vector<int> row0(n);
    for (int s = 0; s < n; s++) row0[s] = (int)s_phr0[s];
    int *d_row0 = nullptr;
    if ((rc = b->upload(d_row0, row0))) return rc;
    if ((rc = b->alloc(d.rrows, phr0))) return rc;
    if ((rc = b->upload(d.ph_i, ph_i))) return rc;
    if ((rc = b->upload(d.ph_x, ph_x))) return rc;
    if ((rc = b->alloc(d.ridx_x, ph0))) return rc;
    if ((rc = b->alloc(d.ridx_y, ph0))) return rc;
    if ((rc = b->alloc(d.xy, d.xy_n))) return rc;
    if ((rc = b->alloc(d.rx, d.xy_n))) return rc;
    if ((rc = b->alloc(d.ph_a, phr0))) return rc;
    if ((rc = b->alloc(d.ph_b, phr0))) return rc;
    if ((rc = b->alloc(d.rpos, amp0))) return rc;
    if ((rc = b->alloc(d.t, amp0))) return rc;
    if ((rc = b->alloc(d.g, amp0))) return rc;
    if ((rc = b->alloc(d.jvv, jvv0))) return rc;
    if ((rc = b->alloc(d.joo, joo0))) return rc;
    const size_t npart = utiles.size();
    if ((rc = b->alloc(d.part_e, npart))) return rc;
    if ((rc = b->alloc(d.part_dt, npart))) return rc;
    if ((rc = b->alloc(d.part_r, npart))) return rc;
    if ((rc = b->alloc(d.red, 3 * (size_t)n))) return rc;
    if ((rc = b->alloc(d.active, n))) return rc;
    b->hsolves = solves;
    b->red.assign(3 * (size_t)n, 0.0);
    b->active.assign(n, 1);
    CU(cudaMemcpyAsync(d.active, b->active.data(), n, cudaMemcpyHostToDevice, b->stream));
    trace.mark("alloc+upload");
    // position map, amplitude list, partners and ring gather indices, from the blocks
    CU(cudaMemsetAsync(d.pos, 0xff, (size_t)pos0 * sizeof(int32_t), b->stream));   // -1: not allowed
    CU(cudaMemsetAsync(d.ph_a, 0xff, (size_t)phr0 * sizeof(int32_t), b->stream));  // -1: no ring pair
    CU(cudaMemsetAsync(d.ph_b, 0xff, (size_t)phr0 * sizeof(int32_t), b->stream));
    CU(cudaMemsetAsync(d.xy, 0, (size_t)d.xy_n * sizeof(double), b->stream));      // padding columns stay 0

    launch_block_tables(d, b->stream);
    launch_ring_rows(d, (int)phr0, d_row0, b->stream);
    launch_mosaic_targets(d, d_tbase, d_lbase, (size_t)max_vo * sizeof(int), b->stream);
    size_t dn = 0;
    for (int s = 0; s < n; s++) dn = std::max(dn, (size_t)b->plans[s].O * b->plans[s].O * b->plans[s].V);
    b->dense_n = dn;
    if ((rc = b->alloc(b->dense, 3 * dn))) return rc;
    trace.mark("device-launch");
    CU(cudaStreamSynchronize(b->stream));
    trace.mark("device-wait");
    out = std::move(b);
    return 0;
}

int set_active_all(UegccdBatch &b, uint8_t v)
{
    std::fill(b.active.begin(), b.active.end(), v);
    CU(cudaMemcpyAsync(b.d.active, b.active.data(), b.active.size(), cudaMemcpyHostToDevice, b.stream));
    b.h2d_bytes += (int64_t)b.active.size();
    return 0;
}

// Where a small device read of `bytes` lands: page-locked, so that the copy is one DMA after the
// kernels before it; the caller's own memory when there is none.
void *small_read(UegccdBatch &b, void *own, size_t bytes)
{
    if (bytes <= kWords - kReadAt) {
        if (!b.words) b.words = words_get();
        return b.words ? b.words + kReadAt : own;
    }
    if (b.pin.bytes < bytes) {
        pinned_put(b.pin);
        b.pin = pinned_get(bytes);
    }
    return b.pin.p ? b.pin.p : own;
}

int read_back(UegccdBatch &b, void *dst, const void *src, size_t bytes)
{
    void *p = small_read(b, dst, bytes);
    CU(cudaMemcpyAsync(p, src, bytes, cudaMemcpyDeviceToHost, b.stream));
    b.d2h_bytes += (int64_t)bytes;
    CU(cudaStreamSynchronize(b.stream));
    CU(cudaGetLastError());
    if (p != dst) std::memcpy(dst, p, bytes);
    return 0;
}

int read_red(UegccdBatch &b)
{
    const int rc = read_back(b, b.red.data(), b.d.red, b.red.size() * sizeof(double));
    if (rc) return rc;
    b.kt.collect();
    return 0;
}

// Copies one solve's amplitudes from a host reference-layout array into the packed t.
int pack_from_host(UegccdBatch &b, int s, const double *host_dense)
{
    const SolvePlan &P = b.plans[s];
    size_t n = (size_t)P.O * P.O * P.V;
    CU(cudaMemcpyAsync(b.dense, host_dense, n * sizeof(double), cudaMemcpyHostToDevice, b.stream));
    b.h2d_bytes += (int64_t)(n * sizeof(double));
    launch_pack(b.d, s, (int)P.namp, b.dense, b.stream);
    b.launches++;
    CU(cudaGetLastError());
    return 0;
}

// One run of device bytes and where it goes.
struct Piece {
    char *dst;
    const char *src;
    size_t bytes;
};
constexpr size_t kPiece = 32ull << 20;
void add_pieces(std::vector<Piece> &out, char *dst, const char *src, size_t bytes)
{
    for (size_t a = 0; a < bytes; a += kPiece) out.push_back(Piece{dst + a, src + a, std::min(kPiece, bytes - a)});
}

// Pieces into pageable host memory through up to three page-locked slots, the host's copy of one
// beside the device's of the next, and the stream's work done at the end: what a call locks does not grow with what it downloads.
// Without page-locked memory the driver copies them.
int download(UegccdBatch &b, const std::vector<Piece> &v, bool cores)
{
    const int n = (int)v.size(), slots = std::min(n, 3);
    size_t size = 0;
    for (const auto &p : v) size = std::max(size, (p.bytes + 63) & ~(size_t)63);
    PinnedScope buf(slots * size, b.stream);
    if (!buf.b.p) {
        for (const auto &p : v) CU(cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToHost, b.stream));
        CU(cudaStreamSynchronize(b.stream));
        return 0;
    }
    for (int k = 0; k < slots; k++)
        if (!b.ev_copy[k]) CU(event_get(b.ev_copy[k], b.dev));
    auto issue = [&](int k) {
        CU(cudaMemcpyAsync(buf.b.p + (k % slots) * size, v[k].src, v[k].bytes, cudaMemcpyDeviceToHost, b.stream));
        CU(cudaEventRecord(b.ev_copy[k % slots], b.stream));
        return 0;
    };
    int rc = 0;
    for (int k = 0; k < slots; k++)
        if ((rc = issue(k))) return rc;
    for (int k = 0; k < n; k++) {
        CU(cudaEventSynchronize(b.ev_copy[k % slots]));
        host_copy(v[k].dst, buf.b.p + (k % slots) * size, v[k].bytes, cores);
        if (k + slots < n && (rc = issue(k + slots))) return rc;
    }
    buf.settled = true;
    return 0;
}

// T2abab / T2abba / T2aaaa of solve s in the reference layout (each may be null) into host
// arrays; with_red: the batch's reduced sums too, in the same wait.  The arrays leave the device
// through page-locked memory, one copied on while the next is on its way (small ones in one run): a
// pageable copy waits for the one before it.  MP2 with its three arrays: N=38 (0.7 MB each) 0.48 ->
// 0.24 ms, N=54 (3.3 MB) 1.28 -> 0.82, N=114 (28 MB) 16 -> 6.5; one array, the residual, of 17 MB
// 3.9 -> 3.4 ms, but of 28 MB 5.7 -> 7.4: a single one above kAloneMax is left to the driver.
int unpack_to_host(UegccdBatch &b, int s, const double *t_dev, double *ab, double *ba, double *aa,
                   bool with_red = false)
{
    const SolvePlan &P = b.plans[s];
    const size_t n = (size_t)P.O * P.O * P.V, bytes = n * sizeof(double);
    double *out[3] = {ab, ba, aa}, *host[3], *dev[3] = {nullptr, nullptr, nullptr};
    int m = 0;
    for (int k = 0; k < 3; k++)
        if (out[k]) {
            dev[k] = b.dense + m * n;
            host[m++] = out[k];
        }
    CU(cudaMemsetAsync(b.dense, 0, m * bytes, b.stream));
    launch_unpack(b.d, s, (int)P.namp, t_dev, dev[0], dev[1], dev[2], b.stream);
    b.launches++;
    CU(cudaGetLastError());
    b.d2h_bytes += (int64_t)(m * bytes);
    const size_t red = with_red ? b.red.size() * sizeof(double) : 0;
    void *sums = red ? small_read(b, b.red.data(), red) : nullptr;
    if (red) {
        CU(cudaMemcpyAsync(sums, b.d.red, red, cudaMemcpyDeviceToHost, b.stream));
        b.d2h_bytes += (int64_t)red;
    }
    constexpr size_t kAloneMax = 24ull << 20, kApartMin = 512ull << 10;
    bool direct = true;   // page-locked destinations take the copies themselves
    for (int k = 0; k < m; k++) direct = direct && is_pinned(host[k]);
    direct = direct || (m == 1 && bytes > kAloneMax);
    if (!direct && bytes >= kApartMin) {
        std::vector<Piece> v;
        for (int k = 0; k < m; k++) add_pieces(v, (char *)host[k], (const char *)(b.dense + k * n), bytes);
        const int rc = download(b, v, m * bytes > 2 * kCoresMin);
        if (rc) return rc;
    } else {
        PinnedScope buf(direct ? 0 : m * bytes, b.stream);
        if (buf.b.p) CU(cudaMemcpyAsync(buf.b.p, b.dense, m * bytes, cudaMemcpyDeviceToHost, b.stream));
        for (int k = 0; !buf.b.p && k < m; k++)
            CU(cudaMemcpyAsync(host[k], b.dense + k * n, bytes, cudaMemcpyDeviceToHost, b.stream));
        CU(cudaStreamSynchronize(b.stream));
        buf.settled = true;
        for (int k = 0; buf.b.p && k < m; k++) std::memcpy(host[k], buf.b.p + k * bytes, bytes);
    }
    if (red && sums != b.red.data()) std::memcpy(b.red.data(), sums, red);
    return 0;
}

// Integral options for every later call on the batch (SetPointers, Main.f90:274-318, with
// no range flags): GapII > 0 zeroes the integrals above GapII (GapERI, HEG.f90:938-940) --
// the |q|^2 tables are filtered; CoreN > 0 zeroes those with an index p <= CoreN
// (CoreERI, HEG.f90:882-885) -- the kernels hold core pairs at zero.
// The |q|^2 tables of every solve for an ERI flag (CasedERI, HEG.f90:725-774; flag 0 is
// BaseERI's value), with the reference's "< 0 -> -100" guard and the GapII filter applied in
// its order.  CoreN is not in the tables: the kernels hold core pairs at zero.
std::vector<double> integral_tables(const UegccdBatch &b, int flag, double gapii)
{
    std::vector<double> vt;
    vt.reserve(b.vtab_base.size());
    for (size_t s = 0; s < b.plans.size(); s++) {
        const double L = b.sys[s].L, mad = b.sys[s].madelung, sd = b.screening;
        for (int q2 = 0; q2 <= b.plans[s].q2max; q2++) {
            double v = 0.0;
            if (flag == 0) {
                v = coulomb_v(L, mad, q2);
            } else if (q2 == 0) {
                if (flag == 1) v = (1.0 / std::pow(L, 3.0)) * 4.0 * kPi / std::pow(sd, 2.0);
                else if (flag == 2) v = -mad - (1.0 / std::pow(L, 3.0)) * 4.0 * kPi / std::pow(sd, 2.0);
            } else {
                const double q2s = (double)q2 * std::pow(2.0 * kPi / L, 2.0);
                if (flag == 1) v = (1.0 / std::pow(L, 3.0)) * 4.0 * kPi / (std::pow(sd, 2.0) + q2s);
                else if (flag == 2)
                    v = (1.0 / std::pow(L, 3.0)) * 4.0 * kPi / (std::pow(sd, 2.0) + q2s) * std::pow(sd, 2.0) / q2s;
            }
            if (flag != 0 && v < 0.0) v = -100.0;
            if (gapii > 0.0 && v > gapii) v = 0.0;
            vt.push_back(v);
        }
    }
    return vt;
}

// Uploads the tables of an ERI flag.
int load_tables(UegccdBatch &b, int flag)
{
    const std::vector<double> vt = integral_tables(b, flag, b.gapii);
    CU(cudaMemcpyAsync(b.d.vtab, vt.data(), vt.size() * sizeof(double), cudaMemcpyHostToDevice, b.stream));
    b.d.w16_valid = false;   // the FP16 Coulomb slabs follow the tables
    CU(cudaGetLastError());
    CU(cudaStreamSynchronize(b.stream));
    b.h2d_bytes += (int64_t)(vt.size() * sizeof(double));
    return 0;
}

int set_integrals(UegccdBatch &b, int core_n, double gapii)
{
    if (core_n < 0) return fail(UEGCCD_ERR_ARG, "CoreN must be >= 0");
    for (const auto &P : b.plans)
        if (core_n > P.O) return fail(UEGCCD_ERR_ARG, "CoreN exceeds NOcc");
    const double g = gapii > 0.0 ? gapii : 0.0;
    if (core_n == b.core_n && g == b.gapii) return 0;
    std::vector<double> vt(b.vtab_base);
    if (g > 0.0)
        for (auto &v : vt)
            if (v > g) v = 0.0;
    CU(cudaMemcpyAsync(b.d.vtab, vt.data(), vt.size() * sizeof(double), cudaMemcpyHostToDevice, b.stream));
    for (auto &S : b.hsolves) S.core_n = core_n;
    CU(cudaMemcpyAsync(b.d.solves, b.hsolves.data(), b.hsolves.size() * sizeof(SolveDev), cudaMemcpyHostToDevice,
                       b.stream));
    b.d.w16_valid = false;   // the FP16 Coulomb slabs follow the tables
    CU(cudaGetLastError());
    CU(cudaStreamSynchronize(b.stream));
    b.h2d_bytes += (int64_t)(vt.size() * sizeof(double) + b.hsolves.size() * sizeof(SolveDev));
    b.core_n = core_n;
    b.gapii = g;
    return 0;
}

// Buffers of the mixed-precision ladder, on first use; the FP16 Coulomb slabs are (re)built
// whenever the integral tables changed since.
int mixed_alloc(UegccdBatch &b)
{
    DevBatch &d = b.d;
    int rc = 0;
    if (!d.t_ref) {
        if ((rc = b.alloc(d.t_ref, d.namp))) return rc;
        if ((rc = b.alloc(d.g_ref, d.namp))) return rc;
        if ((rc = b.alloc(d.tc_err, 1))) return rc;
        uint16_t *w = nullptr, *dd = nullptr;
        if ((rc = b.alloc(w, (size_t)d.w16_n))) return rc;
        if ((rc = b.alloc(dd, (size_t)d.d16_n))) return rc;
        CU(cudaMemsetAsync(dd, 0, (size_t)d.d16_n * sizeof(uint16_t), b.stream));   // the tiles' padding
        if ((rc = b.alloc(d.dscale, (size_t)d.nscale))) return rc;
        d.w16 = w;
        d.d16 = dd;
    }
    if (!d.w16_valid) {
        launch_w16_build(d, b.stream);
        CU(cudaGetLastError());
        d.w16_valid = true;
    }
    return 0;
}

// Lookups and sums of the dRPA terms, on the first dRPA solve.
int drpa_alloc(UegccdBatch &b)
{
    DevBatch &d = b.d;
    if (d.drs2) return 0;
    const int n = d.nsolves;
    std::vector<int4> list;
    std::vector<DrpaSolveDev> ds(n);
    int64_t rij = 0, cp = 0, ph = 0;
    int ranges = 0, jp = 0;
    for (int s = 0; s < n; s++) {
        const SolvePlan &P = b.plans[s];
        const int nc = (P.V + kDrpaCols - 1) / kDrpaCols;
        ds[s] = DrpaSolveDev{rij, cp, ranges, nc, jp, 0};
        ranges += nc;
        jp += nc > 1 ? P.O * nc : 0;
        rij += (int64_t)P.O * P.O;
        cp += (int64_t)P.blocks.size() * P.V;
        ph += (int64_t)P.O * P.V;
        for (int c = 0; c < nc; c++)
            for (int i = 0; i < P.O; i++) list.push_back(make_int4(s, i, c, 0));
    }
    const UegccdBatch::Mark m = b.mark();
    DevBatch x = d;
    int rc = 0;
    if ((rc = b.upload(x.drlist, list)) || (rc = b.upload(x.drsolves, ds)) || (rc = b.alloc(x.drows, (size_t)rij)) ||
        (rc = b.alloc(x.colpos, (size_t)cp)) || (rc = b.alloc(x.drdone, ranges + n)) ||
        (rc = b.alloc(x.drj, (size_t)jp)) || (rc = b.alloc(x.dru, (size_t)ph)) || (rc = b.alloc(x.drs2, (size_t)ph))) {
        cudaStreamSynchronize(b.stream);   // the uploads above read host vectors of this call
        b.rollback(m);
        return rc;
    }
    x.ndrlist = (int)list.size();
    x.ndrranges = ranges;
    CU(cudaMemsetAsync(x.drows, 0xff, (size_t)rij * sizeof(int4), b.stream));
    CU(cudaMemsetAsync(x.colpos, 0xff, (size_t)cp * sizeof(int16_t), b.stream));
    CU(cudaMemsetAsync(x.drdone, 0, (ranges + n) * sizeof(int), b.stream));
    launch_drpa_tables(x, b.stream);
    CU(cudaGetLastError());
    CU(cudaStreamSynchronize(b.stream));
    d = x;
    return 0;
}

int validate_options(const UegccdOptions *o, int drpa, const UegccdBatch &b, bool two_channel = false)
{
    if (!o) return fail(UEGCCD_ERR_ARG, "null options");
    if (two_channel) {
        // the two-channel form takes its integrals from uegccd_ctx_set_eri, not range_flags
        if (o->precision != UEGCCD_FP64) return fail(UEGCCD_ERR_UNSUPPORTED, "the two-channel form runs in FP64");
    } else {
        if (o->range_flags != 0 && drpa)
            return fail(UEGCCD_ERR_UNSUPPORTED,
                        "range-separated dRPA takes per-term flags: uegccd_ctx_set_eri on a context");
        if (o->range_flags != 0 && b.range_flag == 0)
            return fail(UEGCCD_ERR_UNSUPPORTED,
                        "range-separated integrals: set one flag for every term with uegccd_*_set_range, or "
                        "per-term flags with uegccd_ctx_set_eri on a context");
        if (!drpa && (o->do_ring != 0) != (o->do_xring != 0))
            return fail(UEGCCD_ERR_UNSUPPORTED,
                        "Do Rings and Do XRings must agree in a batch solve: alone, either breaks the spin "
                        "symmetry of the batched kernels (a context's uegccd_ccd runs the two-channel form)");
    }
    if (o->max_iter <= 0 || !(o->tol > 0) || !(o->denom_factor != 0)) return fail(UEGCCD_ERR_ARG, "bad iteration options");
    if (o->scheme != UEGCCD_REPLAY && o->scheme != UEGCCD_DIIS) return fail(UEGCCD_ERR_ARG, "unknown scheme");
    if (o->scheme == UEGCCD_DIIS && (o->ndiis < 2 || o->ndiis > kDiisMax))
        return fail(UEGCCD_ERR_ARG, "ndiis must be in [2, 16]");
    if (o->precision != UEGCCD_FP64 && o->precision != UEGCCD_MIXED) return fail(UEGCCD_ERR_ARG, "unknown precision");
    return 0;
}

// Buffers of the device-side iteration control, grown on demand.  Each group of arrays is
// allocated as a whole: when one of them fails, the group's memory goes back and the batch
// keeps what it had.
int ctl_alloc(UegccdBatch &b, int ndiis, int max_rec)
{
    CtlBuffers &c = b.ctl;
    const int n = b.d.nsolves;
    int rc = 0;
    if (!c.done) {
        for (auto &e : b.ev_iter)
            if (!e) CU(event_get(e, b.dev));
        if (!b.words && !(b.words = words_get())) return fail(UEGCCD_ERR_ALLOC, "no page-locked host memory");
        c.done = reinterpret_cast<int *>(b.words);
    }
    if (!c.state) {
        const UegccdBatch::Mark m = b.mark();
        CtlBuffers x = c;
        if ((rc = b.alloc(x.state, n)) || (rc = b.alloc(x.applied, n)) || (rc = b.alloc(x.stopped, 1)) ||
            (rc = b.alloc(x.Bm, (size_t)n * kDiisMax * kDiisMax)) || (rc = b.alloc(x.coef, (size_t)n * kDiisMax)) ||
            (rc = b.alloc(x.part, (size_t)b.d.nutiles * kDiisMax))) {
            b.rollback(m);
            return rc;
        }
        c = x;
    }
    if (max_rec > c.max_rec) {
        const UegccdBatch::Mark m = b.mark();
        double *re = nullptr, *rd = nullptr;
        if ((rc = b.alloc(re, (size_t)n * max_rec)) || (rc = b.alloc(rd, (size_t)n * max_rec))) {
            b.rollback(m);
            return rc;
        }
        c.rec_e = re;
        c.rec_dt = rd;
        c.max_rec = max_rec;
        b.drop_graphs();
    }
    if (ndiis > b.diis_cap) {
        const UegccdBatch::Mark m = b.mark();
        double *ht = nullptr;
        float *he = nullptr;
        if ((rc = b.alloc(ht, (size_t)ndiis * b.d.namp)) || (rc = b.alloc(he, (size_t)ndiis * b.d.namp))) {
            b.rollback(m);
            return rc;
        }
        c.hist_t = ht;
        c.hist_e = he;
        b.diis_cap = ndiis;
        b.drop_graphs();
    }
    return 0;
}

// The side streams of a batch.  The ring classes always run beside each other: each is a launch of
// its own whose last CTAs leave the GPU idle.  In a small batch the rings, the mosaics and the DMMA
// ladders also run beside the FMA ladders; in a large one each kernel fills the GPU, and run
// together they contend for the SMs and L2.  Solve times in ms on one stream, with the ring classes
// apart, with the terms apart: one N=54 system 1.50, 1.2, 0.93; 8 of them 2.72, 2.53, 2.13;
// 32 (7 M packed amplitudes) 6.76, 6.37, 6.30; 48 (10.5 M) 8.70 and 9.16 apart; 100 (22 M) 17.02,
// 16.47, 18.46; four N=114 systems (8.5 M) 11.8, 10.7, 9.7; 8 of them (17 M) 20.9, 18.8, 17.9; 16 of
// them (34 M) 36.0, 34.2, 34.3.
constexpr int64_t kForkAmps = 9000000;
constexpr int kForkSolves = 8;
const Fork *fork_of(UegccdBatch &b)
{
    if (!b.fork_made) {
        b.fork_made = true;
        if (fork_get(b.fork, b.dev)) b.fork.terms = b.d.namp <= kForkAmps || b.d.nsolves <= kForkSolves;
    }
    return b.fork.s[0] ? &b.fork : nullptr;   // else one stream serves all
}

// Captures one iteration as a CUDA graph.
int capture_iteration(UegccdBatch &b, const TermFlags &f, double tol, int max_iter, int ndiis)
{
    UegccdBatch::GraphKey key{f.do_ring, f.do_xring, f.do_ladder, f.do_mosaic, f.drpa, ndiis, max_iter, f.mixed, tol};
    UegccdBatch::IterGraph &G = b.graphs[f.mixed ? 1 : 0];
    if (G.valid && G.key == key) return 0;
    G.valid = false;
    if (G.exec) { cudaGraphExecDestroy(G.exec); G.exec = nullptr; }
    const Fork *fork = f.drpa ? nullptr : fork_of(b);   // dRPA's terms follow one another
    cudaGraph_t g = nullptr;
    CU(cudaStreamBeginCapture(b.stream, cudaStreamCaptureModeThreadLocal));
    int nl = launch_iteration(b.d, b.ctl, f, tol, max_iter, ndiis, b.stream, nullptr, fork);
    cudaError_t e = cudaStreamEndCapture(b.stream, &g);
    if (e != cudaSuccess) return fail(UEGCCD_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&G.exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return fail(UEGCCD_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    G.launches = nl;
    G.key = key;
    G.valid = true;
    return 0;
}

// The launch shape of a batch (k_ring_stage's CTA size): measured once per batch shape in this
// process (the shape: ring pairs and their operands' size), on the first CCD solve, before the
// iteration graph is captured.
std::mutex g_tune_mu;
std::map<std::pair<int64_t, int64_t>, int> g_stage_tuning;

int tune_batch(UegccdBatch &b)
{
    DevBatch &d = b.d;
    const std::pair<int64_t, int64_t> key{d.nrpairs, d.xy_n};
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto it = g_stage_tuning.find(key);
        if (it != g_stage_tuning.end()) {
            d.stage_threads = it->second;
            b.tuned = true;
            return 0;
        }
    }
    const int e = tune_stage(d, b.stream);
    if (e != 0) return fail(UEGCCD_ERR_CUDA, std::string("launch-shape tuning: ") + cudaGetErrorString((cudaError_t)e));
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_stage_tuning[key] = d.stage_threads;
    b.tuned = true;
    return 0;
}

// Runs the iteration for all solves of the batch from the amplitudes in d.t (from_mp2: those
// k_mp2 has just written).
// Iteration control lives on the device; the host replays a captured iteration graph, keeps one
// queued behind the one whose end it waits for, and stops at the flag the last solve to stop
// sets.  With kernel timing on, the last iteration of each round of kPoll runs as direct
// launches between CUDA events: that iteration is the sample the per-kernel times come from.
int run_solves(UegccdBatch &b, const UegccdOptions *opt, int drpa, UegccdResult *res, bool from_mp2 = false)
{
    constexpr int kPoll = 4;
    DevBatch &d = b.d;
    const int n = d.nsolves;
    TermFlags f;
    f.drpa = drpa;
    f.do_driver = 1;
    f.do_mosaic = opt->do_mosaic ? 1 : 0;
    f.do_ladder = (!drpa && opt->do_ladder) ? 1 : 0;
    f.do_ring = opt->do_ring ? 1 : 0;
    f.do_xring = (!drpa && opt->do_xring) ? 1 : 0;
    // range-separated integrals: every CCD term and the energy on the flag's tables (the MP2
    // start before this used the plain ones); the plain tables back on every exit
    struct TableGuard {
        UegccdBatch &b;
        bool on;
        ~TableGuard()
        {
            // a batch left on the range-separated tables would give wrong MP2 and CCD results
            // later: refuse every further call on it instead
            if (on && load_tables(b, 0) != 0) b.broken = true;
        }
    } table_guard{b, false};
    if (opt->range_flags != 0 && b.range_flag != 0) {
        const int rc0 = load_tables(b, b.range_flag);
        if (rc0) return rc0;
        table_guard.on = true;
    }
    const int max_rec = std::min(opt->max_iter, 1100);
    // The DIIS history takes fewer vectors when the device memory (or the library's limit)
    // does not hold ndiis of them, down to 2, as SetUpDIISCC steps Max_N_DIIS down until its
    // Allocate succeeds (DIISCC.f90:22-29); the vectors used are reported per solve.
    int ndiis = opt->scheme == UEGCCD_DIIS ? opt->ndiis : 0;
    int rc = 0;
    while ((rc = ctl_alloc(b, ndiis, max_rec)) == UEGCCD_ERR_ALLOC && ndiis > 2) ndiis--;
    if (rc) return rc;
    for (int s = 0; s < n; s++) b.hsolves[s].denom_factor = opt->denom_factor;
    CU(cudaMemcpyAsync(d.solves, b.hsolves.data(), n * sizeof(SolveDev), cudaMemcpyHostToDevice, b.stream));
    std::vector<IterState> st0(n, IterState{1, 0, 0.0, 0.0});
    CU(cudaMemcpyAsync(b.ctl.state, st0.data(), n * sizeof(IterState), cudaMemcpyHostToDevice, b.stream));
    CU(cudaMemsetAsync(b.ctl.Bm, 0, (size_t)n * kDiisMax * kDiisMax * sizeof(double), b.stream));
    if ((rc = set_active_all(b, 1))) return rc;
    if (opt->precision == UEGCCD_MIXED && (rc = mixed_alloc(b))) return rc;
    if (drpa && (rc = drpa_alloc(b))) return rc;
    if (d.tc_err) CU(cudaMemsetAsync(d.tc_err, 0, sizeof(int), b.stream));
    if (!b.tuned && !drpa && (f.do_ring || f.do_xring) && (rc = tune_batch(b))) return rc;
    b.launches = 0;
    CU(cudaEventRecord(b.ev0, b.stream));
    // CCEnergy of the start amplitudes and dT = max|T| (CCD.f90:63-64, dRPA.f90:68-69).  Those of
    // the MP2 amplitudes on the plain integrals are k_mp2's own sums.
    if (!from_mp2 || drpa || table_guard.on) {
        launch_energy(d, drpa ? 1 : 0, 0.0, b.stream);
        b.launches++;
    }
    *(volatile int *)b.ctl.done = 0;
    launch_tail(d, b.ctl, opt->tol, opt->max_iter, ndiis, 1, b.stream);
    b.launches++;
    // The iterations go in rounds of kPoll (a mixed solve's refreshes).  The GPU does not wait for the
    // host, and a batch that has stopped costs one empty iteration.  (A copy of the count and a wait every four
    // iterations left the GPU idle for 22 us and up to three iterations empty.)
    const int max_rounds = opt->max_iter / kPoll + 2;
    // mixed precision: tensor-core ladder of t - t_ref, t_ref refreshed (FP64) each round,
    // then FP64 iterations from where the mixed phase stopped (refinement)
    const bool mixed = opt->precision == UEGCCD_MIXED && f.do_ladder && f.do_pp;
    for (int phase = mixed ? 0 : 1; phase < 2; phase++) {
        f.mixed = phase == 0 ? 1 : 0;
        if (phase == 1 && mixed) {
            // reopen every solve for the FP64 sweeps
            std::vector<IterState> st1(n);
            if ((rc = read_back(b, st1.data(), b.ctl.state, n * sizeof(IterState)))) return rc;
            for (auto &x : st1) x.status = 0;
            CU(cudaMemcpyAsync(b.ctl.state, st1.data(), n * sizeof(IterState), cudaMemcpyHostToDevice, b.stream));
            if ((rc = set_active_all(b, 1))) return rc;
            CU(cudaMemsetAsync(b.ctl.stopped, 0, sizeof(int), b.stream));
            *(volatile int *)b.ctl.done = 0;
        }
        if ((rc = capture_iteration(b, f, opt->tol, opt->max_iter, ndiis))) return rc;
        const UegccdBatch::IterGraph &G = b.graphs[f.mixed];
        auto stopped = [&](int it) {   // 1 when no solve iterates after iteration `it`, -1: failed
            if (cudaEventSynchronize(b.ev_iter[it & 1]) != cudaSuccess) return -1;
            return (int)*(volatile int *)b.ctl.done;
        };
        const int most = phase == 1 && mixed ? std::min(max_rounds, std::max(1, opt->refine_sweeps)) : max_rounds;
        int it = 0, stop = 0;
        for (int round = 0; round < most && stop == 0; round++) {
            // the refresh is not queued ahead: it costs as much as an iteration
            if (f.mixed && it > 0 && (stop = stopped(it - 1)) != 0) break;
            if (f.mixed) b.launches += launch_refresh(d, b.stream);
            for (int k = 0; k < kPoll && stop == 0; k++, it++) {
                if (b.kt.on && k == kPoll - 1) {
                    // the sampled iteration of the round: direct launches between CUDA events
                    b.launches += launch_iteration(d, b.ctl, f, opt->tol, opt->max_iter, ndiis, b.stream, &b.kt);
                } else {
                    CU(cudaGraphLaunch(G.exec, b.stream));
                    b.launches += G.launches;
                }
                CU(cudaEventRecord(b.ev_iter[it & 1], b.stream));
                if (it > 0) stop = stopped(it - 1);
            }
            if (b.kt.on) {
                CU(cudaStreamSynchronize(b.stream));
                b.kt.collect();
            }
        }
        if (stop < 0) CU(cudaStreamSynchronize(b.stream));
        CU(cudaGetLastError());
        // (the iteration queued behind may still run: what follows is on its stream)
    }
    if (mixed) {
        int err = 0;
        CU(cudaMemcpyAsync(&err, d.tc_err, sizeof(int), cudaMemcpyDeviceToHost, b.stream));
        CU(cudaStreamSynchronize(b.stream));
        if (err) return fail(UEGCCD_ERR_CUDA, "tensor-core ladder: an mbarrier wait expired");
    }
    // final residual (CCD.f90:103-107, dRPA.f90:98-101)
    if ((rc = set_active_all(b, 1))) return rc;
    b.launches += launch_residual(d, f, 1, nullptr, b.stream, &b.kt);
    if ((rc = read_red(b))) return rc;
    std::vector<double> rmax(n), esosex(n, 0.0);
    for (int s = 0; s < n; s++) rmax[s] = b.red[3 * s + 2];
    if (drpa) {
        launch_energy(d, 1, 1.0, b.stream);
        launch_reduce(d, b.stream);
        b.launches += 2;
        if ((rc = read_red(b))) return rc;
        for (int s = 0; s < n; s++) esosex[s] = b.red[3 * s];
    }
    std::vector<IterState> st(n);
    CU(cudaMemcpyAsync(st.data(), b.ctl.state, n * sizeof(IterState), cudaMemcpyDeviceToHost, b.stream));
    int nrec = 0;
    if (opt->max_rec > 0 && (opt->energies || opt->dts)) {
        nrec = std::min(std::min(st[0].niter, max_rec), opt->max_rec);
        std::vector<double> re(nrec), rd(nrec);
        CU(cudaMemcpyAsync(re.data(), b.ctl.rec_e, nrec * sizeof(double), cudaMemcpyDeviceToHost, b.stream));
        CU(cudaMemcpyAsync(rd.data(), b.ctl.rec_dt, nrec * sizeof(double), cudaMemcpyDeviceToHost, b.stream));
        CU(cudaStreamSynchronize(b.stream));
        for (int k = 0; k < nrec; k++) {
            if (opt->energies) opt->energies[k] = re[k];
            if (opt->dts) opt->dts[k] = rd[k];
        }
    }
    CU(cudaEventRecord(b.ev1, b.stream));
    CU(cudaEventSynchronize(b.ev1));
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, b.ev0, b.ev1));
    int status = 0;
    b.last_niter.assign(n, 0);
    for (int s = 0; s < n; s++) b.last_niter[s] = std::min(st[s].niter, max_rec);
    for (int s = 0; s < n; s++) {
        UegccdResult &r = res[s];
        r.ecorr = st[s].e;
        r.max_res = rmax[s];
        r.last_dt = st[s].dt;
        r.niter = st[s].niter;
        r.fail = rmax[s] > opt->fail_ratio * opt->tol;
        r.ecorr_sosex = (drpa && !r.fail) ? esosex[s] : 0.0;
        r.n_recorded = (s == 0) ? nrec : 0;
        r.kernel_launches = b.launches;
        r.gpu_ms = ms;
        r.status = st[s].status == 3 ? UEGCCD_ERR_NUMERIC
                   : (r.fail || st[s].status == 2) ? UEGCCD_NOT_CONVERGED : UEGCCD_OK;
        r.ndiis = ndiis;
        if (r.status == UEGCCD_ERR_NUMERIC) status = UEGCCD_ERR_NUMERIC;
        if (status == 0 && r.status == UEGCCD_NOT_CONVERGED) status = UEGCCD_NOT_CONVERGED;
    }
    if (status == UEGCCD_ERR_NUMERIC) fail(status, "non-finite amplitudes or energy");
    return status;
}

// Opens an incremental solve: the set-up of run_solves (control buffers with the DIIS depth
// step-down, start energy and state, the iteration graph), after the MP2 start.
int session_start(UegccdBatch &b, const UegccdOptions *opt, int drpa)
{
    DevBatch &d = b.d;
    const int n = d.nsolves;
    auto &S = b.ses;
    S = UegccdBatch::Session{};
    TermFlags &f = S.f;
    f.drpa = drpa;
    f.do_driver = 1;
    f.do_mosaic = opt->do_mosaic ? 1 : 0;
    f.do_ladder = (!drpa && opt->do_ladder) ? 1 : 0;
    f.do_ring = opt->do_ring ? 1 : 0;
    f.do_xring = (!drpa && opt->do_xring) ? 1 : 0;
    f.mixed = 0;
    S.max_rec = std::min(opt->max_iter, 1100);
    int ndiis = opt->scheme == UEGCCD_DIIS ? opt->ndiis : 0;
    int rc = 0;
    while ((rc = ctl_alloc(b, ndiis, S.max_rec)) == UEGCCD_ERR_ALLOC && ndiis > 2) ndiis--;
    if (rc) return rc;
    for (int s = 0; s < n; s++) b.hsolves[s].denom_factor = opt->denom_factor;
    CU(cudaMemcpyAsync(d.solves, b.hsolves.data(), n * sizeof(SolveDev), cudaMemcpyHostToDevice, b.stream));
    std::vector<IterState> st0(n, IterState{1, 0, 0.0, 0.0});
    CU(cudaMemcpyAsync(b.ctl.state, st0.data(), n * sizeof(IterState), cudaMemcpyHostToDevice, b.stream));
    CU(cudaMemsetAsync(b.ctl.Bm, 0, (size_t)n * kDiisMax * kDiisMax * sizeof(double), b.stream));
    if ((rc = set_active_all(b, 1))) return rc;
    if (drpa && (rc = drpa_alloc(b))) return rc;
    if (!b.tuned && !drpa && (f.do_ring || f.do_xring) && (rc = tune_batch(b))) return rc;
    if (drpa) {   // else k_mp2's own sums are those of the start amplitudes
        launch_energy(d, 1, 0.0, b.stream);
        b.launches++;
    }
    *(volatile int *)b.ctl.done = 0;
    launch_tail(d, b.ctl, opt->tol, opt->max_iter, ndiis, 1, b.stream);
    b.launches++;
    if ((rc = capture_iteration(b, f, opt->tol, opt->max_iter, ndiis))) return rc;
    CU(cudaStreamSynchronize(b.stream));
    S.opt = *opt;
    S.drpa = drpa;
    S.ndiis = ndiis;
    S.released.assign(n, 0);
    S.on = true;
    return 0;
}

// Up to `rounds` poll rounds of the open incremental solve, then the results of every solve
// that stopped since the last call: their final residual (MaxRes, CCD.f90:103-107) is formed
// with only them active, after which the still-running solves are active again.
int session_advance(UegccdBatch &b, int rounds, int *n_active, int *n_done, int *ids, UegccdResult *res)
{
    constexpr int kPoll = 4;
    DevBatch &d = b.d;
    auto &S = b.ses;
    const int n = d.nsolves;
    const UegccdOptions &opt = S.opt;
    for (int r = 0; r < rounds && *(volatile int *)b.ctl.done == 0; r++) {
        for (int k = 0; k < kPoll; k++) {
            CU(cudaGraphLaunch(b.graphs[0].exec, b.stream));
            b.launches += b.graphs[0].launches;
        }
        if (r + 1 < rounds) CU(cudaStreamSynchronize(b.stream));
    }
    std::vector<IterState> st(n);
    {
        const int rc = read_back(b, st.data(), b.ctl.state, n * sizeof(IterState));
        if (rc) return rc;
    }
    std::vector<int> fresh;
    for (int s = 0; s < n; s++)
        if (st[s].status != 0 && !S.released[s]) fresh.push_back(s);
    *n_done = (int)fresh.size();
    int running = 0;
    for (int s = 0; s < n; s++) running += st[s].status == 0;
    *n_active = running;
    if (!fresh.empty()) {
        std::fill(b.active.begin(), b.active.end(), 0);
        for (int s : fresh) b.active[s] = 1;
        CU(cudaMemcpyAsync(d.active, b.active.data(), n, cudaMemcpyHostToDevice, b.stream));
        b.h2d_bytes += n;
        b.launches += launch_residual(d, S.f, 1, nullptr, b.stream, nullptr);
        int rc = read_red(b);
        if (rc) return rc;
        std::vector<double> rmax(n), esosex(n, 0.0);
        for (int s = 0; s < n; s++) rmax[s] = b.red[3 * s + 2];
        if (S.drpa) {
            launch_energy(d, 1, 1.0, b.stream);
            launch_reduce(d, b.stream);
            b.launches += 2;
            if ((rc = read_red(b))) return rc;
            for (int s = 0; s < n; s++) esosex[s] = b.red[3 * s];
        }
        for (size_t k = 0; k < fresh.size(); k++) {
            const int s = fresh[k];
            UegccdResult &r = res[k];
            std::memset(&r, 0, sizeof r);
            ids[k] = s;
            r.ecorr = st[s].e;
            r.max_res = rmax[s];
            r.last_dt = st[s].dt;
            r.niter = st[s].niter;
            r.fail = rmax[s] > opt.fail_ratio * opt.tol;
            r.ecorr_sosex = (S.drpa && !r.fail) ? esosex[s] : 0.0;
            r.kernel_launches = b.launches;
            r.status = st[s].status == 3 ? UEGCCD_ERR_NUMERIC
                       : (r.fail || st[s].status == 2) ? UEGCCD_NOT_CONVERGED : UEGCCD_OK;
            r.ndiis = S.ndiis;
            S.released[s] = 1;
        }
        for (int s = 0; s < n; s++) b.active[s] = st[s].status == 0 ? 1 : 0;
        CU(cudaMemcpyAsync(d.active, b.active.data(), n, cudaMemcpyHostToDevice, b.stream));
        b.h2d_bytes += n;
        CU(cudaStreamSynchronize(b.stream));
    }
    if (running == 0) S.on = false;
    return 0;
}

}  // namespace

namespace uegccd {
// The message uegccd_last_error returns, for entry points defined in other files.
int set_last_error(int code, const char *msg) { return fail(code, msg); }
// 0 when a compute-capability-10 device is current, else an error status (message set).
int device_ok() { return check_device(); }
}  // namespace uegccd

// SendForAllocation (HEG.f90:1051-1065): SfLength = maxval(nVec)*2+1
int sf_length(const SystemHost &h)
{
    int m = h.n.empty() ? 0 : h.n[0][0];
    for (const auto &v : h.n) m = std::max(m, std::max(v[0], std::max(v[1], v[2])));
    return m * 2 + 1;
}

// Structure factors of solve s from the batch's amplitudes: the sums on the device
// (k_sf), then SfG and SfV -- functions of q alone -- at the points the sums reached,
// with the reference's expressions: SfG = (|q|^2 (2 pi/L)^2)**0.5 (dK2scaled,
// HEG.f90:1011-1031), SfV = the integral of the last contribution in the reference's
// loop order: BaseERI (HEG.f90:969-976) with the GapII filter, 0 for a core pair.
int structure_factor(UegccdBatch &b, int s, const UegccdSfGrid &out)
{
    DevBatch &d = b.d;
    const int n = d.nsolves;
    int rc = 0;
    if (!b.sf_groups) {
        std::vector<int2> g;
        b.sf_g0.assign(n + 1, 0);
        int64_t w3max = 1;
        for (int k = 0; k < n; k++) {
            for (const auto &G : b.plans[k].groups) g.push_back(make_int2(G.r0, G.n));
            b.sf_g0[k + 1] = (int)g.size();
            const int64_t w = 2 * sf_length(b.sys[k]) + 1;
            w3max = std::max(w3max, w * w * w);
        }
        if ((rc = b.upload(b.sf_groups, g))) return rc;
        if ((rc = b.alloc(b.sf_grid, 5 * (size_t)w3max))) return rc;
        if ((rc = b.alloc(b.sf_err, 1))) return rc;

    }
    const SystemHost &H = b.sys[s];
    const int S = sf_length(H);
    const int64_t W = 2 * S + 1, W3 = W * W * W;
    CU(cudaMemsetAsync(b.sf_grid, 0, 5 * (size_t)W3 * sizeof(double), b.stream));
    CU(cudaMemsetAsync(b.sf_err, 0, sizeof(int), b.stream));
    launch_sf(d, b.sf_groups + b.sf_g0[s], b.sf_g0[s + 1] - b.sf_g0[s], s, S, b.sf_grid, b.sf_err, b.stream);
    b.launches++;
    CU(cudaGetLastError());
    double *dst[3] = {out.sum, out.dsum, out.xsum};
    for (int k = 0; k < 3; k++)
        if (dst[k]) CU(cudaMemcpyAsync(dst[k], b.sf_grid + k * W3, W3 * sizeof(double), cudaMemcpyDeviceToHost, b.stream));
    // contributions, and where the last one is a core pair (read under CoreN only)
    const int ntail = b.core_n > 0 ? 2 : 1;
    std::vector<double> cnt((size_t)ntail * W3);
    CU(cudaMemcpyAsync(cnt.data(), b.sf_grid + 3 * W3, ntail * W3 * sizeof(double), cudaMemcpyDeviceToHost,
                       b.stream));
    int err = 0;
    CU(cudaMemcpyAsync(&err, b.sf_err, sizeof(int), cudaMemcpyDeviceToHost, b.stream));
    CU(cudaStreamSynchronize(b.stream));
    b.d2h_bytes += (int64_t)((3 + ntail) * W3 * sizeof(double));
    if (err) return fail(UEGCCD_ERR_ARG, "a momentum transfer falls outside the structure-factor grid");
    const double c = 2.0 * kPi / H.L, scale = c * c;
    for (int64_t z = 0; z < W; z++)
        for (int64_t y = 0; y < W; y++)
            for (int64_t x = 0; x < W; x++) {
                const int64_t k = x + W * (y + W * z);
                double g = 0.0, v = 0.0;
                if (cnt[k] > 0.0) {
                    const int q2 = (int)((x - S) * (x - S) + (y - S) * (y - S) + (z - S) * (z - S));
                    g = std::pow((double)q2 * scale, 0.5);
                    v = coulomb_v(H.L, H.madelung, q2);
                    if (b.gapii > 0.0 && v > b.gapii) v = 0.0;        // GapERI
                    if (ntail == 2 && cnt[W3 + k] != 0.0) v = 0.0;    // CoreERI of the last pair
                }
                if (out.g) out.g[k] = g;
                if (out.v) out.v[k] = v;
            }
    return UEGCCD_OK;
}

// Every call on a batch or context runs on the device the object was created on (whatever
// device the calling thread has current), and is refused once the batch is unusable.
// The two-channel state of a context, made on first use in the context's batch memory, with
// the integrals of the context's selection (uegccd_ctx_set_eri; none: SetPointers without
// range flags) for CoreN and GapII.
// A two-channel state for system s of a batch, its device memory carved from the batch's.
int make_two_channel(UegccdBatch &b, int s, std::unique_ptr<uegccd::TwoChannel> &out)
{
    struct Arena {
        UegccdBatch *b;
        UegccdBatch::Mark m;
    };
    auto ar = std::make_shared<Arena>(Arena{&b, b.mark()});
    uegccd::TcAlloc al;
    al.get = [ar](void **p, size_t bytes) {
        char *q = nullptr;
        const int rc = ar->b->alloc(q, bytes);
        *p = q;
        return rc;
    };
    al.begin = [ar]() { ar->m = ar->b->mark(); };
    al.rollback = [ar]() { ar->b->rollback(ar->m); };
    al.hold = [ar](const void *who, size_t bytes, bool *kept) -> void * {
        bool fresh = false;
        char *p = spare_hold(ar->b->tc_work, bytes, ar->b->dev, fresh);
        *kept = p && !fresh && ar->b->tc_work_user == who;
        ar->b->tc_work_user = p ? who : nullptr;
        return p;
    };
    al.rest = [ar]() { spare_rest(ar->b->tc_work); };
    if (!b.words && !(b.words = words_get())) return fail(UEGCCD_ERR_ALLOC, "no page-locked host memory");
    al.words = reinterpret_cast<double *>(b.words + kFlagBytes);
    auto tc = std::make_unique<uegccd::TwoChannel>();
    const int rc = tc->init(b.sys[s], b.plans[s], b.stream, al);
    if (rc) return rc;
    out = std::move(tc);
    return 0;
}

int two_channel_ready(UegccdCtx &c, int core_n, double gapii)
{
    if (!c.tc) {
        const int rc = make_two_channel(*c.batch, 0, c.tc);
        if (rc) return rc;
    }
    UegccdRangeTerms none{};
    const UegccdRangeTerms &fl = c.eri_set ? c.flags : none;
    const int safe = c.eri_set ? c.safe_eri : 0;
    const int routine = uegccd::tc_pick_routine(fl, safe, core_n, gapii);
    return c.tc->set_integrals(routine, fl, core_n, gapii, c.screening);
}

// A batch CCD solve in the two-channel form (do_ring != do_xring): every system in turn from its
// MP2 amplitudes, on a two-channel state of its own; the integrals of the batch's options (and
// its uniform range flag, as CasedERI applies it).  The batch keeps each solve's T2abab (what
// uegccd_batch_get_amplitudes reads) and its iteration table (uegccd_batch_history).
int run_two_channel_solves(UegccdBatch &b, const UegccdOptions *opt, UegccdResult *res)
{
    const int n = b.d.nsolves;
    if (b.tcs.size() != (size_t)n) b.tcs.resize(n);
    b.tc_en.assign(n, {});
    b.tc_dt.assign(n, {});
    UegccdRangeTerms flags{};
    int routine = uegccd::tc_pick_routine(flags, 0, opt->core_n, opt->gapii);
    if (opt->range_flags != 0) {
        int32_t *p = &flags.ring;
        for (int k = 0; k < 15; k++) p[k] = b.range_flag;
        routine = uegccd::TC_CASED;
    }
    const int max_rec = std::min(opt->max_iter, 1100);
    int status = 0;
    for (int s = 0; s < n; s++) {
        const SystemHost &H = b.sys[s];
        const size_t na = (size_t)H.O * H.O * (H.M - H.O);
        std::vector<double> aa(na), ab(na), ba(na);
        int rc = unpack_to_host(b, s, b.d.t, ab.data(), ba.data(), aa.data());
        if (rc) return rc;
        if (!b.tcs[s] && (rc = make_two_channel(b, s, b.tcs[s]))) return rc;
        if ((rc = b.tcs[s]->set_integrals(routine, flags, opt->core_n, opt->gapii, b.screening))) return rc;
        UegccdOptions o = *opt;
        b.tc_en[s].assign(max_rec, 0.0);
        b.tc_dt[s].assign(max_rec, 0.0);
        o.energies = b.tc_en[s].data();
        o.dts = b.tc_dt[s].data();
        o.max_rec = max_rec;
        rc = b.tcs[s]->solve(o, false, H.eigen, aa.data(), ab.data(), ba.data(), res[s]);
        if (rc < 0 && rc != UEGCCD_ERR_NUMERIC) return rc;
        b.tc_en[s].resize(res[s].n_recorded);
        b.tc_dt[s].resize(res[s].n_recorded);
        // the caller's arrays receive solve 0's table, as run_solves gives them
        if (s == 0 && opt->max_rec > 0) {
            const int k = std::min(res[s].n_recorded, opt->max_rec);
            if (opt->energies) std::copy(b.tc_en[s].begin(), b.tc_en[s].begin() + k, opt->energies);
            if (opt->dts) std::copy(b.tc_dt[s].begin(), b.tc_dt[s].begin() + k, opt->dts);
            res[s].n_recorded = k;
        } else {
            res[s].n_recorded = 0;
        }
        if ((rc = pack_from_host(b, s, ab.data()))) return rc;
        if (res[s].status == UEGCCD_ERR_NUMERIC) status = UEGCCD_ERR_NUMERIC;
        if (status == 0 && res[s].status == UEGCCD_NOT_CONVERGED) status = UEGCCD_NOT_CONVERGED;
    }
    b.two_channel_amps = true;
    if (status == UEGCCD_ERR_NUMERIC) fail(status, "non-finite amplitudes or energy");
    return status;
}

#define ENTER_DEVICE(bp)                                                                               \
    DeviceScope dev_scope_((bp)->dev);                                                                 \
    if (dev_scope_.rc != cudaSuccess)                                                                  \
        return fail(UEGCCD_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(dev_scope_.rc))
#define ENTER(bp)                                                                                      \
    ENTER_DEVICE(bp);                                                                                  \
    if ((bp)->broken) return fail(UEGCCD_ERR_CUDA, "batch unusable: restoring its plain integral tables failed")

extern "C" {

const char *uegccd_last_error(void) { return g_last_error.c_str(); }
const char *uegccd_version(void) { return "uegccd_b200 0.1 (sm_100a)"; }

void uegccd_default_options(UegccdOptions *o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->do_ring = o->do_xring = o->do_ladder = o->do_mosaic = 1;
    o->max_iter = 1000;
    o->tol = 1.0e-8;
    o->denom_factor = 2.0;
    o->fail_ratio = 100.0;
    o->scheme = UEGCCD_REPLAY;
    o->ndiis = 6;
    o->precision = UEGCCD_FP64;
    o->refine_sweeps = 2;
}

int uegccd_ctx_create(const UegccdSystem *sys, UegccdCtx **out)
{
    if (!out) return fail(UEGCCD_ERR_ARG, "null out");
    *out = nullptr;
    std::unique_ptr<UegccdBatch> b;
    int rc = build_batch(sys, 1, b);
    if (rc) return rc;
    auto *c = new UegccdCtx;
    c->batch = std::move(b);
    *out = c;
    return 0;
}

int uegccd_ctx_destroy(UegccdCtx *c)
{
    if (!c) return 0;
    ENTER_DEVICE(c->batch);
    delete c;
    return 0;
}

int uegccd_ctx_set_eigen(UegccdCtx *c, const double *eigen)
{
    if (!c || !eigen) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    b.sys[0].eigen.assign(eigen, eigen + b.sys[0].M);
    CU(cudaMemcpyAsync(b.d.eigen, eigen, b.sys[0].M * sizeof(double), cudaMemcpyHostToDevice, b.stream));
    CU(cudaStreamSynchronize(b.stream));
    return 0;
}

int set_range(UegccdBatch &b, int32_t flag, double screening)
{
    if (flag < 0 || flag > 3) return fail(UEGCCD_ERR_ARG, "range flag must be 0, 1, 2 or 3");
    if (flag != 0 && !(screening > 0.0)) return fail(UEGCCD_ERR_ARG, "screening distance must be > 0");
    b.range_flag = flag;
    b.screening = flag != 0 ? screening : 0.0;
    return 0;
}

int uegccd_ctx_set_range(UegccdCtx *c, int32_t flag, double screening)
{
    if (!c) return fail(UEGCCD_ERR_ARG, "null context");
    return set_range(*c->batch, flag, screening);
}

int uegccd_batch_set_range(UegccdBatch *b, int32_t flag, double screening)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    return set_range(*b, flag, screening);
}

int uegccd_ctx_set_integrals(UegccdCtx *c, int32_t core_n, double gapii)
{
    if (!c) return fail(UEGCCD_ERR_ARG, "null context");
    ENTER(c->batch);
    return set_integrals(*c->batch, core_n, gapii);
}

int uegccd_batch_set_integrals(UegccdBatch *b, int32_t core_n, double gapii)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    ENTER(b);
    return set_integrals(*b, core_n, gapii);
}

int uegccd_mp2(UegccdCtx *c, double *t_aaaa, double *t_abab, double *t_abba, double *e2)
{
    if (!c) return fail(UEGCCD_ERR_ARG, "null context");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    launch_mp2(b.d, b.stream);
    launch_reduce(b.d, b.stream);
    CU(cudaGetLastError());
    const int rc = t_aaaa || t_abab || t_abba ? unpack_to_host(b, 0, b.d.t, t_abab, t_abba, t_aaaa, true) : read_red(b);
    if (rc) return rc;
    if (e2) *e2 = b.red[0];
    return std::isfinite(b.red[0]) ? 0 : fail(UEGCCD_ERR_NUMERIC, "non-finite MP2 energy");
}

int uegccd_ccd(UegccdCtx *c, const UegccdOptions *opt, double *t_aaaa, double *t_abab, double *t_abba,
               UegccdResult *res)
{
    if (!c || !t_abab || !res) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    const bool two = opt && (c->eri_set || (opt->do_ring != 0) != (opt->do_xring != 0));
    int rc = validate_options(opt, 0, b, two);
    if (rc) return rc;
    if ((rc = set_integrals(b, opt->core_n, opt->gapii))) return rc;
    if (two) {
        if ((rc = two_channel_ready(*c, opt->core_n, opt->gapii))) return rc;
        return c->tc->solve(*opt, false, b.sys[0].eigen, t_aaaa, t_abab, t_abba, *res);
    }
    if ((rc = pack_from_host(b, 0, t_abab))) return rc;
    int st = run_solves(b, opt, 0, res);
    if (st < 0) return st;
    if ((rc = unpack_to_host(b, 0, b.d.t, t_abab, t_abba, t_aaaa))) return rc;
    return st;
}

int uegccd_drpa(UegccdCtx *c, const UegccdOptions *opt, double *t2, UegccdResult *res)
{
    if (!c || !t2 || !res) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    int rc = validate_options(opt, 1, b, c->eri_set);
    if (rc) return rc;
    if ((rc = set_integrals(b, opt->core_n, opt->gapii))) return rc;
    if (c->eri_set) {
        if ((rc = two_channel_ready(*c, opt->core_n, opt->gapii))) return rc;
        return c->tc->solve(*opt, true, b.sys[0].eigen, nullptr, t2, nullptr, *res);
    }
    if ((rc = pack_from_host(b, 0, t2))) return rc;
    int st = run_solves(b, opt, 1, res);
    if (st < 0) return st;
    if ((rc = unpack_to_host(b, 0, b.d.t, t2, nullptr, nullptr))) return rc;
    return st;
}

int uegccd_ccd_g2_ex(UegccdCtx *c, const double *t_abab, int32_t mask, int32_t precision, double *g_abab)
{
    if (!c || !t_abab || !g_abab) return fail(UEGCCD_ERR_ARG, "null argument");
    if (precision != UEGCCD_FP64 && precision != UEGCCD_MIXED) return fail(UEGCCD_ERR_ARG, "unknown precision");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    int rc = pack_from_host(b, 0, t_abab);
    if (rc) return rc;
    if ((rc = set_active_all(b, 1))) return rc;
    TermFlags f;
    f.do_driver = (mask & 1) ? 1 : 0;
    f.do_mosaic = (mask & 2) ? 1 : 0;
    f.do_ladder = (mask & 4) ? 1 : 0;
    f.do_ring = (mask & 8) ? 1 : 0;
    f.do_xring = (mask & 16) ? 1 : 0;
    DevBatch &d = b.d;
    if (precision == UEGCCD_MIXED) {
        // the tensor-core ladder of t itself: refresh point t_ref = 0, g_ref = 0
        if ((rc = mixed_alloc(b))) return rc;
        CU(cudaMemsetAsync(d.t_ref, 0, d.namp * sizeof(double), b.stream));
        CU(cudaMemsetAsync(d.g_ref, 0, d.namp * sizeof(double), b.stream));
        CU(cudaMemsetAsync(d.tc_err, 0, sizeof(int), b.stream));
        f.mixed = 1;
    }
    // G takes the ladder's place: k_update reads an amplitude's ladder value where it writes its G, and
    // none of a mirror
    launch_residual(d, f, 1, d.g, b.stream);
    CU(cudaGetLastError());
    if (precision == UEGCCD_MIXED) {
        int err = 0;
        CU(cudaMemcpyAsync(&err, d.tc_err, sizeof(int), cudaMemcpyDeviceToHost, b.stream));
        CU(cudaStreamSynchronize(b.stream));
        if (err) return fail(UEGCCD_ERR_CUDA, "tensor-core ladder: an mbarrier wait expired");
    }
    return unpack_to_host(b, 0, d.g, g_abab, nullptr, nullptr);
}

int32_t uegccd_sf_length(const UegccdSystem *sys)
{
    if (!sys || !sys->nvec || sys->nao <= 0) return fail(UEGCCD_ERR_ARG, "bad system");
    int m = sys->nvec[0];
    for (int64_t k = 0; k < 3 * (int64_t)sys->nao; k++) m = std::max(m, (int)sys->nvec[k]);
    return m * 2 + 1;
}

int uegccd_structure_factor(UegccdCtx *c, const double *t_abab, const UegccdSfGrid *out)
{
    if (!c || !t_abab || !out) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    UegccdBatch &b = *c->batch;
    int rc = pack_from_host(b, 0, t_abab);
    if (rc) return rc;
    return structure_factor(b, 0, *out);
}

int uegccd_ccd_g2(UegccdCtx *c, const double *t_abab, int32_t mask, double *g_abab)
{
    return uegccd_ccd_g2_ex(c, t_abab, mask, UEGCCD_FP64, g_abab);
}

int uegccd_ctx_set_eri(UegccdCtx *c, const UegccdRangeTerms *flags, int32_t safe_eri, double screening)
{
    if (!c) return fail(UEGCCD_ERR_ARG, "null context");
    if (!flags) {
        c->eri_set = false;
        return 0;
    }
    const int32_t *p = &flags->ring;
    bool screened = false;
    for (int k = 0; k < 15; k++) {
        if (p[k] < 0 || p[k] > 3) return fail(UEGCCD_ERR_ARG, "range flags must be 0, 1, 2 or 3");
        screened = screened || p[k] == 1 || p[k] == 2;
    }
    if (screened && !(screening > 0.0)) return fail(UEGCCD_ERR_ARG, "screening distance must be > 0");
    c->flags = *flags;
    c->safe_eri = safe_eri ? 1 : 0;
    c->screening = screening;
    c->eri_set = true;
    return 0;
}

int uegccd_ccd_g2_2ch(UegccdCtx *c, const double *t_abab, const double *t_abba, int32_t mask, double *g_abab,
                      double *g_abba)
{
    if (!c || !t_abab || !t_abba || !g_abab || !g_abba) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    int rc = two_channel_ready(*c, c->batch->core_n, c->batch->gapii);
    if (rc) return rc;
    return c->tc->ccd_g2(t_abab, t_abba, mask, g_abab, g_abba);
}

int uegccd_drpa_g2(UegccdCtx *c, const double *t2, int32_t mask, double *g2)
{
    if (!c || !t2 || !g2) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(c->batch);
    int rc = two_channel_ready(*c, c->batch->core_n, c->batch->gapii);
    if (rc) return rc;
    return c->tc->drpa_g2(t2, mask, g2);
}

int uegccd_batch_create(const UegccdSystem *systems, int32_t n, UegccdBatch **out)
{
    if (!out || !systems) return fail(UEGCCD_ERR_ARG, "null argument");
    *out = nullptr;
    std::unique_ptr<UegccdBatch> b;
    int rc = build_batch(systems, n, b);
    if (rc) return rc;
    *out = b.release();
    return 0;
}

int uegccd_batch_destroy(UegccdBatch *b)
{
    if (!b) return 0;
    ENTER_DEVICE(b);
    delete b;
    return 0;
}

int uegccd_batch_solve(UegccdBatch *b, const UegccdOptions *opt, int32_t drpa, double *e2, UegccdResult *results)
{
    if (!b || !results) return fail(UEGCCD_ERR_ARG, "null argument");
    ENTER(b);
    b->ses.on = false;   // a full solve ends an open incremental one
    const bool two = opt && !drpa && (opt->do_ring != 0) != (opt->do_xring != 0);
    if (two && opt->range_flags != 0 && b->range_flag == 0)
        return fail(UEGCCD_ERR_UNSUPPORTED, "range-separated integrals: set one flag with uegccd_batch_set_range");
    int rc = validate_options(opt, drpa, *b, two);
    if (rc) return rc;
    if ((rc = set_integrals(*b, opt->core_n, opt->gapii))) return rc;
    b->two_channel_amps = false;
    CU(cudaEventRecord(b->ev_solve0, b->stream));
    b->kt.begin(KID_MP2, b->stream);
    launch_mp2(b->d, b->stream);
    b->kt.end(b->stream);
    launch_reduce(b->d, b->stream);
    if ((rc = read_red(*b))) return rc;
    if (e2)
        for (int s = 0; s < b->d.nsolves; s++) e2[s] = b->red[3 * s];
    if (drpa) {
        // the reference starts dRPA from T2aaaa of the MP2 step (Main.f90:85-91)
        launch_to_aaaa(b->d, b->stream);
    }
    int st = two ? run_two_channel_solves(*b, opt, results) : run_solves(*b, opt, drpa, results, true);
    if (st < 0) return st;
    CU(cudaEventRecord(b->ev_solve1, b->stream));
    CU(cudaEventSynchronize(b->ev_solve1));
    float ms = 0.f;
    CU(cudaEventElapsedTime(&ms, b->ev_solve0, b->ev_solve1));
    for (int s = 0; s < b->d.nsolves; s++) results[s].gpu_ms = ms;
    return st;
}

int uegccd_batch_start(UegccdBatch *b, const UegccdOptions *opt, int32_t drpa, double *e2)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    ENTER(b);
    int rc = validate_options(opt, drpa, *b);
    if (rc) return rc;
    if (opt->precision != UEGCCD_FP64)
        return fail(UEGCCD_ERR_UNSUPPORTED, "an incremental solve runs in FP64 (use uegccd_batch_solve for MIXED)");
    if (opt->range_flags != 0)
        return fail(UEGCCD_ERR_UNSUPPORTED, "an incremental solve takes no range flags (use uegccd_batch_solve)");
    if ((rc = set_integrals(*b, opt->core_n, opt->gapii))) return rc;
    b->two_channel_amps = false;
    b->launches = 0;
    launch_mp2(b->d, b->stream);
    launch_reduce(b->d, b->stream);
    b->launches += 2;
    if ((rc = read_red(*b))) return rc;
    if (e2)
        for (int s = 0; s < b->d.nsolves; s++) e2[s] = b->red[3 * s];
    if (drpa) {
        launch_to_aaaa(b->d, b->stream);   // the dRPA start is T2aaaa of the MP2 step (Main.f90:85-91)
        b->launches++;
    }
    return session_start(*b, opt, drpa);
}

int uegccd_batch_advance(UegccdBatch *b, int32_t rounds, int32_t *n_active, int32_t *n_done, int32_t *done_ids,
                         UegccdResult *done_results)
{
    if (!b || !n_active || !n_done || !done_ids || !done_results || rounds < 0)
        return fail(UEGCCD_ERR_ARG, "bad argument");
    ENTER(b);
    *n_active = 0;
    *n_done = 0;
    if (!b->ses.on) return fail(UEGCCD_ERR_ARG, "no incremental solve is open on this batch (uegccd_batch_start)");
    return session_advance(*b, rounds, n_active, n_done, done_ids, done_results);
}

// The four ring entries of the two calls below, by the pairs a CTA of k_rings works on at a time
static constexpr int kRingShapes = 4, kRingPairs[kRingShapes] = {8, 4, 2, 1};

int32_t uegccd_batch_ring_threads(UegccdBatch *b, int32_t *threads, int32_t max)
{
    if (!b || !threads || max <= 0) return fail(UEGCCD_ERR_ARG, "bad argument");
    const int n = std::min<int>(max, kRingShapes);
    for (int c = 0; c < n; c++) threads[c] = ring_cta_threads(kRingPairs[c]);
    return n;
}

int32_t uegccd_batch_launch_shapes(UegccdBatch *b, int32_t *vals, int32_t max)
{
    if (!b || !vals || max <= 0) return fail(UEGCCD_ERR_ARG, "bad argument");
    int32_t v[kRingShapes + 3];
    for (int c = 0; c < kRingShapes; c++) v[c] = ring_cta_threads(kRingPairs[c]);
    v[kRingShapes] = b->d.stage_threads;
    v[kRingShapes + 1] = 1;   // ladder tiles: always the longest first (ladder_tiles)
    v[kRingShapes + 2] = ladder_chunk();
    const int n = std::min<int>(max, kRingShapes + 3);
    for (int k = 0; k < n; k++) vals[k] = v[k];
    return n;
}

int uegccd_batch_set_profiling(UegccdBatch *b, int32_t on)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    ENTER(b);
    if (on && !b->kt_events) {
        for (auto &e : b->kt.ev) CU(cudaEventCreate(&e));
        b->kt_events = true;
    }
    b->kt.on = on != 0;
    for (int k = 0; k < KID_COUNT; k++) { b->kt.ms[k] = 0.0; b->kt.launches[k] = 0; }
    b->drop_graphs();  // re-capture with (or without) the timer events
    return 0;
}

int32_t uegccd_batch_kernel_stats(UegccdBatch *b, int32_t max, const char **names, double *ms, int64_t *launches)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    int n = 0;
    for (int k = 0; k < KID_COUNT && n < max; k++) {
        if (b->kt.launches[k] == 0) continue;
        if (names) names[n] = kKernelNames[k];
        if (ms) ms[n] = b->kt.ms[k];
        if (launches) launches[n] = b->kt.launches[k];
        n++;
    }
    return n;
}

int uegccd_footprint(const UegccdSystem *sys, int32_t ndiis, int32_t mixed, int64_t *bytes, int64_t *namp)
{
    if (!sys || !bytes) return fail(UEGCCD_ERR_ARG, "null argument");
    SystemHost h;
    int rc = read_system(sys, h);
    if (rc) return rc;
    SolvePlan P;
    std::string msg = build_solve_plan(h, P);
    if (!msg.empty()) return fail(UEGCCD_ERR_ARG, msg);
    const int64_t A = P.namp, O = P.O, V = P.V, M = P.M;
    const int64_t nblk = (int64_t)P.blocks.size();
    int64_t b = 0;
    int64_t sum_ov = 0;
    for (const auto &B : P.blocks) sum_ov += B.o + B.v;
    b += A * (8 * 2 + sizeof(AmpInfo) + 4 + 8);      // t, g; amps; partner, ring positions
    b += sum_ov * (8 + 4) + (V + O + 1) * (4 + 8);   // mosaic partials and target lists
    b += O * O * V * 4;                              // pos
    b += O * V * 8 * 2 + O * O * 16 + nblk * V * 2;  // dRPA sums and lookups (allocated for dRPA only)
    b += O * V * (2 * 2 + 16);                       // ph rows, their lookup sides
    int64_t xy = 0;                                  // particle-hole operands and results of the rings
    for (size_t gi = 0; gi < P.groups.size(); gi++) {
        const auto &G = P.groups[gi];
        if (G.partner < 0 || G.partner < (int)gi) continue;
        const auto &H2 = P.groups[G.partner];
        const int64_t n1 = std::min(G.n, H2.n), n2 = std::max(G.n, H2.n);
        xy += n1 * 2 * ((n2 + 7) & ~7);
    }
    b += xy * 8 * 2 + O * V * 4 * 2;                 // xy, rx; ph_a, ph_b
    b += O * V * O * 4 * 2;                          // ring gather indices
    b += sum_ov * 8 + nblk * (sizeof(BlockDev) + 2 * sizeof(LadderTile64)) + M * (16 + 8) + (P.q2max + 1) * 8;
    b += A * (8 + 4) * (int64_t)std::max(0, (int)ndiis);  // DIIS history (t' FP64, e FP32)
    if (mixed) {
        b += A * 8 * 2;                              // t_ref, g_ref
        for (const auto &B : P.blocks) {             // FP16 Coulomb slabs and d tiles, row scales
            const int64_t nch = (B.v + 31) / 32, ntc = B.o <= 16 ? 16 : B.o <= 32 ? 32 : 64;
            b += ((B.v + 127) / 128) * nch * 128 * 32 * 2;
            b += ((B.o + ntc - 1) / ntc) * (nch * ntc * 32 * 2 + ntc * 4);
        }
    }
    b += (int64_t)O * O * V * 8 * 3;                 // reference-layout staging (one solve)
    *bytes = b;
    if (namp) *namp = A;
    return 0;
}

int uegccd_batch_transfer_bytes(UegccdBatch *b, int64_t *h2d, int64_t *d2h)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    if (h2d) *h2d = b->h2d_bytes;
    if (d2h) *d2h = b->d2h_bytes;
    return 0;
}

int uegccd_batch_get_amplitudes(UegccdBatch *b, int32_t s, double *t_abab)
{
    if (!b || !t_abab || s < 0 || s >= b->d.nsolves) return fail(UEGCCD_ERR_ARG, "bad argument");
    ENTER(b);
    return unpack_to_host(*b, s, b->d.t, t_abab, nullptr, nullptr);
}

int uegccd_batch_get_all_amplitudes(UegccdBatch *b, double *t_abab)
{
    if (!b || !t_abab) return fail(UEGCCD_ERR_ARG, "bad argument");
    ENTER(b);
    const int n = b->d.nsolves;
    if (!b->dense_all) {
        std::vector<int64_t> off(n + 1, 0);
        for (int s = 0; s < n; s++) off[s + 1] = off[s] + (int64_t)b->plans[s].O * b->plans[s].O * b->plans[s].V;
        int rc = b->upload(b->dense_off, off);
        if (rc) return rc;
        if ((rc = b->alloc(b->dense_all, (size_t)off[n]))) return rc;
        b->dense_all_n = (size_t)off[n];
    }
    CU(cudaMemsetAsync(b->dense_all, 0, b->dense_all_n * sizeof(double), b->stream));
    launch_unpack_all(b->d, b->dense_off, b->d.t, b->dense_all, b->stream);
    b->launches++;
    CU(cudaGetLastError());
    const size_t bytes = b->dense_all_n * sizeof(double);
    b->d2h_bytes += (int64_t)bytes;
    // Large ones into pageable memory go through page-locked memory, copied on on all host cores: the
    // driver's own staging, one thread, is as fast or faster below kCoresMin (0.36 MB 0.087 ms against
    // 0.081, 2.0 MB 0.16 against 0.20, 6.6 MB 0.42 against 0.57; 80 MB 16.7 against 4.4).
    if (bytes >= kCoresMin && !is_pinned(t_abab)) {
        std::vector<Piece> v;
        add_pieces(v, (char *)t_abab, (const char *)b->dense_all, bytes);
        return download(*b, v, true);
    }
    CU(cudaMemcpyAsync(t_abab, b->dense_all, bytes, cudaMemcpyDeviceToHost, b->stream));
    CU(cudaStreamSynchronize(b->stream));
    return UEGCCD_OK;
}

int uegccd_batch_mp2(UegccdBatch *b, double *e2)
{
    if (!b) return fail(UEGCCD_ERR_ARG, "null batch");
    ENTER(b);
    b->two_channel_amps = false;
    b->kt.begin(KID_MP2, b->stream);
    launch_mp2(b->d, b->stream);
    b->kt.end(b->stream);
    launch_reduce(b->d, b->stream);
    b->launches += 2;
    int rc = read_red(*b);
    if (rc) return rc;
    int status = UEGCCD_OK;
    for (int s = 0; s < b->d.nsolves; s++) {
        if (e2) e2[s] = b->red[3 * s];
        if (!std::isfinite(b->red[3 * s])) status = fail(UEGCCD_ERR_NUMERIC, "non-finite MP2 energy");
    }
    return status;
}

int uegccd_batch_structure_factor(UegccdBatch *b, int32_t s, const UegccdSfGrid *out)
{
    if (!b || !out || s < 0 || s >= b->d.nsolves) return fail(UEGCCD_ERR_ARG, "bad argument");
    ENTER(b);
    if (b->two_channel_amps)
        return fail(UEGCCD_ERR_UNSUPPORTED, "structure factors of two-channel amplitudes are outside the GPU path");
    return structure_factor(*b, s, *out);
}

int uegccd_trim_cache(void)
{
    pinned_trim();
    idle_trim();
    drop_spares(-1);
    std::vector<DevChunk> drop;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        drop.swap(g_pool);
        g_pool_bytes = 0;
    }
    for (auto &c : drop) {
        DeviceScope on(c.dev);
        cudaFree(c.p);
    }
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        for (auto &c : drop) g_dev_bytes[c.dev % kMaxDevices] -= (int64_t)c.size;
        g_released++;
    }
    return UEGCCD_OK;
}

int uegccd_set_memory_limit(int64_t bytes)
{
    if (bytes < 0) return fail(UEGCCD_ERR_ARG, "memory limit must be >= 0");
    std::lock_guard<std::mutex> lock(g_pool_mu);
    g_mem_limit = bytes;
    g_released++;
    return UEGCCD_OK;
}

int uegccd_memory_info(int64_t *held, int64_t *cached)
{
    const int dev = current_device() % kMaxDevices;
    std::lock_guard<std::mutex> lock(g_pool_mu);
    int64_t c = 0;
    for (const auto &x : g_pool)
        if (x.dev == dev) c += (int64_t)x.size;
    if (held) *held = g_dev_bytes[dev];
    if (cached) *cached = c;
    return UEGCCD_OK;
}

int uegccd_batch_history(UegccdBatch *b, int32_t s, double *energies, double *dts, int32_t max_rec,
                         int32_t *n_recorded)
{
    if (!b || s < 0 || s >= b->d.nsolves || max_rec < 0 || !n_recorded)
        return fail(UEGCCD_ERR_ARG, "bad argument");
    ENTER(b);
    if (b->two_channel_amps) {
        const auto &e = b->tc_en[s], &d = b->tc_dt[s];
        const int n = std::min((int)e.size(), max_rec);
        if (energies) std::copy(e.begin(), e.begin() + n, energies);
        if (dts) std::copy(d.begin(), d.begin() + n, dts);
        *n_recorded = n;
        return UEGCCD_OK;
    }
    if (b->last_niter.size() != (size_t)b->d.nsolves || !b->ctl.rec_e)
        return fail(UEGCCD_ERR_ARG, "no solve has run on this batch");
    const int n = std::min(b->last_niter[s], max_rec);
    const size_t off = (size_t)s * b->ctl.max_rec;
    if (n > 0 && energies)
        CU(cudaMemcpyAsync(energies, b->ctl.rec_e + off, n * sizeof(double), cudaMemcpyDeviceToHost, b->stream));
    if (n > 0 && dts)
        CU(cudaMemcpyAsync(dts, b->ctl.rec_dt + off, n * sizeof(double), cudaMemcpyDeviceToHost, b->stream));
    CU(cudaStreamSynchronize(b->stream));
    *n_recorded = n;
    return UEGCCD_OK;
}

}  // extern "C"
