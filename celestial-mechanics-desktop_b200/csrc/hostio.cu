// hostio.cu - copies between the caller's pageable arrays and the device.
//
// The seam's arrays are ordinary pageable memory (C# arrays, numpy arrays).
// cudaMemcpyAsync stages such copies through its own pinned memory with one
// thread: 10 GB/s up and 19 GB/s down on the measured host, less into pages
// that were never touched (4 GB/s), where pinned memory moves at 50 GB/s.
//   * A small transfer (all arrays within a handle's pinned half) is packed by
//     the calling thread and sent row by row, or as one 2-D copy where the
//     device rows are evenly spaced: no lock, no thread, one synchronisation
//     per call.
//   * A large one is cut into chunks that a pool of threads moves through a
//     ring of pinned slots, so the host copies run side by side and overlap
//     the bus.  There is one pool per device; its threads (at most kMaxThreads)
//     and the first of its slots (up to kSlots MB pinned) come when kPoolAfter
//     bytes have gone the plain way, and go with the device's last handle.  A
//     transfer holds the pool for itself; when another thread's transfer has it,
//     the plain copy is used instead, so handles never wait for each other.
// Before -> now, by these transfers: forces of 2^20 bodies 11.8 -> 8.7 ms a call
// (5.4 of them on the GPU) and of 1,000 bodies 136 -> 82 us; read-backs into new
// arrays, of 2^20 bodies' state 35 -> 2.3 ms and of an ensemble's 804,337 bodies
// 19 -> 1.5 ms.  A closed handle's pinned buffer waits for the next handle.
#include "hostio.cuh"

#include <sched.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace nb {

namespace {

constexpr int kSlots = 16;
constexpr size_t kSlotBytes = 1 << 20;
constexpr size_t kMinChunk = 128 << 10;
constexpr int kMaxThreads = 7;  // besides the calling one, and of half the CPUs
constexpr int kMinThreads = 2;
constexpr size_t kRowAlign = 256;
// The pool takes transfers from these sizes on.  Up, the driver's own staging
// keeps pace with the pool while the arrays come from the caches, and to some
// 20 MB where they do not (plain / pool, ms, caller's arrays hot: 8 MB 0.44 / 0.92,
// 16 MB 0.94 / 1.3, 24 MB 1.23 / 1.53, 28 MB 1.6 / 1.5, 48 MB 2.7 / 2.2, 96 MB
// 8.4 / 3.3; cold: 8 MB 0.7 / 0.9, 16 MB 1.3 / 1.4, 24 MB 2.0 / 1.7, 48 MB 4.3 / 2.4).
// Down the pool is ahead from 1 MB on (2 MB 0.27 / 0.18, 12 MB 0.97 / 0.43, 96 MB
// 5.7 / 2.2).
constexpr size_t kPoolUp = 28 << 20, kPoolDown = 2 << 20;
// The slots come once a program has moved this much by plain copies: one that
// moves less never pays for them.  They come a few at a time, so that the call
// that gets the first (and the threads) is held up by some 2 ms and the six after
// it by 0.6 (all 16 MB at once by cudaHostAlloc took 7 to 20).
constexpr size_t kPoolAfter = 32 << 20;
constexpr int kBlockSlots = 2;  // pinned together: one huge page
constexpr int kFirstSlots = 2 * kBlockSlots, kMoreSlots = kBlockSlots;
static_assert(kSlots % kBlockSlots == 0, "whole blocks");
constexpr size_t kPage = 4096, kHugePage = 2 << 20, kHugeFrom = 512 << 10;
constexpr size_t kMaxSpare = 8;

// A handle's pinned memory: two halves and kHostExtra bytes.
struct PinBuf {
    char* p;
    size_t half;
};

struct Chunk {
    char* dst;
    const char* src;
    size_t bytes;
};

// Pinned memory as ordinary pages that are registered, huge ones from kHugeFrom
// bytes on: 0.4 to 0.7 ms for the 230 KB of a 1,000-body handle, 0.45 ms for 1 or
// 2 MB (1.3 and 2 without huge pages), where cudaHostAlloc takes 1.3 to 3 ms for
// any of them unless other pinned memory is about (ms to create a handle for
// 1,000 bodies: 4.2 without pinned memory, 4.9 so, 6.5 that way).  A child process
// does not inherit them: a fork would otherwise have the parent write to copies
// of the pages while the device keeps to the old ones, where the kernel does
// not look after registered pages itself.
size_t mapped(size_t bytes) {
    return bytes < kHugeFrom ? bytes : (bytes + kHugePage - 1) / kHugePage * kHugePage;
}

char* pin(size_t bytes) {
    const size_t size = mapped(bytes);
    const size_t slack = bytes < kHugeFrom ? 0 : kHugePage;  // to start at a huge page
    char* p = (char*)mmap(nullptr, size + slack, PROT_READ | PROT_WRITE,
                          MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) return nullptr;
    if (slack) {
        const size_t head = (kHugePage - (size_t)p % kHugePage) % kHugePage;
        if (head) munmap(p, head);
        if (slack > head) munmap(p + head + size, slack - head);
        p += head;
        madvise(p, size, MADV_HUGEPAGE);  // where the kernel has none: small pages
    }
    if (madvise(p, size, MADV_DONTFORK) != 0 ||
        cudaHostRegister(p, bytes, cudaHostRegisterDefault) != cudaSuccess) {
        cudaGetLastError();
        munmap(p, size);
        return nullptr;
    }
    return p;
}

void unpin(char* p, size_t bytes) {
    if (!p) return;
    cudaHostUnregister(p);
    munmap(p, mapped(bytes));
}

size_t pin_bytes(size_t half) { return 2 * half + kHostExtra; }

// CPUs this process may run on.
int cpus_here() {
    cpu_set_t set;
    if (sched_getaffinity(0, sizeof(set), &set) == 0) return CPU_COUNT(&set);
    return (int)std::thread::hardware_concurrency();
}

}  // namespace

struct CopyPool {
    int device = 0;
    int users = 0;
    std::vector<PinBuf> spare;  // closed handles' pinned buffers (under g_pools_lock)
    int slots = 0;              // that are there (under busy)
    bool full = false;          // no more to be had (under busy)
    char* buf[kSlots] = {};
    cudaEvent_t ev[kSlots] = {};
    bool pending[kSlots] = {};  // an upload's copy out of the slot may still run
    std::mutex busy;            // held for a transfer
    // the transfer under way
    std::vector<Chunk> chunks;
    bool up = false;
    cudaStream_t st = nullptr;
    std::atomic<int> next{0};
    std::atomic<int> turn[kSlots];
    std::atomic<int> failed{0};
    // threads
    std::mutex m;
    std::condition_variable wake, rest;
    std::vector<std::thread> threads;
    unsigned long long job = 0;
    bool open = false;  // the job still takes threads
    int inside = 0;     // threads at work on it
    bool stop = false;
    size_t moved = 0;   // bytes that went the plain way before the slots (under busy)

    // Chunk c goes through slot c % slots when the slot's earlier chunks have
    // left it (up: its copy was enqueued, and its event says when it ended;
    // down: its data is in the host array).
    void work() {
        for (;;) {
            const int c = next.fetch_add(1);
            if (c >= (int)chunks.size()) return;
            const int slot = c % slots, my_turn = c / slots;
            char* const own = buf[slot];
            while (turn[slot].load(std::memory_order_acquire) != my_turn) std::this_thread::yield();
            cudaError_t e = cudaSuccess;
            if (pending[slot]) {
                e = cudaEventSynchronize(ev[slot]);
                pending[slot] = false;
            }
            const Chunk& k = chunks[c];
            if (up) {
                std::memcpy(own, k.src, k.bytes);
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(k.dst, own, k.bytes, cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[slot], st);
                pending[slot] = true;
            } else {
                if (e == cudaSuccess)
                    e = cudaMemcpyAsync(own, k.src, k.bytes, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[slot], st);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[slot]);
                if (e == cudaSuccess) std::memcpy(k.dst, own, k.bytes);
            }
            if (e != cudaSuccess) failed.store((int)e);
            turn[slot].store(my_turn + 1, std::memory_order_release);
        }
    }

    void loop() {
        cudaSetDevice(device);
        unsigned long long seen = 0;
        std::unique_lock<std::mutex> lk(m);
        for (;;) {
            // (more threads than slots would only wait for one another)
            wake.wait(lk, [&] { return stop || (open && job != seen && inside < slots - 1); });
            if (stop) return;
            seen = job;
            inside++;
            lk.unlock();
            work();
            lk.lock();
            if (--inside == 0) rest.notify_one();
        }
    }

    // `count` more slots, in blocks (busy held).
    void grow(int count) {
        // another thread of the program may be capturing a graph
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        for (; count > 0 && slots < kSlots && !full; count -= kBlockSlots) {
            char* block = pin(kBlockSlots * kSlotBytes);
            bool ok = block != nullptr;
            for (int k = slots; ok && k < slots + kBlockSlots; k++)
                ok = ev[k] || cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) == cudaSuccess;
            if (ok) {
                for (int k = 0; k < kBlockSlots; k++) buf[slots++] = block + k * kSlotBytes;
            } else {
                cudaGetLastError();
                unpin(block, kBlockSlots * kSlotBytes);
                full = true;
            }
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }

    // Slots and threads, once kPoolAfter bytes have gone without (busy held).  A
    // pool of one or two threads moves no more than the plain copy does: false
    // then, and where there is no pinned memory to be had.
    bool ready(size_t total) {
        const int want = std::min(kMaxThreads, cpus_here() / 2 - 1);
        if (want < kMinThreads) return false;
        if (slots == 0) {
            moved += total;
            if (moved < kPoolAfter) return false;
        }
        grow(slots ? kMoreSlots : kFirstSlots);
        if (slots < kFirstSlots) return false;
        try {
            if (threads.empty())
                for (int k = 0; k < want; k++) threads.emplace_back([this] { loop(); });
        } catch (...) {
            // fewer threads, or none: the calling thread does the rest
        }
        return (int)threads.size() >= kMinThreads;
    }

    // The whole transfer, with `busy` held.  Returns when every host array has
    // been read or written.
    cudaError_t run(bool upward, cudaStream_t stream, const CopySeg* seg, int n, size_t total) {
        const size_t parts = 2 * std::min(threads.size() + 1, (size_t)slots);
        const size_t want = std::min(kSlotBytes, std::max(kMinChunk, total / parts));
        const size_t chunk = (want + 4095) / 4096 * 4096;
        chunks.clear();
        for (int i = 0; i < n; i++)
            for (size_t o = 0; o < seg[i].bytes; o += chunk)
                chunks.push_back({(char*)seg[i].dst + o, (const char*)seg[i].src + o,
                                  std::min(chunk, seg[i].bytes - o)});
        up = upward;
        st = stream;
        next.store(0);
        failed.store(0);
        for (auto& t : turn) t.store(0);
        {
            std::lock_guard<std::mutex> lk(m);
            open = true;
            job++;
        }
        wake.notify_all();
        work();
        // a thread that only wakes now has nothing to do here any more
        std::unique_lock<std::mutex> lk(m);
        open = false;
        rest.wait(lk, [&] { return inside == 0; });
        return (cudaError_t)failed.load();
    }
};

namespace {

std::mutex g_pools_lock;
std::vector<CopyPool*> g_pools;

void pool_destroy(CopyPool* p) {
    {
        std::lock_guard<std::mutex> lk(p->m);
        p->stop = true;
        p->wake.notify_all();
    }
    for (auto& t : p->threads) t.join();
    for (int k = 0; k < kSlots; k++)
        if (p->ev[k]) {
            if (p->pending[k]) cudaEventSynchronize(p->ev[k]);
            cudaEventDestroy(p->ev[k]);
        }
    for (const PinBuf& b : p->spare) unpin(b.p, pin_bytes(b.half));
    for (int k = 0; k < p->slots; k += kBlockSlots) unpin(p->buf[k], kBlockSlots * kSlotBytes);
    delete p;
}

CopyPool* pool_acquire(int device) {
    std::lock_guard<std::mutex> lk(g_pools_lock);
    for (CopyPool* p : g_pools)
        if (p->device == device) {
            p->users++;
            return p;
        }
    CopyPool* p = new (std::nothrow) CopyPool();
    if (!p) return nullptr;
    p->device = device;
    p->users = 1;
    try {
        p->spare.reserve(kMaxSpare);
        g_pools.push_back(p);
    } catch (...) {
        pool_destroy(p);
        return nullptr;
    }
    return p;
}

void pool_release(CopyPool* p) {
    std::lock_guard<std::mutex> lk(g_pools_lock);
    if (--p->users > 0) return;
    g_pools.erase(std::find(g_pools.begin(), g_pools.end(), p));
    pool_destroy(p);
}

size_t padded(size_t b) { return (b + kRowAlign - 1) / kRowAlign * kRowAlign; }

// Runs of equal rows whose device addresses are evenly spaced go as one 2-D
// copy: f(first, rows, device pitch).
template <typename F>
cudaError_t for_runs(const CopySeg* seg, int n, bool up, F f) {
    auto dev = [&](int i) { return up ? (const char*)seg[i].dst : (const char*)seg[i].src; };
    for (int i = 0; i < n;) {
        int rows = 1;
        ptrdiff_t pitch = 0;
        while (i + rows < n && seg[i + rows].bytes == seg[i].bytes) {
            const ptrdiff_t d = dev(i + rows) - dev(i + rows - 1);
            if (rows == 1 && d >= (ptrdiff_t)seg[i].bytes) pitch = d;
            if (d != pitch || pitch == 0 || pitch > 0x7FFFFFFF) break;
            rows++;
        }
        const cudaError_t e = f(i, rows, (size_t)pitch);
        if (e != cudaSuccess) return e;
        i += rows;
    }
    return cudaSuccess;
}

size_t total_bytes(const CopySeg* seg, int n) {
    size_t t = 0;
    for (int i = 0; i < n; i++) t += seg[i].bytes;
    return t;
}

size_t packed_bytes(const CopySeg* seg, int n) {
    size_t t = 0;
    for (int i = 0; i < n; i++) t += padded(seg[i].bytes);
    return t;
}

}  // namespace

bool hostio_init(HostIO& io, int device, int rows, size_t row_bytes) {
    try {
        io.pool = pool_acquire(device);
    } catch (...) {
        io.pool = nullptr;
    }
    const size_t all = (rows * padded(row_bytes) + kPage - 1) / kPage * kPage;
    io.half = std::min(kHalfBytes, all);
    if (io.pool && io.half) {
        std::lock_guard<std::mutex> lk(g_pools_lock);
        auto& spare = io.pool->spare;
        const auto fit = std::find_if(spare.begin(), spare.end(),
                                      [&](const PinBuf& b) { return b.half >= io.half; });
        if (fit != spare.end()) {
            io.pin = fit->p;
            io.half = fit->half;
            spare.erase(fit);
        }
    }
    if (!io.pin && io.half) io.pin = pin(pin_bytes(io.half));
    if (!io.pin) {
        // none wanted or none to be had: every array takes the plain copy, and
        // the handle's own bytes are ordinary memory
        io.half = 0;
        io.pin = (char*)malloc(kHostExtra);
    }
    return io.pin != nullptr;
}

void hostio_free(HostIO& io) {
    if (io.half == 0) {
        free(io.pin);
        io.pin = nullptr;
    }
    if (io.pin && io.pool) {
        std::lock_guard<std::mutex> lk(g_pools_lock);
        auto& spare = io.pool->spare;
        if (spare.size() < kMaxSpare) {
            spare.push_back({io.pin, io.half});  // capacity was reserved
            io.pin = nullptr;
        }
    }
    unpin(io.pin, pin_bytes(io.half));
    if (io.pool) pool_release(io.pool);
    io = HostIO();
}

namespace {

// An array the caller pinned moves at the bus rate by itself; through the
// slots 2^20 bodies' forces from pinned arrays took 5.3 ms instead of 3.8.
bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// The pageable arrays of a large transfer through the pool, if it is there and
// free, the others by plain copies; false: nothing was done.  Nothing is
// thrown on.
bool by_pool(HostIO& io, bool up, cudaStream_t st, const CopySeg* seg, int n, cudaError_t* e) {
    const size_t least = up ? kPoolUp : kPoolDown;
    if (!io.pool || total_bytes(seg, n) < least) return false;
    try {
        std::vector<CopySeg> own, rest;
        for (int i = 0; i < n; i++)
            (pageable(up ? seg[i].src : seg[i].dst) ? rest : own).push_back(seg[i]);
        const size_t total = total_bytes(rest.data(), (int)rest.size());
        if (total < least) return false;
        std::unique_lock<std::mutex> lk(io.pool->busy, std::try_to_lock);
        if (!lk.owns_lock() || !io.pool->ready(total)) return false;
        for (const CopySeg& k : own) {
            *e = cudaMemcpyAsync(k.dst, k.src, k.bytes,
                                 up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st);
            if (*e != cudaSuccess) return true;
        }
        *e = io.pool->run(up, st, rest.data(), (int)rest.size(), total);
        if (!up && !own.empty() && *e == cudaSuccess) *e = cudaStreamSynchronize(st);
        return true;
    } catch (...) {
        return false;
    }
}

}  // namespace

cudaError_t copy_up(HostIO& io, cudaStream_t st, const CopySeg* seg, int n) {
    cudaError_t e = cudaSuccess;
    if (packed_bytes(seg, n) <= io.half) {
        char* p = io.pin;
        return for_runs(seg, n, true, [&](int first, int rows, size_t pitch) {
            const size_t b = seg[first].bytes, hp = padded(b);
            char* q = p;
            for (int k = 0; k < rows; k++) std::memcpy(q + k * hp, seg[first + k].src, b);
            p += rows * hp;
            if (rows == 1) return cudaMemcpyAsync(seg[first].dst, q, b, cudaMemcpyHostToDevice, st);
            return cudaMemcpy2DAsync(seg[first].dst, pitch, q, hp, b, rows, cudaMemcpyHostToDevice, st);
        });
    }
    if (by_pool(io, true, st, seg, n, &e)) return e;
    for (int i = 0; i < n && e == cudaSuccess; i++)
        e = cudaMemcpyAsync(seg[i].dst, seg[i].src, seg[i].bytes, cudaMemcpyHostToDevice, st);
    return e;
}

cudaError_t start_down(HostIO& io, cudaStream_t st, const CopySeg* seg, int n, bool* queued) {
    *queued = packed_bytes(seg, n) <= io.half;
    if (!*queued) return cudaSuccess;
    char* p = io.pin + io.half;
    return for_runs(seg, n, false, [&](int first, int rows, size_t pitch) {
        const size_t b = seg[first].bytes, hp = padded(b);
        char* q = p;
        p += rows * hp;
        if (rows == 1) return cudaMemcpyAsync(q, seg[first].src, b, cudaMemcpyDeviceToHost, st);
        return cudaMemcpy2DAsync(q, hp, seg[first].src, pitch, b, rows, cudaMemcpyDeviceToHost, st);
    });
}

cudaError_t finish_down(HostIO& io, cudaStream_t st, const CopySeg* seg, int n, bool queued) {
    if (queued) {
        const char* p = io.pin + io.half;
        for (int i = 0; i < n; i++) {
            std::memcpy(seg[i].dst, p, seg[i].bytes);
            p += padded(seg[i].bytes);
        }
        return cudaSuccess;
    }
    cudaError_t e = cudaSuccess;
    if (by_pool(io, false, st, seg, n, &e)) return e;
    for (int i = 0; i < n && e == cudaSuccess; i++)
        e = cudaMemcpyAsync(seg[i].dst, seg[i].src, seg[i].bytes, cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

}  // namespace nb
