// Results from device memory into the caller's (pageable) host arrays.
//
// cudaMemcpyAsync into pageable memory costs about 20 us a call for a few
// kilobytes, runs at 16 GB/s into a few megabytes that the allocator hands out
// again and again, and at 4.7 GB/s into a fresh large array (one thread takes
// the page faults and the copy out of the driver's staging).  So: up to SMALL
// through a pinned buffer, pieces that follow each other on the device in one
// copy; from LARGE up through pinned slots that worker threads empty -- while
// the GPU is still at work on the steps queued before, the workers touch the
// pages of the destination, so the faults are over when the data comes -- and
// directly in between.  Only ordinary host memory is staged (pageable below).
// B200 host, rho and u: 48 x 64 43 -> 28 us, 129^2
// 63 -> 45 us, 2048^2 (101 MB) 22.4 -> 4.7 ms, 4096^2 (403 MB) 86 -> 25 ms, or
// 12 ms behind queued steps; with the slots 500^2 (6 MB) would take 0.9 ms
// against 0.39 ms.
//
// Both buffers are the process's, allocated on first use and used by one call at
// a time: a call that finds one taken copies directly.  The mutex guards who has
// them and is never held while a call allocates, frees or waits for the GPU, so
// a lattice is created and destroyed on one thread while another waits for its
// results.  The small buffer stays for the process, the slots (SLOT x SLOTS
// bytes) are freed with the last lattice.
#include "llb_copyout.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace llb {

namespace {

constexpr size_t SMALL = size_t{1} << 19, LARGE = size_t{1} << 25;
constexpr size_t SLOT = size_t{1} << 20;  // bytes of a staging slot
constexpr size_t SLOTS = 8;
constexpr size_t MAX_WORKERS = 8;

// A pinned buffer of the process.
struct Staging {
    const size_t bytes;
    char* p = nullptr;
    bool taken = false;  // a call uses it, or allocates or frees it
};
std::mutex g_mu;  // guards the two below and the count of lattices
Staging g_small{SMALL}, g_slots{SLOT * SLOTS};
int g_users = 0;

void give_back(Staging& s) {
    std::lock_guard<std::mutex> lk(g_mu);
    s.taken = false;
}

// The buffer for one call, allocated if it is not there; null if another call
// has it or no pinned memory can be had.
char* take(Staging& s) {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (s.taken) return nullptr;
        s.taken = true;
    }
    if (!s.p && cudaHostAlloc(reinterpret_cast<void**>(&s.p), s.bytes, cudaHostAllocPortable) != cudaSuccess) {
        (void)cudaGetLastError();
        s.p = nullptr;
        give_back(s);
        return nullptr;
    }
    return s.p;
}

struct Piece {
    char* dst;
    const char* src;
    size_t bytes;
};

void touch(char* p, size_t bytes) {
    for (size_t o = 0; o < bytes; o += 4096) {
        volatile char* q = p + o;
        *q = *q;
    }
}

// Whether p is ordinary host memory, which the staging is for.  Memory that CUDA
// knows (pinned, managed, on a device) takes a copy as it is: pinned memory one
// DMA (2048^2, 101 MB: 1.8 ms, 4.0 through the slots), and a device's memory
// cannot be written by the host.
bool pageable(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type == cudaMemoryTypeUnregistered;
    (void)cudaGetLastError();
    return false;
}

cudaError_t direct(cudaStream_t stream, const HostCopy* c, int n) {
    for (int q = 0; q < n; ++q)
        if (cudaError_t e = cudaMemcpyAsync(c[q].dst, c[q].src, c[q].bytes, cudaMemcpyDeviceToHost, stream);
            e != cudaSuccess)
            return e;
    return cudaStreamSynchronize(stream);
}

cudaError_t small(cudaStream_t stream, const HostCopy* c, int n, char* stage) {
    size_t at = 0;
    for (int q = 0; q < n;) {
        size_t bytes = c[q].bytes;
        int r = q + 1;
        while (r < n && static_cast<const char*>(c[q].src) + bytes == c[r].src) bytes += c[r++].bytes;
        if (cudaError_t e = cudaMemcpyAsync(stage + at, c[q].src, bytes, cudaMemcpyDeviceToHost, stream);
            e != cudaSuccess)
            return e;
        at += bytes;
        q = r;
    }
    if (cudaError_t e = cudaStreamSynchronize(stream); e != cudaSuccess) return e;
    at = 0;
    for (int q = 0; q < n; ++q) {
        std::memcpy(c[q].dst, stage + at, c[q].bytes);
        at += c[q].bytes;
    }
    return cudaSuccess;
}

// The calling thread feeds the copy engine and waits for it, slot by slot in
// turn; worker w moves pieces w, w + W, ... on and makes no CUDA call.  Until the
// first piece is there, which may be seconds of queued steps away, the workers
// sleep (2048^2 behind 10000 steps: 1.1 processors busy, 9.0 when they polled);
// after it the pieces follow every 20 us, and they poll.
cudaError_t large(cudaStream_t stream, const std::vector<Piece>& pieces, int workers, char* slots) {
    const size_t n = pieces.size();
    std::atomic<size_t> ready{0};  // pieces in their slots, in order
    std::atomic<bool> stop{false};
    std::mutex mu;
    std::condition_variable first;  // the first piece is there, or stop
    std::unique_ptr<std::atomic<bool>[]> done(new std::atomic<bool>[n]);
    for (size_t q = 0; q < n; ++q) done[q].store(false, std::memory_order_relaxed);
    auto slot = [slots](size_t q) { return slots + (q % SLOTS) * SLOT; };
    std::vector<std::thread> pool;
    pool.reserve(static_cast<size_t>(workers));  // (from here on nothing throws out of the call)
    cudaEvent_t ev[SLOTS] = {};
    cudaError_t e = cudaSuccess;
    auto issue = [&](size_t q) {
        if (!ev[q % SLOTS]) e = cudaEventCreateWithFlags(&ev[q % SLOTS], cudaEventDisableTiming);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(slot(q), pieces[q].src, pieces[q].bytes, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(ev[q % SLOTS], stream);
    };
    for (size_t q = 0; q < n && q < SLOTS && e == cudaSuccess; ++q) issue(q);

    auto work = [&](size_t w) {
        const size_t step = static_cast<size_t>(workers);
        for (size_t q = w; q < n; q += step) touch(pieces[q].dst, pieces[q].bytes);  // while the stream works
        {
            std::unique_lock<std::mutex> lk(mu);
            first.wait(lk, [&] { return ready.load() > 0 || stop.load(); });
        }
        for (size_t q = w; q < n; q += step) {
            while (ready.load(std::memory_order_acquire) <= q) {
                if (stop.load(std::memory_order_relaxed)) return;
                std::this_thread::yield();
            }
            std::memcpy(pieces[q].dst, slot(q), pieces[q].bytes);
            done[q].store(true, std::memory_order_release);
        }
    };
    int started = 0;
    try {
        for (; started < workers; ++started) pool.emplace_back(work, static_cast<size_t>(started));
    } catch (...) {
        // a worker whose thread could not start: its pieces are moved here
    }
    auto move_here = [&](size_t q) {
        if (static_cast<int>(q % static_cast<size_t>(workers)) < started) return;
        std::memcpy(pieces[q].dst, slot(q), pieces[q].bytes);
        done[q].store(true, std::memory_order_release);
    };
    auto wait_done = [&](size_t q) {
        while (!done[q].load(std::memory_order_acquire)) std::this_thread::yield();
    };
    constexpr size_t LAG = SLOTS / 2;  // a slot is refilled this many pieces after it arrived
    for (size_t q = 0; q < n && e == cudaSuccess; ++q) {
        e = cudaEventSynchronize(ev[q % SLOTS]);
        if (e != cudaSuccess) break;
        if (q == 0) {
            {
                std::lock_guard<std::mutex> lk(mu);
                ready.store(1);
            }
            first.notify_all();
        } else {
            ready.store(q + 1, std::memory_order_release);
        }
        move_here(q);
        if (q >= LAG && q - LAG + SLOTS < n) {
            wait_done(q - LAG);
            issue(q - LAG + SLOTS);
        }
    }
    if (e != cudaSuccess) {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop.store(true);
        }
        first.notify_all();
    }
    for (auto& t : pool) t.join();
    for (auto& v : ev)
        if (v) cudaEventDestroy(v);
    const cudaError_t s = cudaStreamSynchronize(stream);  // no copy into the slots outlives the call
    return e != cudaSuccess ? e : s;
}

}  // namespace

cudaError_t copy_to_host(cudaStream_t stream, const HostCopy* c, int n) {
    size_t total = 0;
    for (int q = 0; q < n; ++q) total += c[q].bytes;
    if (total > SMALL && total < LARGE) return direct(stream, c, n);
    for (int q = 0; q < n; ++q)
        if (!pageable(c[q].dst)) return direct(stream, c, n);
    Staging& stage = total <= SMALL ? g_small : g_slots;
    char* const buf = take(stage);
    if (!buf) return direct(stream, c, n);
    cudaError_t e;
    try {
        if (total <= SMALL) {
            e = small(stream, c, n, buf);
        } else {
            std::vector<Piece> pieces;
            for (int q = 0; q < n; ++q)
                for (size_t o = 0; o < c[q].bytes; o += SLOT)
                    pieces.push_back({static_cast<char*>(c[q].dst) + o, static_cast<const char*>(c[q].src) + o,
                                      std::min(SLOT, c[q].bytes - o)});
            const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
            const int workers =
                static_cast<int>(std::min<size_t>({MAX_WORKERS, static_cast<size_t>(hw), pieces.size()}));
            e = large(stream, pieces, workers, buf);
        }
    } catch (const std::bad_alloc&) {
        e = direct(stream, c, n);
    }
    give_back(stage);
    return e;
}

void staging_add_user() {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        ++g_users;
    }
    if (take(g_small)) give_back(g_small);
}

void staging_drop_user() {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (--g_users > 0 || g_slots.taken || !g_slots.p) return;
        g_slots.taken = true;
    }
    cudaFreeHost(g_slots.p);
    g_slots.p = nullptr;
    give_back(g_slots);
}

}  // namespace llb
