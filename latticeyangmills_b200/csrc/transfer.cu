// Transfers of pageable host memory through pinned slots, filled and emptied
// by several threads.
//
// The driver copies pageable memory through its own pinned buffer with one
// thread, about 10 GB/s; a fresh destination also takes its page faults on that
// thread.  Here up to kMaxWorkers threads each move every n-th chunk through
// two pinned slots of their own, so the copies to and from the slots (and the
// page faults) run side by side while the DMA engine moves other chunks.  On a
// B200 host with 16 cores, upload of a field in the .bin layout / download into
// a fresh array / into one whose pages are there: 75.5 MB 6.6-7.3 / 15-16 / 3.9-4.9
// -> 2.2-2.4 / 3.6-4.7 / 2.5-3.0 ms, 604 MB 55-59 / 121-127 / 32-36 -> 14 / 35-38 /
// 19-24 ms (604 MB in chunks of 2 MB 13 and, fresh, 36, of 512 KB 20 and 43, at 32
// and 8 MB of slots).
//
// Transfers below kDirectBytes, from or to memory that is pinned already, and
// those that find the slots in use by another thread's transfer go to the
// driver as they are.  The slots (kMaxWorkers x 2 x kChunk = 16 MiB) are
// allocated when the transfers have earned them and freed with the last
// context.
#include "transfer.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <type_traits>

namespace ym {

namespace {

constexpr size_t kChunk = size_t(1) << 20;
constexpr int kMaxWorkers = 8;
constexpr size_t kDirectBytes = size_t(16) << 20;
// Allocating the slots takes about 7 ms.  They are allocated once the transfers
// that could have used them add up to this; a downloaded byte, which saves
// three times as much, counts three times.
constexpr size_t kEarnSlots = size_t(128) << 20;

struct Slots {
    std::mutex users_mu;
    int users = 0;
    std::mutex busy;  // held by the transfer that uses the slots
    char* base = nullptr;
    size_t earned = 0;     // see kEarnSlots
};

// Neither allocated (its first user is a C entry) nor destroyed (contexts may
// outlive static destruction).
static_assert(std::is_trivially_destructible<Slots>::value, "Slots outlives static destruction");
Slots g_slots;
Slots& slots() { return g_slots; }

bool pinned_or_device(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;  // let the copy itself report it
    }
    return a.type != cudaMemoryTypeUnregistered;
}

int workers_for(size_t bytes) {
    const int cores = int(std::thread::hardware_concurrency());
    const int chunks = int(std::min<size_t>((bytes + kChunk - 1) / kChunk, size_t(kMaxWorkers)));
    return std::max(1, std::min({kMaxWorkers, cores / 2, chunks}));
}

// Ends a worker's use of its slots: they are free for the next transfer once the
// copies of its last two events are done, or, after an error, whatever the
// stream holds (the failed call may have been the record of a copy's event).
cudaError_t release_slots(cudaEvent_t done[2], cudaStream_t st, cudaError_t e) {
    if (e != cudaSuccess) cudaStreamSynchronize(st);
    for (int i = 0; i < 2; i++) {
        if (!done[i]) continue;
        const cudaError_t r = cudaEventSynchronize(done[i]);
        if (e == cudaSuccess) e = r;
        cudaEventDestroy(done[i]);
    }
    return e;
}

// One worker's chunks (w, w + n, w + 2 n, ...) of an upload.
cudaError_t upload_chunks(int device, char* dev, const char* host, size_t bytes, cudaStream_t st, char* slot, int w,
                          int n) {
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t done[2] = {nullptr, nullptr};
    for (int i = 0; i < 2 && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    int k = 0;
    for (size_t off = size_t(w) * kChunk; off < bytes && e == cudaSuccess; off += size_t(n) * kChunk, k++) {
        const size_t m = std::min(kChunk, bytes - off);
        char* const p = slot + size_t(k & 1) * kChunk;
        if (k >= 2) e = cudaEventSynchronize(done[k & 1]);
        if (e != cudaSuccess) break;
        std::memcpy(p, host + off, m);
        e = cudaMemcpyAsync(dev + off, p, m, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(done[k & 1], st);
    }
    return release_slots(done, st, e);
}

// One worker's chunks of a download.
cudaError_t download_chunks(int device, char* host, const char* dev, size_t bytes, cudaStream_t st, char* slot, int w,
                            int n) {
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t done[2] = {nullptr, nullptr};
    for (int i = 0; i < 2 && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming);
    const size_t step = size_t(n) * kChunk, first = size_t(w) * kChunk;
    auto fetch = [&](size_t off, int b) {
        const size_t m = std::min(kChunk, bytes - off);
        const cudaError_t r = cudaMemcpyAsync(slot + size_t(b) * kChunk, dev + off, m, cudaMemcpyDeviceToHost, st);
        return r == cudaSuccess ? cudaEventRecord(done[b], st) : r;
    };
    if (e == cudaSuccess && first < bytes) e = fetch(first, 0);
    int k = 0;
    for (size_t off = first; off < bytes && e == cudaSuccess; off += step, k++) {
        if (off + step < bytes) e = fetch(off + step, (k + 1) & 1);
        if (e == cudaSuccess) e = cudaEventSynchronize(done[k & 1]);
        if (e == cudaSuccess) std::memcpy(host + off, slot + size_t(k & 1) * kChunk, std::min(kChunk, bytes - off));
    }
    return release_slots(done, st, e);  // a fetch in flight still writes its slot
}

// Runs chunks(w, n) on n workers, the calling thread among them; a thread that
// cannot be started, for want of a thread or of memory, leaves its share to the
// caller: no exception leaves through the C entries.
template <class Chunks>
cudaError_t on_workers(int n, const Chunks& chunks) {
    std::thread threads[kMaxWorkers];
    std::atomic<int> error{int(cudaSuccess)};
    auto work = [&](int w) {
        const cudaError_t e = chunks(w, n);
        if (e != cudaSuccess) error.store(int(e));
    };
    for (int w = 1; w < n; w++) {
        try {
            threads[w] = std::thread(work, w);
        } catch (const std::system_error&) {
        } catch (const std::bad_alloc&) {
        }
    }
    work(0);
    for (int w = 1; w < n; w++) {
        if (threads[w].joinable())
            threads[w].join();
        else
            work(w);
    }
    return cudaError_t(error.load());
}

// The slots, held, for a transfer that goes through them; null: copy directly.
std::unique_lock<std::mutex> take_slots(const void* host, size_t bytes, size_t weight) {
    std::unique_lock<std::mutex> none;
    if (bytes < kDirectBytes || pinned_or_device(host)) return none;
    std::unique_lock<std::mutex> held(slots().busy, std::try_to_lock);
    if (!held) return none;
    if (!slots().base && (slots().earned += weight * bytes) < kEarnSlots) return none;
    if (!slots().base &&
        cudaHostAlloc((void**)&slots().base, size_t(kMaxWorkers) * 2 * kChunk, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        slots().base = nullptr;
        return none;
    }
    return held;
}

}  // namespace

void transfer_retain() {
    std::lock_guard<std::mutex> lk(slots().users_mu);
    slots().users++;
}

void transfer_release() {
    std::lock_guard<std::mutex> lk(slots().users_mu);
    if (--slots().users > 0) return;
    std::lock_guard<std::mutex> held(slots().busy);
    if (slots().base) cudaFreeHost(slots().base);
    slots().base = nullptr;
    slots().earned = 0;
}

cudaError_t transfer_upload(int device, void* dev, const void* host, size_t bytes, cudaStream_t st) {
    const std::unique_lock<std::mutex> held = take_slots(host, bytes, 1);
    if (!held) return cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st);
    char* const base = slots().base;
    return on_workers(workers_for(bytes), [=](int w, int n) {
        return upload_chunks(device, static_cast<char*>(dev), static_cast<const char*>(host), bytes, st,
                             base + size_t(w) * 2 * kChunk, w, n);
    });
}

cudaError_t transfer_download(int device, void* host, const void* dev, size_t bytes, cudaStream_t st) {
    const std::unique_lock<std::mutex> held = take_slots(host, bytes, 3);
    if (!held) return cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
    char* const base = slots().base;
    return on_workers(workers_for(bytes), [=](int w, int n) {
        return download_chunks(device, static_cast<char*>(host), static_cast<const char*>(dev), bytes, st,
                               base + size_t(w) * 2 * kChunk, w, n);
    });
}

}  // namespace ym
