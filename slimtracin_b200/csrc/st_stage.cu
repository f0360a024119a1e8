// st_stage.cu — copies between pageable host memory and the device for the calls that take or return
// whole arrays there (mesh BVH builds, texture baking).
//
// The driver stages a pageable copy through page-locked memory with one thread, whose memcpy (10 to
// 17 GB/s) is what such a copy takes: 42 + 10 MB of BLAS results 3.1 ms, a 16.8 MB mip chain 1.04 ms,
// on a bus that moves 52 GB/s.  Here a few threads take chunks in turn, each with two page-locked slots
// and a stream of its own, so that one slot is filled or emptied while the other is on the bus; a whole
// updateMeshBVH of 327,680 triangles went from 6.5 to 4.7 ms with it, a bake from 1.9 to 1.5 (slots of
// 1 MB: 3.6 and 1.5, of 64 KB 7.5 and 2.1).  Page-locking the slots costs 1 to 5 ms, 12 to 24 for 8 MB
// of them, which takes some 60 MB of copies to earn back: a context's first kStageAfter pageable bytes
// go the plain way.  Page-locked host memory is copied directly and does not count, small copies as they are.
#include <algorithm>
#include <cstring>
#include <thread>
#include "st_kernels.h"

namespace st {

namespace {

constexpr size_t kSlotBytes = 256 << 10;
constexpr size_t kStagedFrom = 2 << 20;        // less pageable than this in one call is not worth the threads
constexpr size_t kStageAfter = 64 << 20;
constexpr int kStageArrays = 8;                // a call's arrays that can go through the slots (a mesh build's: 6)

struct Chunk { char *host, *dev; size_t bytes; };

// The copies that go through the slots, a slot's size at a time.  (No allocation: an exception must not
// leave the C entry points above, nor a thread.)
struct Chunks {
    HostCopy copies[kStageArrays];
    int arrays = 0;
    size_t count = 0;
    static size_t of(const HostCopy &c) { return (c.bytes + kSlotBytes - 1) / kSlotBytes; }
    void add(const HostCopy &c) {
        copies[arrays++] = c;
        count += of(c);
    }
    Chunk at(size_t k) const {
        const HostCopy *c = copies;
        for (; k >= of(*c); c++) k -= of(*c);
        const size_t at = k * kSlotBytes;
        return {static_cast<char *>(c->host) + at, static_cast<char *>(c->dev) + at, std::min(kSlotBytes, c->bytes - at)};
    }
};

// Thread t's chunks: t, t + kStageThreads, ...
cudaError_t copy_share(Stage &s, int t, const Chunks &chunks, bool to_host) {
    cudaError_t e = cudaSetDevice(s.device);
    cudaStream_t st = s.stream[t];
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, s.ready, 0);
    const size_t count = chunks.count > (size_t)t ? (chunks.count - t - 1) / kStageThreads + 1 : 0;
    auto chunk = [&](size_t j) { return chunks.at(t + j * kStageThreads); };
    auto slot = [&](size_t j) { return s.pinned + (2 * t + (j & 1)) * kSlotBytes; };
    auto fetch = [&](size_t j) {
        const Chunk c = chunk(j);
        cudaError_t r = cudaMemcpyAsync(slot(j), c.dev, c.bytes, cudaMemcpyDeviceToHost, st);
        return r == cudaSuccess ? cudaEventRecord(s.done[t][j & 1], st) : r;
    };
    // (a slot may still be on the bus for the call before)
    for (int k = 0; k < 2 && e == cudaSuccess; k++) e = cudaEventSynchronize(s.done[t][k]);
    if (to_host) {
        for (size_t j = 0; j < std::min<size_t>(2, count) && e == cudaSuccess; j++) e = fetch(j);
        for (size_t j = 0; j < count && e == cudaSuccess; j++) {
            e = cudaEventSynchronize(s.done[t][j & 1]);
            if (e != cudaSuccess) break;
            const Chunk c = chunk(j);
            memcpy(c.host, slot(j), c.bytes);
            if (j + 2 < count) e = fetch(j + 2);
        }
    } else {
        for (size_t j = 0; j < count && e == cudaSuccess; j++) {
            e = cudaEventSynchronize(s.done[t][j & 1]);
            if (e != cudaSuccess) break;
            const Chunk c = chunk(j);
            memcpy(slot(j), c.host, c.bytes);
            e = cudaMemcpyAsync(c.dev, slot(j), c.bytes, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(s.done[t][j & 1], st);
        }
    }
    return e;
}

bool stage_ready(Stage &s) {
    if (s.pinned) return true;
    cudaError_t e = cudaHostAlloc((void **)&s.pinned, 2 * kStageThreads * kSlotBytes, cudaHostAllocDefault);
    for (int t = 0; t < kStageThreads && e == cudaSuccess; t++) {
        e = cudaStreamCreateWithFlags(&s.stream[t], cudaStreamNonBlocking);
        for (int k = 0; k < 2 && e == cudaSuccess; k++) e = cudaEventCreateWithFlags(&s.done[t][k], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming);
    if (e == cudaSuccess) return true;
    stage_release(s);
    cudaGetLastError();
    return false;
}

}  // namespace

void stage_release(Stage &s) {
    for (int t = 0; t < kStageThreads; t++) {
        for (cudaEvent_t &ev : s.done[t]) {
            if (ev) cudaEventSynchronize(ev);
            if (ev) cudaEventDestroy(ev);
            ev = nullptr;
        }
        if (s.stream[t]) cudaStreamDestroy(s.stream[t]);
        s.stream[t] = nullptr;
    }
    if (s.ready) cudaEventDestroy(s.ready);
    s.ready = nullptr;
    if (s.pinned) cudaFreeHost(s.pinned);
    s.pinned = nullptr;
}

cudaError_t stage_copy(Stage &s, std::initializer_list<HostCopy> copies, bool to_host, cudaStream_t st) {
    const cudaMemcpyKind kind = to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
    auto pageable = [](const HostCopy &c) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, c.host) == cudaSuccess) return a.type != cudaMemoryTypeHost;
        cudaGetLastError();                            // (of this call alone: an earlier error is the caller's)
        return true;
    };
    size_t all = 0, total = 0;                         // of all, of the pageable ones
    for (const HostCopy &c : copies) all += c.bytes;
    if (all >= kStagedFrom)
        for (const HostCopy &c : copies) total += c.bytes && pageable(c) ? c.bytes : 0;
    bool staged = false;
    if (total >= kStagedFrom) {
        staged = s.copied >= kStageAfter && stage_ready(s);
        s.copied += total;
    }
    cudaError_t e = cudaSuccess;
    Chunks chunks;
    for (const HostCopy &c : copies) {
        if (staged && chunks.arrays < kStageArrays && pageable(c)) chunks.add(c);
        else if (c.bytes && e == cudaSuccess) e = cudaMemcpyAsync(to_host ? c.host : c.dev, to_host ? c.dev : c.host, c.bytes, kind, st);
    }
    if (e != cudaSuccess || !chunks.count) return e;
    if ((e = cudaEventRecord(s.ready, st)) != cudaSuccess) return e;
    cudaError_t got[kStageThreads] = {};
    std::thread threads[kStageThreads];
    int started = 1;                                   // the caller is the first of them
    try {
        for (; started < kStageThreads; started++)
            threads[started] = std::thread([&, t = started] { got[t] = copy_share(s, t, chunks, to_host); });
    } catch (...) {                                    // no more threads, or memory: the caller takes the other shares
    }
    got[0] = copy_share(s, 0, chunks, to_host);
    for (int t = started; t < kStageThreads; t++) got[t] = copy_share(s, t, chunks, to_host);
    for (int t = 1; t < started; t++) threads[t].join();
    for (int t = 0; t < kStageThreads; t++) {
        if (e == cudaSuccess) e = got[t];
        // what follows on `st` comes after the copies
        for (int k = 0; k < 2 && !to_host && e == cudaSuccess; k++) e = cudaStreamWaitEvent(st, s.done[t][k], 0);
    }
    // where one failed the others are not left on the bus: the caller gives up the memory they use
    for (int t = 0; t < kStageThreads && e != cudaSuccess; t++) cudaStreamSynchronize(s.stream[t]);
    return e;
}

}  // namespace st
