// A stand-in for the CUDA runtime that needs no device: memory is host memory, copies are made at once,
// kernels do nothing, and a driver can have an allocation, a copy or a launch refused.  It keeps track
// of what a real device would leave in flight: each stream and event carries how far it is ordered after
// every stream's copies, and the host learns of their end by waiting.  Linked with the library's own
// objects in place of cudart.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <pthread.h>
#include <cerrno>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <vector>
#include "runtime.h"

FakeRuntime fake;
static thread_local int fake_inside = 0;         // > 0 in the stand-in itself

void *operator new(size_t bytes) {
    if (!fake_inside && fake.fail_new > 0 && --fake.fail_new == 0) throw std::bad_alloc();
    return malloc(bytes);
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }
extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *arg) {
    static auto real = reinterpret_cast<decltype(&pthread_create)>(dlsym(RTLD_NEXT, "pthread_create"));
    return fake.no_threads ? EAGAIN : real(t, a, f, arg);
}

namespace {
typedef std::map<const void *, long> Clock;      // stream -> its copies that are known to come before
struct Copy { const void *stream; long at; const char *dev; size_t bytes; };
std::recursive_mutex m;
std::map<const void *, Clock> clocks;            // of streams and events
std::map<const void *, long> issued;
Clock host_seen;
std::vector<Copy> copies;
std::map<const char *, size_t> device_blocks, pinned_blocks;
std::map<const void *, std::string> kernels;
struct Pool { size_t reserved = 0, used = 0; uint64_t threshold = 0; std::map<char *, size_t> blocks; };
std::map<char *, Pool *> pool_of;
thread_local cudaError_t last = cudaSuccess;

struct Lock {
    std::lock_guard<std::recursive_mutex> guard;
    explicit Lock(std::recursive_mutex &mutex) : guard(mutex) { fake_inside++; }
    ~Lock() { fake_inside--; }
};
cudaError_t fail(cudaError_t e) { return last = e; }
void merge(Clock &into, const Clock &from) {
    for (auto &kv : from) if (into[kv.first] < kv.second) into[kv.first] = kv.second;
}
void host_waits(const void *what) {
    merge(host_seen, clocks[what]);
    std::vector<Copy> left;
    for (const Copy &c : copies) if (host_seen[c.stream] < c.at) left.push_back(c);
    copies.swap(left);
}
const std::pair<const char *const, size_t> *block(const std::map<const char *, size_t> &blocks, const void *p) {
    auto it = blocks.upper_bound(static_cast<const char *>(p));
    if (it == blocks.begin()) return nullptr;
    --it;
    return static_cast<const char *>(p) < it->first + it->second ? &*it : nullptr;
}
constexpr size_t kGranule = (size_t)2 << 20;
size_t granules(size_t b) { return (b + kGranule - 1) / kGranule * kGranule; }
bool resize(Pool &P, size_t reserved) {
    if (reserved > P.reserved && fake.device_held + reserved - P.reserved > fake.device_bytes) return false;
    fake.device_held += reserved - P.reserved;
    P.reserved = reserved;
    return true;
}
cudaError_t host_alloc(void **p, size_t bytes) {
    Lock l(m);
    *p = calloc(1, bytes);
    pinned_blocks[static_cast<char *>(*p)] = bytes;
    fake.host_allocs++;
    fake.host_bytes += bytes;
    return cudaSuccess;
}
}  // namespace

int FakeRuntime::in_flight() { Lock l(m); return (int)copies.size(); }

extern "C" {
// memory
cudaError_t cudaMalloc(void **p, size_t bytes) {
    Lock l(m);
    if (fake.device_held + bytes > fake.device_bytes) { *p = nullptr; return fail(cudaErrorMemoryAllocation); }
    fake.device_held += bytes;
    *p = calloc(1, bytes);
    device_blocks[static_cast<char *>(*p)] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    Lock l(m);
    if (!p) return cudaSuccess;
    fake.device_held -= device_blocks[static_cast<char *>(p)];
    device_blocks.erase(static_cast<char *>(p));
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return host_alloc(p, bytes); }
cudaError_t cudaMallocHost(void **p, size_t bytes) { return host_alloc(p, bytes); }
cudaError_t cudaFreeHost(void *p) { Lock l(m); pinned_blocks.erase(static_cast<char *>(p)); free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    Lock l(m);
    memset(a, 0, sizeof(*a));
    a->type = block(pinned_blocks, p) ? cudaMemoryTypeHost : block(device_blocks, p) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->devicePointer = a->hostPointer = const_cast<void *>(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *) {
    *pool = reinterpret_cast<cudaMemPool_t>(new Pool());
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t pool, cudaMemPoolAttr, void *v) {
    reinterpret_cast<Pool *>(pool)->threshold = *static_cast<uint64_t *>(v);
    return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t pool, cudaMemPoolAttr attr, void *v) {
    Lock l(m);
    Pool *P = reinterpret_cast<Pool *>(pool);
    *static_cast<uint64_t *>(v) = attr == cudaMemPoolAttrUsedMemCurrent ? P->used : P->reserved;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
    Lock l(m);
    Pool *P = reinterpret_cast<Pool *>(pool);
    const size_t floor = granules(P->used > keep ? P->used : keep);
    if (floor < P->reserved) resize(*P, floor);
    fake.trims++;
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t pool) {
    Lock l(m);
    Pool *P = reinterpret_cast<Pool *>(pool);
    resize(*P, 0);
    delete P;
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t) {
    Lock l(m);
    Pool *P = reinterpret_cast<Pool *>(pool);
    if (granules(P->used + bytes) > P->reserved && !resize(*P, granules(P->used + bytes))) return fail(cudaErrorMemoryAllocation);
    P->used += bytes;
    char *q = static_cast<char *>(calloc(1, bytes));
    device_blocks[q] = bytes;
    pool_of[q] = P;
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t st) {
    Lock l(m);
    const size_t bytes = device_blocks[static_cast<char *>(p)];
    for (const Copy &c : copies)
        if (c.dev >= static_cast<char *>(p) && c.dev < static_cast<char *>(p) + bytes && clocks[st][c.stream] < c.at)
            fake.unordered_frees++;
    Pool *P = pool_of[static_cast<char *>(p)];
    P->used -= bytes;
    if (P->reserved > P->threshold) resize(*P, granules(P->used > P->threshold ? P->used : P->threshold));
    pool_of.erase(static_cast<char *>(p));
    device_blocks.erase(static_cast<char *>(p));
    return cudaSuccess;                           // (the block itself is left to the process' end)
}
// streams and events
static void *handle() { return calloc(1, 8); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { Lock l(m); *s = static_cast<cudaStream_t>(handle()); fake.streams++; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t) { Lock l(m); fake.streams--; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { Lock l(m); host_waits(s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { Lock l(m); copies.clear(); return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *least, int *greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = static_cast<cudaEvent_t>(handle()); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { Lock l(m); clocks[e] = clocks[s]; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { Lock l(m); host_waits(e); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { Lock l(m); merge(clocks[s], clocks[e]); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind kind, cudaStream_t st) {
    Lock l(m);
    if (fake.fail_copy > 0 && --fake.fail_copy == 0) return fail(cudaErrorInvalidValue);
    for (const void *p : {(const void *)dst, src})
        for (auto *blocks : {&device_blocks, &pinned_blocks})
            if (auto *b = block(*blocks, p))
                if (static_cast<const char *>(p) + bytes > b->first + b->second) {
                    fake.out_of_range++;
                    return fail(cudaErrorInvalidValue);
                }
    memcpy(dst, src, bytes);
    const long at = ++issued[st];
    clocks[st][st] = at;
    copies.push_back({st, at, static_cast<const char *>(kind == cudaMemcpyHostToDevice ? dst : src), bytes});
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t bytes, cudaStream_t) { memset(p, v, bytes); return cudaSuccess; }
// the device, errors
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) { memset(p, 0, sizeof(*p)); p->major = 10; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }
// launches
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 1; }
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t) {
    Lock l(m);
    if (!fake.refuse_kernel.empty() && kernels[f].find(fake.refuse_kernel) != std::string::npos) return fail(cudaErrorLaunchOutOfResources);
    fake.launches++;
    fake.log += kernels[f] + "\n";
    return cudaSuccess;
}
}
