// stage_copy (st_stage.cu) on the stand-in runtime; one scenario a process.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "runtime.h"
#include "st_kernels.h"

#define EXPECT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

using namespace st;

constexpr size_t MB = (size_t)1 << 20;
static cudaStream_t stream;

struct Buffers {
    std::vector<char> pageable;
    char *locked = nullptr, *dev = nullptr;
    cudaMemPool_t pool = nullptr;
    explicit Buffers(size_t bytes) : pageable(bytes) {
        cudaMallocHost((void **)&locked, bytes);
        cudaMemPoolProps props = {};
        cudaMemPoolCreate(&pool, &props);
        cudaMallocFromPoolAsync((void **)&dev, bytes, pool, stream);
        for (size_t i = 0; i < bytes; i++) pageable[i] = locked[i] = (char)(i * 7 + (i >> 12));
    }
};

// Page-locked arrays are copied directly: they make no slots however many bytes have gone by, nor does a
// call whose pageable part is small.  Pageable ones make them, after the first 64 MB.
static int locked_only() {
    Stage s;
    Buffers b(8 * MB);
    const int allocs = fake.host_allocs, streams = fake.streams;
    for (int k = 0; k < 20; k++)
        for (bool to_host : {false, true})
            EXPECT(stage_copy(s, {{b.locked, b.dev, 7 * MB}, {b.pageable.data(), b.dev + 7 * MB, MB / 4}}, to_host, stream) == cudaSuccess);
    EXPECT(!s.pinned && fake.host_allocs == allocs && fake.streams == streams);
    for (int k = 0; k < 8; k++) {
        EXPECT(stage_copy(s, {{b.pageable.data(), b.dev, 8 * MB}}, false, stream) == cudaSuccess);
        EXPECT(!s.pinned);
    }
    EXPECT(stage_copy(s, {{b.pageable.data(), b.dev, 8 * MB}}, false, stream) == cudaSuccess);
    EXPECT(s.pinned && !memcmp(b.dev, b.pageable.data(), 8 * MB));
    stage_release(s);
    return 0;
}

// An error that something before left for the caller to see is still there afterwards.
static int keeps_errors() {
    Stage s;
    s.copied = 64 * MB;
    Buffers b(4 * MB);
    void *p;
    fake.device_bytes = 0;
    EXPECT(cudaMalloc(&p, 1) == cudaErrorMemoryAllocation);
    fake.device_bytes = (size_t)1 << 40;
    for (bool to_host : {false, true})
        EXPECT(stage_copy(s, {{b.pageable.data(), b.dev, 3 * MB}, {b.locked, b.dev, MB}}, to_host, stream) == cudaSuccess);
    EXPECT(s.pinned && cudaGetLastError() == cudaErrorMemoryAllocation);
    return 0;
}

// Whichever of a call's copies is refused, the others are over, or before what the stream does next, when
// the call returns with the error: the caller gives the device memory back then.
static int refused_copies(bool to_host) {
    Stage s;
    s.copied = 64 * MB;
    Buffers b(5 * MB + 12345);
    auto copy = [&] {
        return stage_copy(s, {{b.pageable.data(), b.dev, 3 * MB}, {b.pageable.data() + 3 * MB, b.dev + 3 * MB, 2 * MB + 12345}},
                          to_host, stream);
    };
    EXPECT(copy() == cudaSuccess);
    int refused = 0;
    for (int k = 1; k <= 24; k++) {
        cudaStreamSynchronize(stream);
        fake.fail_copy = k;
        const cudaError_t e = copy();
        refused += e != cudaSuccess;
        EXPECT(fake.fail_copy ? e == cudaSuccess : e == cudaErrorInvalidValue);
        fake.fail_copy = 0;
        cudaGetLastError();
        cudaFreeAsync(b.dev, stream);
        EXPECT(fake.unordered_frees == 0);
        EXPECT(!to_host || fake.in_flight() == 0);
        cudaMallocFromPoolAsync((void **)&b.dev, 5 * MB + 12345, b.pool, stream);
        // and the slots are fit for the next call
        for (size_t i = 0; i < 5 * MB + 12345; i++) (to_host ? b.dev : b.pageable.data())[i] = (char)(i * k);
        EXPECT(stage_copy(s, {{b.pageable.data(), b.dev, 5 * MB + 12345}}, to_host, stream) == cudaSuccess);
        EXPECT(!memcmp(b.pageable.data(), b.dev, 5 * MB + 12345));
    }
    EXPECT(refused == 21);                             // 256 KB at a time
    return 0;
}

// Without memory for it, or without more threads, a copy is still made, and no exception leaves it.
static int no_resources() {
    Stage s;
    s.copied = 64 * MB;
    Buffers b(5 * MB);
    for (bool to_host : {false, true}) {
        for (int k = 0; k <= 12; k++) {
            for (size_t i = 0; i < 5 * MB; i++) (to_host ? b.dev : b.pageable.data())[i] = (char)(i * 3 + k);
            fake.fail_new = k;
            fake.no_threads = k == 0;
            const cudaError_t e = stage_copy(s, {{b.pageable.data(), b.dev, 5 * MB}}, to_host, stream);
            fake.fail_new = 0;
            fake.no_threads = false;
            EXPECT(e == cudaSuccess && !memcmp(b.pageable.data(), b.dev, 5 * MB));
        }
    }
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    cudaStreamCreateWithFlags(&stream, 0);
    if (what == "locked_only") return locked_only();
    if (what == "keeps_errors") return keeps_errors();
    if (what == "refused_copies") return refused_copies(argv[2] == std::string("to_host"));
    if (what == "no_resources") return no_resources();
    printf("no such scenario\n");
    return 2;
}
