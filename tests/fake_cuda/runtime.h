// What a test driver sets and reads of the stand-in CUDA runtime (runtime.cpp).
#pragma once
#include <atomic>
#include <cstddef>
#include <string>

struct FakeRuntime {
    // set by a driver
    size_t device_bytes = (size_t)1 << 40;   // cudaMalloc and pool growth fail beyond this
    int fail_copy = 0;                       // > 0: the n-th cudaMemcpyAsync from now fails
    std::string refuse_kernel;               // launches of kernels whose name contains this fail
    std::atomic<int> fail_new{0};            // > 0: the n-th operator new from now throws (the stand-in's own excepted)
    bool no_threads = false;                 // no further thread can be made
    // read by a driver
    size_t device_held = 0;                  // what cudaMalloc and the pools hold of it
    size_t host_bytes = 0;                   // page-locked, all told
    int host_allocs = 0, streams = 0, launches = 0, trims = 0;
    int out_of_range = 0;                    // copies past the end of a block (not made)
    int unordered_frees = 0;                 // cudaFreeAsync of memory that a copy elsewhere may still use
    std::string log;                         // the launched kernels' names, in order
    int in_flight();                         // copies that neither the host nor a later wait has seen the end of
};
extern FakeRuntime fake;
