// What fake_cuda.cpp's CUDA calls see and do.
#pragma once
#include <driver_types.h>

#include <cstddef>
#include <vector>

struct Range {
    const char* p;
    size_t n;
    cudaMemoryType type;
};
extern std::vector<Range> g_ranges;     // memory that is not pageable
extern bool g_no_pinned;                // cudaHostAlloc fails
extern int g_threads_left;              // pthread_create fails after as many
extern int g_direct, g_staged;          // copies from or to the caller's memory, and the ring's
