// A CUDA runtime for tests of host code: allocations come from the heap and
// fail while `fail_next` counts down, or for good while a pool holds memory
// that is not given back.
#pragma once

#include <cstdlib>
#include <string>

#include "unap_internal.hpp"

namespace fake {
int fail_next = 0;         // this many allocations fail
bool pool_holds = false;   // allocations fail until the workspace pool is trimmed
int trims = 0, live = 0, calls = 0;

inline cudaError_t get(void** p, size_t bytes)
{
    ++calls;
    if (pool_holds || fail_next > 0) {
        if (fail_next > 0) --fail_next;
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    *p = std::malloc(bytes ? bytes : 1);
    ++live;
    return cudaSuccess;
}
inline cudaError_t put(void* p)
{
    if (p) --live;
    std::free(p);
    return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::get(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return fake::get(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t)
{
    return fake::get(p, n);
}
cudaError_t cudaFree(void* p) { return fake::put(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return fake::put(p); }
cudaError_t cudaMallocHost(void** p, size_t n)
{
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
}

namespace unapgpu {
std::shared_mutex& capture_gate()
{
    static std::shared_mutex m;
    return m;
}
bool& thread_in_capture()
{
    static thread_local bool v = false;
    return v;
}
cudaStream_t& thread_alloc_stream()
{
    static thread_local cudaStream_t s = nullptr;
    return s;
}
cudaMemPool_t& thread_alloc_pool()
{
    static thread_local cudaMemPool_t p = nullptr;
    return p;
}
void keep_pool_memory() {}
void trim_workspace_pool()
{
    ++fake::trims;
    fake::pool_holds = false;
}
void* pinned_block_alloc(size_t bytes) { return std::malloc(bytes); }
void pinned_block_free(void* p) { std::free(p); }
}  // namespace unapgpu

#define EXPECT(c)                                             \
    do {                                                      \
        if (!(c)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #c);       \
            return 1;                                         \
        }                                                     \
    } while (0)
