// A row per block in registers, eight neighbouring elements per thread: what the row kernels (norms, adds, copies) share.
//
// Rows of a multiple of 8 elements up to 8192 whose starts lie on 16 bytes go this way; others keep the kernels that walk a row
// element by element.  Bound by latency where a step has few rows (the loads of a row are all in flight at once, and weights are
// asked into L2 before the wait for the kernel in front, which may be the one that writes them: they are read behind it) and by
// bytes where it has many.  Measured against the
// walk (us, one launch after another): add and RMS norm, 2048 rows of 2304, 18.6 -> 9.3 (6.1 TB/s), 8 rows 4.8 -> 2.7; add and layer
// norm, 2813 rows of 1536, 21.1 -> 12.7; the same of the mean of two branches 37.4 -> 22.8; norm of a 768-wide piece of 2048 rows
// 5.3 -> 3.8.  Wide rows, add and RMS norm / layer norm / add and layer norm / norm of a piece: 8192 wide, 8 rows, add and layer norm
// 9.9 -> 3.6; 2048 rows 59 -> 36 / 34 -> 20 / 83 -> 62 / 30 -> 15; 6144 wide, 2048 rows 41 -> 28 / 27 -> 16 / 57 -> 47 / 23 -> 12.  (Add and layer norm of 512
// or 1024 rows of 6144 lose 4 %, 11.2 -> 11.7: a block of 768 threads has an SM to itself.)
#pragma once
#include <initializer_list>

#include "common.cuh"

namespace qnn {

constexpr int ROW8_MAX = 8192, ROW8_THREADS = ROW8_MAX / 8;

// rows of n elements, all of these on 16 bytes (null: not there)
inline bool row8_fits(int n, std::initializer_list<const void*> ps, std::initializer_list<long long> pitches_in_bytes = {}) {
    if (n <= 0 || n % 8 != 0 || n > ROW8_MAX) return false;
    for (const void* p : ps)
        if (((uintptr_t)p & 15) != 0) return false;
    for (long long b : pitches_in_bytes)
        if (b % 16 != 0) return false;
    return true;
}
inline int row8_threads(int n) { return (n / 8 + 31) / 32 * 32; }
inline long long dt_bytes(int dt) { return dt == QNN_DT_BF16 ? 2 : 4; }

__device__ __forceinline__ void zero8(float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
}
// this thread's eight (zeros beyond the row)
__device__ __forceinline__ void row8_load(const void* p, int dt, size_t base, int n, float (&v)[8]) {
    const int j = threadIdx.x * 8;
    if (j < n) load8_as_f(p, dt, base + j, v);
    else zero8(v);
}
// asks the lines of a row of weights into L2, where whoever writes them writes them too; nothing is read.  The first block does it for
// all (every block: add and layer norm of 2048 rows of 2304 11.7 -> 12.3 us)
__device__ __forceinline__ void row8_ask(const void* p, int dt, int n) {
    const int j = threadIdx.x * 8, size = dt == QNN_DT_BF16 ? 2 : 4;
    if (blockIdx.x == 0 && j < n && j * size % 128 < 8 * size) asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p + (size_t)j * size));
}
__device__ __forceinline__ void row8_store(void* p, int dt, size_t base, int n, const float (&v)[8]) {
    const int j = threadIdx.x * 8;
    if (j < n) store8_from_f(p, dt, base + j, v);
}
__device__ __forceinline__ float squares8(const float (&v)[8]) {
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += v[e] * v[e];
    return s;
}
__device__ __forceinline__ float sum8(const float (&v)[8]) {
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s += v[e];
    return s;
}

}  // namespace qnn
