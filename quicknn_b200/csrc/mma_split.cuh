// mma.sync products of float32 matrices in bfloat16 parts: what the scans of the recurrent mixers share.
//
// A float32 number is the sum of three bfloat16 numbers (8 bits of its 24 each), so a product with one factor that is a
// bfloat16 number already costs three products on the tensor cores and one of two float32 matrices six (the three smallest of
// the nine terms lie below float32's rounding); accumulation is float32.
#pragma once
#include "common.cuh"

namespace qnn {


__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a b without an accumulator to start from
__device__ __forceinline__ void mma_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ float low_of(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float high_of(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
struct Split3 { uint32_t h[4], m[4], l[4]; };
// The upper half of a float32 is a bfloat16 with its first 8 significant bits; what is left has 16, and once more 8: the three
// parts add up to the number exactly (but for what lies below float32's smallest normal numbers).
__device__ __forceinline__ float upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ uint32_t uppers(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
__device__ __forceinline__ void split(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = uppers(a, b);
    a -= upper(a);
    b -= upper(b);
    m = uppers(a, b);
    l = uppers(a - upper(a), b - upper(b));
}
// two accumulator tiles (16 x 8 each, side by side) as the A operand of a product over those 16 columns
__device__ __forceinline__ void split_tiles(const float (&x)[4], const float (&y)[4], Split3& s) {
    split(x[0], x[1], s.h[0], s.m[0], s.l[0]);
    split(x[2], x[3], s.h[1], s.m[1], s.l[1]);
    split(y[0], y[1], s.h[2], s.m[2], s.l[2]);
    split(y[2], y[3], s.h[3], s.m[3], s.l[3]);
}
// Products of 8 bfloat16 rows with up to MT * 16 rows of weights, for the few outputs per row that feed float32 math (gates, router
// logits): dots[row][output], from all warps of the block (`warps` of them share the width in pieces of 32; `part` is scratch for
// warps * MT * 128 doubles).  x: `rows` (1 to 8) of them, ldx apart; w: n rows of `width`; both on 16 bytes, width a multiple of 8.  A dot
// product per warp, row and output on the FMA pipe costs a load and an unpacking of both factors per product of eight, most of its
// time; here a warp's instruction does 16 outputs of 8 rows.  Every piece's sums of 16 start from zero and are added in float64 (a few
// additions per output), so that neither the tensor cores' cutting of an accumulator's last bits nor the additions' rounding adds
// up: no further from 64 bits than float32 sums (measured).  The order of sums depends on the width and the warps only.
constexpr int DOT_ROWS = 8;
template <int MT>
__device__ __forceinline__ void row_dots(const bf16* x, long long ldx, int rows, const bf16* w, int n, int width, int warps, double* part,
                                         float* dots, int ldd) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double acc[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][e] = 0.0;
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 3
    for (int k0 = warp * 32; k0 < width; k0 += warps * 32) {
        const int k = k0 + t * 8;
        const bool in = k < width;
        const uint4 b = in && g < rows ? *reinterpret_cast<const uint4*>(x + (size_t)g * ldx + k) : none;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int r = m * 16 + g;
            const uint4 lo = in && r < n ? __ldg(reinterpret_cast<const uint4*>(w + (size_t)r * width + k)) : none;
            const uint4 hi = in && r + 8 < n ? __ldg(reinterpret_cast<const uint4*>(w + (size_t)(r + 8) * width + k)) : none;
            const uint32_t first[4] = {lo.x, hi.x, lo.y, hi.y}, second[4] = {lo.z, hi.z, lo.w, hi.w};
            float f[4], s[4];
            mma_first(f, first, b.x, b.y);
            mma_first(s, second, b.z, b.w);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][e] += (double)f[e] + (double)s[e];
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {                               // [warp][output][row]
        double* at = part + ((size_t)warp * MT * 16 + m * 16 + g) * DOT_ROWS + 2 * t;
        *reinterpret_cast<double2*>(at) = make_double2(acc[m][0], acc[m][1]);
        *reinterpret_cast<double2*>(at + 8 * DOT_ROWS) = make_double2(acc[m][2], acc[m][3]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < MT * 16 * DOT_ROWS; i += blockDim.x) {
        double d = 0.0;
        for (int u = 0; u < warps; ++u) d += part[u * MT * 16 * DOT_ROWS + i];
        if (i / DOT_ROWS < n) dots[(i % DOT_ROWS) * ldd + i / DOT_ROWS] = (float)d;
    }
    __syncthreads();
}
__device__ __forceinline__ void cp16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

}  // namespace qnn
