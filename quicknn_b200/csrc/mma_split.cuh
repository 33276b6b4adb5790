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
__device__ __forceinline__ void cp16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

}  // namespace qnn
