// Matrix memories over prompts, in chunks of 64 rows on the tensor cores.
//
//   S_t = D_t S_{t-1} + w_t k_t v_t^T,   o_t = S_t^T (q_t q_scale)        S: [dim, vdim] float32 per (sequence, head)
//
// with D_t a number per head (retention, mLSTM, lightning: `w` an input gate or 1) or a diagonal over the key channels (gated
// linear attention; HGRN2, whose keys are 1 - decay).  The same results as the row-by-row scans of gla.cu, which serve single
// tokens, short steps, other sizes and float32 values.
//
//   memory_chunk_local   per (chunk, head): the chunk's outputs from its own rows, O = A V with A the masked and decayed
//                        products of queries and keys; the state L = K~^T V that it builds from nothing; its decay product
//   memory_chunk_prefix  per state element: walks the chunks in order, leaves in L's place the state before each chunk, and
//                        moves the slot's state on
//   memory_chunk_out     per (chunk, head): O += Q~ S, Q~ the queries times the decays since the chunk's start
//
// Queries, keys and values are bfloat16 numbers as they come (retention's rotated queries and keys are float32); every other
// matrix is float32 and meets them in three bfloat16 parts (mma_split.cuh), so products keep float32's 24 bits; sums are float32.
// Decays between two rows are products of the rows' decays, all at most 1 where decays are; nothing is
// divided and no logarithm is taken, so no decay is too strong.  One per head: in 64 bits, rounded once.  Within 16 rows (a sub-chunk)
// the per-channel decays stand between query and key, and those products, decays included, run in float32 on the FMA pipes; between
// sub-chunks j < i they part into (suffix of j) (whole sub-chunks between) (prefix of i), each in 64 bits and rounded once, and the
// products are matrix products again.
//
// Against the recurrence in 64 bits, on what eight layers of Fuposun and Tumudra at two widths hand over (2-norm, the row-by-row walk in
// brackets): a decay per channel around 0.92: outputs 0.9e-7 to 1.1e-7 (1.0e-7 to 1.1e-7), states 5.8e-8 (6.1e-8 to 6.7e-8); constant decays from 0.97 on:
// 1.0e-7 to 1.4e-7 (2.1e-7 to 5.4e-7), 5e-8 to 8e-8 (2.4e-7 to 8.4e-7); an mLSTM's gates around 0.5: 0.7e-7 to 1.0e-7 (0.8e-7 to 1.1e-7), states
// 3.6e-8 to 6.7e-8 (2.8e-8 to 5.1e-8: two roundings for the last row where here there are five).
//
// Bound by latency, not by a unit (one prompt of 4096 rows, 9 heads of 128 x 256, a decay per channel): a block of 512 threads per SM, or
// two of 256 in the outputs' kernel, fill a quarter of the warps; the tensor pipe is busy 20 and 33 % of the time, L2 18 and 15 %, and warps
// wait in turn at the barriers between a block's stages, for shared memory and for the pipe (about 20 cycles per product and
// scheduler, six products per pair of float32 tiles).  The prefix is bound by the chunk states' way: 16 bytes per state element and
// chunk, written once, read and written by the prefix, read once, 1.2 MB of state per chunk.  Measured at 2048 rows: 47 + 9 + 35 us; the
// walk in segments of 256 rows took 320.  Prompts of 1777, 731 and 301 rows, 12 heads of 64 x 128, a gate per head: 36 + 9 + 25 us against 820.
// A number that is Inf or NaN reaches what depends on it and nothing else, as in the walk: rows before it, other columns of a value's
// head and other heads keep their results (what does depend on it is Inf or NaN; the parts of an Inf are Inf and NaN).
// A block takes a chunk that there is: the chunks of all sequences are counted through, so unequal sequences cost what their rows do.
// Steps whose states would not stay in L2 run in rounds of chunks (the caller's scratch limits them), each from the slots'
// states and back into them.
#include "mma_split.cuh"

using namespace qnn;

namespace {

constexpr int CH = 64, SB = 16, NS = CH / SB;     // rows of a chunk, of a sub-chunk; sub-chunks
constexpr int LOCAL_THREADS = 512, OUT_THREADS = 256, MAX_VDIM = 256;

struct ChunkArgs {
    const void *q, *k;
    long long ldq;
    const bf16* v;
    long long ldv;
    const float* decay;                           // decay[row * ldd + h (* DIM + channel)]
    long long ldd;
    const float* kw;                              // w: kw[row * ldw + h], null: 1
    long long ldw;
    float q_scale;
    const int *seq_row0, *seq_len, *slots;        // [B]
    int B, least;                                 // sequences of fewer than `least` rows are not this path's
    float* out;                                   // [rows, ldo], vs columns per head
    long long ldo;
    float* state;                                 // slot s: [H, DIM, vs] at state + s * state_stride
    long long state_stride;
    float* local;                                 // [units, H, DIM, vdim]
    float* local_n;                               // [units, H, DIM]: the normaliser's column (vs = vdim + 1)
    float* chunk_decay;                           // [units, H (, DIM)] pairs
    int unit0, units;                             // this round's chunks, counted through all sequences in order
    int H, vdim, vs, key_from_decay;
};

__device__ __forceinline__ int chunks_of(int rows, int least) { return rows >= least ? (rows + CH - 1) / CH : 0; }
__device__ __forceinline__ int inclusive_sum(int x, int lane, int n) {       // of the first n lanes
    for (int o = 1; o < 32 && o < n; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}
// The chunk of a block, unit `u` of the step: its first row, the slot of its sequence, and how many rows it has (0: there are not so
// many chunks).  Every warp finds it by itself, 32 sequences at a time.
__device__ __forceinline__ int find_chunk(const ChunkArgs& a, int u, int lane, int& row0, int& slot) {
    for (int b0 = 0; b0 < a.B; b0 += 32) {
        const int b = b0 + lane;
        const bool has = b < a.B;
        const int len = has ? a.seq_len[b] : 0, first = has ? a.seq_row0[b] : 0, s = has ? a.slots[b] : -1;
        const int mine = chunks_of(len, a.least), upto = inclusive_sum(mine, lane, a.B), at = (u - (upto - mine)) * CH;
        const bool here = has && at >= 0 && u < upto;            // in one lane at most; sums over the warp are uniform registers
        if (__any_sync(0xffffffffu, here)) {
            row0 = __reduce_add_sync(0xffffffffu, here ? first + at : 0);
            slot = __reduce_add_sync(0xffffffffu, here ? s : 0);
            return __reduce_add_sync(0xffffffffu, here ? min(CH, len - at) : 0);
        }
        u -= __shfl_sync(0xffffffffu, upto, 31);           // (more sequences to come: all 32 lanes have one)
    }
    return 0;
}
// chunks of the sequences before sequence b
__device__ __forceinline__ int chunks_before(const ChunkArgs& a, int b, int lane) {
    int n = 0;
    for (int i = lane; i < b; i += 32) n += chunks_of(a.seq_len[i], a.least);
    return b == 0 ? 0 : __reduce_add_sync(0xffffffffu, n);
}

template <typename TQ, int DIM>
struct Sizes {
    static constexpr int PARTS = sizeof(TQ) == 2 ? 1 : 3;        // bfloat16 matrices that hold the rows exactly
    static constexpr int P = DIM * 2 + 16, MAT = CH * P;         // bytes of a row (rows 4 banks apart), of a matrix
    static constexpr int AP = CH * 2 + 16, AMAT = CH * AP;
    static constexpr int FP = DIM + 8;                           // floats of a row of the float32 rows
};

__device__ __forceinline__ void store_split(char* at, int part_bytes, float x, float y) {       // two neighbours, three matrices
    uint32_t h, m, l;
    split(x, y, h, m, l);
    *reinterpret_cast<uint32_t*>(at) = h;
    *reinterpret_cast<uint32_t*>(at + part_bytes) = m;
    *reinterpret_cast<uint32_t*>(at + 2 * part_bytes) = l;
}
__device__ __forceinline__ void store_split1(char* at, int part_bytes, float x) {
    const float r = x - upper(x);
    *reinterpret_cast<uint16_t*>(at) = (uint16_t)(__float_as_uint(x) >> 16);
    *reinterpret_cast<uint16_t*>(at + part_bytes) = (uint16_t)(__float_as_uint(r) >> 16);
    *reinterpret_cast<uint16_t*>(at + 2 * part_bytes) = (uint16_t)(__float_as_uint(r - upper(r)) >> 16);
}
// two bfloat16 numbers: not 0 where one of them is Inf or NaN (an exponent of ones carries into the sign's place)
__device__ __forceinline__ uint32_t exponent_carry(uint32_t w) { return ((w & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }
__device__ __forceinline__ float bf_at(const char* at) { return __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t*>(at) << 16); }

// A chunk's decay as the sum of two floats: where every chunk has the same decay, close to 1, its rounding would not average out
__device__ __forceinline__ void store_decay(float* at, double d) {
    const float hi = (float)d;
    *reinterpret_cast<float2*>(at) = make_float2(hi, (float)(d - (double)hi));
}
__device__ __forceinline__ float decayed(float2 d, float carry, float more) { return fmaf(d.x, carry, fmaf(d.y, carry, more)); }

// rows of a chunk -> shared memory (bfloat16 as they are; float32 in three parts); rows beyond the chunk's are zero
template <typename TQ, int DIM, int THREADS>
__device__ __forceinline__ void stage_rows(const TQ* src, long long ld, int n, char* dst) {
    using Z = Sizes<TQ, DIM>;
    if constexpr (sizeof(TQ) == 2) {
        constexpr int PER_ROW = DIM / 8, N = CH * PER_ROW / THREADS;
        uint4 r[N];
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = threadIdx.x + e * THREADS, t = i / PER_ROW, c = i % PER_ROW;
            r[e] = t < n ? *reinterpret_cast<const uint4*>(src + (size_t)t * ld + c * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = threadIdx.x + e * THREADS, t = i / PER_ROW, c = i % PER_ROW;
            *reinterpret_cast<uint4*>(dst + t * Z::P + c * 16) = r[e];
        }
    } else {
        constexpr int PER_ROW = DIM / 4, N = CH * PER_ROW / THREADS;
        float4 r[N];
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = threadIdx.x + e * THREADS, t = i / PER_ROW, c = i % PER_ROW;
            r[e] = t < n ? *reinterpret_cast<const float4*>(src + (size_t)t * ld + c * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = threadIdx.x + e * THREADS, t = i / PER_ROW, c = i % PER_ROW;
            char* at = dst + t * Z::P + c * 8;
            store_split(at, Z::MAT, r[e].x, r[e].y);
            store_split(at + 4, Z::MAT, r[e].z, r[e].w);
        }
    }
}

// addresses of ldmatrix: `lane`'s row of the four 8 x 8 tiles of a 16 x 16 block
__device__ __forceinline__ unsigned a_row(unsigned base, int pitch, int lane) {          // A stored [m][k]; also B stored [k][n], .trans
    return base + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + (lane >> 4) * 16;
}
__device__ __forceinline__ unsigned b_row(unsigned base, int pitch, int lane) {          // B stored [n][k]; also A stored [k][m], .trans
    return base + ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 16;
}

// A tile of float32 sums.  The tensor cores cut off what lies below an accumulator's last bit, always towards zero: along a chain
// of products into one accumulator that adds up (1e-6 of the result after 48 of them, ten times float32's own rounding).  So the
// products of the leading parts start from zero and are added with float32's rounding; the others, at most 2^-7 of them, are
// a chain of their own.
struct Tile {
    float hi[4] = {}, lo[4] = {};
    __device__ __forceinline__ void lead(const uint32_t (&x)[4], uint32_t y0, uint32_t y1) {
        float f[4];
        mma_first(f, x, y0, y1);
#pragma unroll
        for (int e = 0; e < 4; ++e) hi[e] += f[e];
    }
    // a matrix in three parts (x) with one that is bfloat16, either way round
    __device__ __forceinline__ void add3(const uint32_t (&xh)[4], const uint32_t (&xm)[4], const uint32_t (&xl)[4], uint32_t y0, uint32_t y1) {
        mma(lo, xl, y0, y1);
        mma(lo, xm, y0, y1);
        lead(xh, y0, y1);
    }
    __device__ __forceinline__ void add3(const uint32_t (&x)[4], uint32_t h0, uint32_t h1, uint32_t m0, uint32_t m1, uint32_t l0, uint32_t l1) {
        mma(lo, x, l0, l1);
        mma(lo, x, m0, m1);
        lead(x, h0, h1);
    }
    // the six products of two matrices in three parts that reach float32's rounding
    __device__ __forceinline__ void add6(const uint32_t (&h)[4], const uint32_t (&m)[4], const uint32_t (&l)[4],
                                         uint32_t h0, uint32_t h1, uint32_t m0, uint32_t m1, uint32_t l0, uint32_t l1) {
        mma(lo, l, h0, h1);
        mma(lo, h, l0, l1);
        mma(lo, m, m0, m1);
        mma(lo, m, h0, h1);
        mma(lo, h, m0, m1);
        lead(h, h0, h1);
    }
    __device__ __forceinline__ float operator[](int e) const { return hi[e] + lo[e]; }
};

// Shared memory of memory_chunk_local.  One decay per head: [queries | later A], keys (their parts, later K~'s), values.
// Per channel: float32 decays (later the queries times their prefixes), [queries, keys | later A], K^ (later K~), values.
template <typename TQ, int DIM, bool CHANNELS>
struct LocalPlan {
    using Z = Sizes<TQ, DIM>;
    static constexpr int max2(int a, int b) { return a > b ? a : b; }
    static constexpr int F = 0, F_BYTES = CHANNELS ? CH * Z::FP * 4 : 0;
    static constexpr int Q = F + F_BYTES;
    static constexpr int K_RAW = Q + Z::MAT;                     // per channel
    static constexpr int A = Q, A_BYTES = max2(3 * Z::AMAT, CHANNELS ? 2 * Z::MAT : Z::PARTS * Z::MAT);
    static constexpr int K = A + A_BYTES, K_BYTES = 3 * Z::MAT;
    static constexpr int D = K + K_BYTES;                        // [64][16] floats: decays or products inside a sub-chunk
    // per head: E, P [64], F [4] doubles, decays, w [64], sums [512] floats; per channel: F [4][DIM] doubles
    static constexpr int V4 = D + CH * SB * 4;
    static constexpr int V4_BYTES = CHANNELS ? NS * DIM * 8 : 2 * CH * 8 + NS * 8 + 2 * CH * 4 + LOCAL_THREADS * 4;
    static constexpr int V = (V4 + V4_BYTES + 15) / 16 * 16;
    static int bytes(int vdim) { return V + CH * (vdim * 2 + 16); }
};

template <typename TQ, int DIM, bool CHANNELS>
__global__ void __launch_bounds__(LOCAL_THREADS) memory_chunk_local_kernel(const ChunkArgs a) {
    using Z = Sizes<TQ, DIM>;
    using L = LocalPlan<TQ, DIM, CHANNELS>;
    extern __shared__ __align__(16) char sm[];
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_wait();
    int row0 = 0, slot = -1;
    const int n = find_chunk(a, a.unit0 + blockIdx.y, lane, row0, slot), vdim = a.vdim;
    if (n <= 0) return;
    if (slot < 0) {                                        // rows of no sequence: nothing but zeros
        for (int i = tid; i < n * a.vs; i += LOCAL_THREADS) a.out[(size_t)(row0 + i / a.vs) * a.ldo + h * a.vs + i % a.vs] = 0.f;
        return;
    }
    const size_t unit = (size_t)blockIdx.y * a.H + h;
    const int VP = vdim * 2 + 16;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    float* Dd = reinterpret_cast<float*>(sm + L::D);             // [s][t mod 16]
    // ---- the chunk's rows -----------------------------------------------------------------------------------------------
    const TQ* q = (const TQ*)a.q + (size_t)row0 * a.ldq + h * DIM;
    const TQ* k = (const TQ*)a.k + (size_t)row0 * a.ldq + h * DIM;
    if constexpr (CHANNELS) {
        float* F = reinterpret_cast<float*>(sm + L::F);
        constexpr int PER_ROW = DIM / 4, N = CH * PER_ROW / LOCAL_THREADS;
        float4 r[N];
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = tid + e * LOCAL_THREADS, t = i / PER_ROW, x = i % PER_ROW;
            r[e] = t < n ? *reinterpret_cast<const float4*>(a.decay + (size_t)(row0 + t) * a.ldd + h * DIM + x * 4)
                         : make_float4(1.f, 1.f, 1.f, 1.f);
        }
#pragma unroll
        for (int e = 0; e < N; ++e) {
            const int i = tid + e * LOCAL_THREADS;
            *reinterpret_cast<float4*>(F + (i / PER_ROW) * Z::FP + (i % PER_ROW) * 4) = r[e];
        }
        stage_rows<TQ, DIM, LOCAL_THREADS>(q, a.ldq, n, sm + L::Q);
        if (!a.key_from_decay) stage_rows<TQ, DIM, LOCAL_THREADS>(k, a.ldq, n, sm + L::K_RAW);
    } else {
        float* dec = reinterpret_cast<float*>(sm + L::V4 + (2 * CH + NS) * 8);
        if (tid < CH) {
            dec[tid] = tid < n ? a.decay[(size_t)(row0 + tid) * a.ldd + h] : 1.f;
            dec[CH + tid] = (tid < n && a.kw != nullptr) ? a.kw[(size_t)(row0 + tid) * a.ldw + h] : 1.f;
        }
        stage_rows<TQ, DIM, LOCAL_THREADS>(q, a.ldq, n, sm + L::Q);
        stage_rows<TQ, DIM, LOCAL_THREADS>(k, a.ldq, n, sm + L::K);
    }
    uint32_t carries = 0u;
    constexpr int NV = CH * MAX_VDIM / 8 / LOCAL_THREADS;
    uint4 w[NV];
    const int pieces = vdim / 8;
#pragma unroll
    for (int e = 0; e < NV; ++e) {
        const int i = tid + e * LOCAL_THREADS, t = i / pieces, x = i - t * pieces;
        w[e] = t < n ? *reinterpret_cast<const uint4*>(a.v + (size_t)(row0 + t) * a.ldv + h * vdim + x * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int e = 0; e < NV; ++e) {
        const int i = tid + e * LOCAL_THREADS, t = i / pieces, x = i - t * pieces;
        if (t < CH) *reinterpret_cast<uint4*>(sm + L::V + t * VP + x * 16) = w[e];
        carries |= exponent_carry(w[e].x) | exponent_carry(w[e].y) | exponent_carry(w[e].z) | exponent_carry(w[e].w);
    }
    const bool endless = __syncthreads_or(carries != 0u);        // a value that is Inf or NaN

    // ---- A [t][s], s <= t, 16 x 16 blocks (i, j): a warp per block ---------------------------------------------------------
    Tile prod[2];                                                // columns s = 16 j + 8 nt + 2 (lane & 3) + {0, 1}
    float acc[2][4];
    const int g = lane >> 2, l2 = 2 * (lane & 3);
    int bi = 0, bj = 0;                                          // warp 0..9: (0,0) (1,0) (1,1) (2,0) ...
    if (warp < 10) {
        while ((bi + 1) * (bi + 2) / 2 <= warp) ++bi;
        bj = warp - bi * (bi + 1) / 2;
    }
    if constexpr (!CHANNELS) {
        double *E = reinterpret_cast<double*>(sm + L::V4), *P = E + CH, *Fs = P + CH;
        const float* dec = reinterpret_cast<const float*>(Fs + NS);
        const float* w = dec + CH;
        if (warp >= 14) {                                        // decays inside a sub-chunk: row s walks to its end
            const int s = tid - 14 * 32;
            double p = 1.0;
            Dd[s * SB + (s & 15)] = 1.f;
            for (int t = (s & 15) + 1; t < SB; ++t) {
                p *= (double)dec[(s & ~15) + t];
                Dd[s * SB + t] = (float)p;
            }
            E[s] = p;
            p = 1.0;                                             // and from the sub-chunk's start to the row
            for (int t = s & ~15; t <= s; ++t) p *= (double)dec[t];
            P[s] = p;
            if ((s & 15) == 15) Fs[s >> 4] = p;
        }
        if (warp < 10) {
            const unsigned aq = a_row(base + L::Q + bi * SB * Z::P, Z::P, lane), bk = b_row(base + L::K + bj * SB * Z::P, Z::P, lane);
#pragma unroll
            for (int ks = 0; ks < DIM / 16; ++ks) {
                uint32_t x[Z::PARTS][4], y[Z::PARTS][4];
#pragma unroll
                for (int p = 0; p < Z::PARTS; ++p) {
                    ldsm4(x[p], aq + p * Z::MAT + ks * 32);
                    ldsm4(y[p], bk + p * Z::MAT + ks * 32);
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    if constexpr (Z::PARTS == 1) prod[nt].lead(x[0], y[0][2 * nt], y[0][2 * nt + 1]);
                    else prod[nt].add6(x[0], x[1], x[2], y[0][2 * nt], y[0][2 * nt + 1], y[1][2 * nt], y[1][2 * nt + 1], y[2][2 * nt], y[2][2 * nt + 1]);
                }
            }
        }
        __syncthreads();                                         // the queries' place becomes A's; decays are there
        if (warp < 10) {
            double mid = 1.0;
            for (int j = bj + 1; j < bi; ++j) mid *= Fs[j];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = bi * SB + g + (e >> 1) * 8, s = bj * SB + nt * 8 + l2 + (e & 1);
                    const float d = bi == bj ? (t >= s ? Dd[s * SB + (t & 15)] : 0.f) : (float)(E[s] * (mid * P[t]));
                    acc[nt][e] = (bi == bj && t < s) ? 0.f : prod[nt][e] * a.q_scale * (w[s] * d);
                }
        }
        // K~: the keys times their weight and the decays to the chunk's end, in three parts
        for (int i = tid; i < CH * DIM / 2; i += LOCAL_THREADS) {
            const int s = i / (DIM / 2), x = i % (DIM / 2);
            char* at = sm + L::K + s * Z::P + x * 4;
            double to_end = E[s] * (double)w[s];
            for (int j = (s >> 4) + 1; j < NS; ++j) to_end *= Fs[j];
            const float f = (float)to_end;
            uint32_t r = *reinterpret_cast<uint32_t*>(at);
            float u = low_of(r), v = high_of(r);
            if constexpr (Z::PARTS == 3) {
                const uint32_t m = *reinterpret_cast<uint32_t*>(at + Z::MAT), l = *reinterpret_cast<uint32_t*>(at + 2 * Z::MAT);
                u = u + (low_of(m) + low_of(l));
                v = v + (high_of(m) + high_of(l));
            }
            store_split(at, Z::MAT, u * f, v * f);
        }
        if (tid == 0) store_decay(a.chunk_decay + 2 * unit, Fs[0] * Fs[1] * (Fs[2] * Fs[3]));
    } else {
        float* F = reinterpret_cast<float*>(sm + L::F);
        double* Fs = reinterpret_cast<double*>(sm + L::V4);      // [sub-chunk][channel]: its decay product
        {   // inside a sub-chunk: warp (sub, four rows s), eight lanes per row s with an eighth of the channels each
            const int sub = warp >> 2, s0 = (warp & 3) * 4, s = s0 + (lane >> 3), part = lane & 7;
            constexpr int NV = DIM / 32;                         // float4 groups of a lane: channels 32 x + 4 part
            float kk[NV * 4], d[NV * 4];
            const char* kr = sm + L::K_RAW + (sub * SB + s) * Z::P;
#pragma unroll
            for (int x = 0; x < NV; ++x)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int ch = x * 32 + part * 4 + u;
                    kk[x * 4 + u] = a.key_from_decay ? 1.f - F[(sub * SB + s) * Z::FP + ch] : bf_at(kr + ch * 2);
                    d[x * 4 + u] = 1.f;
                }
            for (int t = s0; t < SB; ++t) {
                const float* fr = F + (sub * SB + t) * Z::FP;
                const char* qr = sm + L::Q + (sub * SB + t) * Z::P;
                float sum = 0.f;
#pragma unroll
                for (int x = 0; x < NV; ++x) {
                    const float4 f4 = *reinterpret_cast<const float4*>(fr + x * 32 + part * 4);
                    const uint2 q2 = *reinterpret_cast<const uint2*>(qr + (x * 32 + part * 4) * 2);
                    const float fv[4] = {f4.x, f4.y, f4.z, f4.w};
                    const float qv[4] = {low_of(q2.x), high_of(q2.x), low_of(q2.y), high_of(q2.y)};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (t > s) d[x * 4 + u] *= fv[u];
                        sum += qv[u] * (kk[x * 4 + u] * d[x * 4 + u]);
                    }
                }
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                if (part == 0 && t >= s) Dd[(sub * SB + s) * SB + t] = sum;
            }
        }
        __syncthreads();
        const int ch = tid % DIM, sub = tid / DIM;               // a thread per (channel, sub-chunk)
        const bool walks = sub < NS;
        if (walks) {
            float f[SB];
            double p = 1.0;
#pragma unroll
            for (int t = 0; t < SB; ++t) {
                float* at = F + (sub * SB + t) * Z::FP + ch;
                f[t] = *at;
                p *= (double)f[t];
                *at = bf_at(sm + L::Q + (sub * SB + t) * Z::P + ch * 2) * (float)p;      // the query times the decays since the sub-chunk's start
            }
            Fs[sub * DIM + ch] = p;
            double e = 1.0;
#pragma unroll
            for (int t = SB - 1; t >= 0; --t) {
                const float kv = a.key_from_decay ? 1.f - f[t] : bf_at(sm + L::K_RAW + (sub * SB + t) * Z::P + ch * 2);
                store_split1(sm + L::K + (sub * SB + t) * Z::P + ch * 2, Z::MAT, kv * (float)e);     // K^: times those to its end
                e *= (double)f[t];
            }
        }
        __syncthreads();
        if (warp < 10) {
            if (bi == bj) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = g + (e >> 1) * 8, s = nt * 8 + l2 + (e & 1);
                        acc[nt][e] = t >= s ? Dd[(bi * SB + s) * SB + t] * a.q_scale : 0.f;
                    }
            } else {
                const unsigned bk = b_row(base + L::K + bj * SB * Z::P, Z::P, lane);
                const float* q0 = F + (bi * SB + g) * Z::FP + l2;
#pragma unroll 2
                for (int ks = 0; ks < DIM / 16; ++ks) {
                    uint32_t y[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) ldsm4(y[p], bk + p * Z::MAT + ks * 32);
                    Split3 x;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {                // columns 16 ks + 8 u + l2 of rows g and g + 8
                        double m0 = 1.0, m1 = 1.0;
                        for (int j = bj + 1; j < bi; ++j) {
                            const double2 w = *reinterpret_cast<const double2*>(Fs + j * DIM + ks * 16 + u * 8 + l2);
                            m0 *= w.x;
                            m1 *= w.y;
                        }
                        const float2 m = make_float2((float)m0, (float)m1);
                        const float2 r0 = *reinterpret_cast<const float2*>(q0 + ks * 16 + u * 8);
                        const float2 r8 = *reinterpret_cast<const float2*>(q0 + 8 * Z::FP + ks * 16 + u * 8);
                        split(r0.x * m.x, r0.y * m.y, x.h[2 * u], x.m[2 * u], x.l[2 * u]);
                        split(r8.x * m.x, r8.y * m.y, x.h[2 * u + 1], x.m[2 * u + 1], x.l[2 * u + 1]);
                    }
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
                        prod[nt].add6(x.h, x.m, x.l, y[0][2 * nt], y[0][2 * nt + 1], y[1][2 * nt], y[1][2 * nt + 1], y[2][2 * nt], y[2][2 * nt + 1]);
                }
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[nt][e] = prod[nt][e] * a.q_scale;
            }
        }
        __syncthreads();                                         // K^ becomes K~; the queries' and keys' place becomes A's
        if (walks) {
            double to_end = 1.0;
            for (int j = sub + 1; j < NS; ++j) to_end *= Fs[j * DIM + ch];
            const float m = (float)to_end;
            if (sub < NS - 1)
#pragma unroll 4
                for (int t = 0; t < SB; ++t) {
                    char* at = sm + L::K + (sub * SB + t) * Z::P + ch * 2;
                    store_split1(at, Z::MAT, (bf_at(at) + (bf_at(at + Z::MAT) + bf_at(at + 2 * Z::MAT))) * m);
                }
            if (sub == 0) store_decay(a.chunk_decay + 2 * (unit * DIM + ch), to_end * Fs[ch]);
        }
    }
    if (warp < 10) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                store_split(sm + L::A + (bi * SB + g + r * 8) * Z::AP + (bj * SB + nt * 8 + l2) * 2, Z::AMAT, acc[nt][2 * r], acc[nt][2 * r + 1]);
    }
    __syncthreads();

    // ---- O = A V: warp (16 rows, every fourth of 32 columns) ----------------------------------------------------------------
    const bool pairs = (a.vs & 1) == 0 && (a.ldo & 1) == 0;       // two neighbours of a row of `out` lie on 8 bytes
    {
        const int i = warp >> 2;
        for (int col0 = (warp & 3) * 32; col0 < vdim; col0 += 128) {
            Tile o[4];
            for (int j = 0; j <= i; ++j) {
                if (endless && j == i) {                         // the zeros above A's diagonal must not meet an Inf or NaN
                    for (int s = 0; s < SB; ++s)
#pragma unroll
                        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int t = g + (e >> 1) * 8, col = min(col0 + nt * 8 + l2 + (e & 1), vdim - 1);
                                if (s > t) continue;
                                const char* at = sm + L::A + (i * SB + t) * Z::AP + (i * SB + s) * 2;
                                const float w = bf_at(at) + (bf_at(at + Z::AMAT) + bf_at(at + 2 * Z::AMAT));
                                o[nt].hi[e] += w * bf_at(sm + L::V + (i * SB + s) * VP + col * 2);
                            }
                    continue;
                }
                uint32_t x[3][4], y[2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) ldsm4(x[p], a_row(base + L::A + p * Z::AMAT + i * SB * Z::AP + j * 32, Z::AP, lane));
#pragma unroll
                for (int u = 0; u < 2; ++u)                      // columns beyond vdim: the next row's, or the pad; not written
                    ldsm4t(y[u], a_row(base + L::V + j * SB * VP + min(col0 + u * 16, vdim - 8) * 2, VP, lane));
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) o[nt].add3(x[0], x[1], x[2], y[nt >> 1][2 * (nt & 1)], y[nt >> 1][2 * (nt & 1) + 1]);
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int col = col0 + nt * 8 + l2;
                if (col0 + nt * 8 >= vdim) continue;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int t = i * SB + g + r * 8;
                    if (t >= n) continue;
                    float* at = a.out + (size_t)(row0 + t) * a.ldo + (size_t)h * a.vs + col;
                    if (pairs) *reinterpret_cast<float2*>(at) = make_float2(o[nt][2 * r], o[nt][2 * r + 1]);
                    else {
                        at[0] = o[nt][2 * r];
                        at[1] = o[nt][2 * r + 1];
                    }
                }
            }
        }
    }
    // ---- L = K~^T V: warp (a quarter of the channels, every fourth of 32 columns) -----------------------------------------------
    {
        constexpr int MT = DIM / 64;
        const int m0 = (warp >> 2) * MT * 16;
        float* loc = a.local + unit * DIM * vdim;
        for (int col0 = (warp & 3) * 32; col0 < vdim; col0 += 128) {
            Tile s[MT][4];
#pragma unroll
            for (int ks = 0; ks < CH / 16; ++ks) {
                uint32_t y[2][4];
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    ldsm4t(y[u], a_row(base + L::V + ks * 16 * VP + min(col0 + u * 16, vdim - 8) * 2, VP, lane));
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    uint32_t x[3][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) ldsm4t(x[p], b_row(base + L::K + p * Z::MAT + ks * 16 * Z::P + (m0 + mt * 16) * 2, Z::P, lane));
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt) s[mt][nt].add3(x[0], x[1], x[2], y[nt >> 1][2 * (nt & 1)], y[nt >> 1][2 * (nt & 1) + 1]);
                }
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    if (col0 + nt * 8 >= vdim) continue;
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        *reinterpret_cast<float2*>(loc + (size_t)(m0 + mt * 16 + g + r * 8) * vdim + col0 + nt * 8 + l2) =
                            make_float2(s[mt][nt][2 * r], s[mt][nt][2 * r + 1]);
                }
        }
    }
    // ---- the normaliser: a value that is 1 in every row -------------------------------------------------------------------------
    if constexpr (!CHANNELS) {
        if (a.vs > vdim) {
            float* red = reinterpret_cast<float*>(sm + L::V4 + (2 * CH + NS) * 8) + 2 * CH;
            {   // sums of K~ over the rows: (channel, a share of the rows)
                constexpr int G = LOCAL_THREADS / DIM;
                const int ch = tid % DIM, gr = tid / DIM;
                float x = 0.f;
                for (int s = gr * (CH / G); s < (gr + 1) * (CH / G); ++s) {
                    const char* at = sm + L::K + s * Z::P + ch * 2;
                    x += bf_at(at) + (bf_at(at + Z::MAT) + bf_at(at + 2 * Z::MAT));
                }
                red[tid] = x;
                __syncthreads();
                if (tid < DIM) {
                    float y = 0.f;
                    for (int i = 0; i < G; ++i) y += red[i * DIM + tid];
                    a.local_n[unit * DIM + tid] = y;
                }
            }
            const int t = tid >> 3, part = tid & 7;              // sums of A's rows: eight threads each
            float x = 0.f;
            for (int s = part; s <= t; s += 8) {
                const char* at = sm + L::A + t * Z::AP + s * 2;
                x += bf_at(at) + (bf_at(at + Z::AMAT) + bf_at(at + 2 * Z::AMAT));
            }
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            x += __shfl_xor_sync(0xffffffffu, x, 2);
            x += __shfl_xor_sync(0xffffffffu, x, 4);
            if (part == 0 && t < n) a.out[(size_t)(row0 + t) * a.ldo + (size_t)h * a.vs + vdim] = x;
        }
    }
}

// The state before every chunk, in place of the states that the chunks build from nothing: a thread per four columns of a
// state row (or one number of the normaliser), eight chunks' loads in flight.
template <int DIM, bool CHANNELS>
__global__ void __launch_bounds__(256, CHANNELS ? 2 : 3) memory_chunk_prefix_kernel(const ChunkArgs a) {
    const int h = blockIdx.y, b = blockIdx.z, q4 = a.vdim / 4;
    const int e = blockIdx.x * 256 + threadIdx.x, n4 = DIM * q4;
    pdl_wait();
    const int slot = a.slots[b], chunks = chunks_of(a.seq_len[b], a.least);
    if (slot < 0 || chunks == 0) return;
    // the sequence's chunks that this round holds
    const int start = chunks_before(a, b, threadIdx.x & 31) - a.unit0;
    const int from = max(start, 0), nb = min(start + chunks, a.units) - from;
    if (nb <= 0 || e >= n4 + (a.vs > a.vdim ? DIM : 0)) return;
    const bool column = e >= n4;                                 // the normaliser's
    const int ch = column ? e - n4 : e / q4, col = column ? a.vdim : (e - ch * q4) * 4;
    float* st = a.state + (size_t)slot * a.state_stride + ((size_t)h * DIM + ch) * a.vs + col;
    const size_t u0 = (size_t)from * a.H + h;
    const float2* dec = reinterpret_cast<const float2*>(a.chunk_decay) + (CHANNELS ? u0 * DIM + ch : u0);
    const size_t dstep = CHANNELS ? (size_t)a.H * DIM : (size_t)a.H;
    if (column) {
        float* at = a.local_n + u0 * DIM + ch;
        float carry = *st;
        for (int i = 0; i < nb; ++i) {
            const float x = at[(size_t)i * a.H * DIM];
            at[(size_t)i * a.H * DIM] = carry;
            carry = decayed(dec[i * dstep], carry, x);
        }
        *st = carry;
        return;
    }
    const size_t step = (size_t)a.H * DIM * a.vdim;
    float* at = a.local + (u0 * DIM + ch) * a.vdim + col;
    float4 carry = make_float4(st[0], st[1], st[2], st[3]);
    // (offsets from the first chunk with a decay per channel, pointers that move with one per head: the compiler's registers then let two
    // and three blocks onto an SM.  9 heads of 128 x 256: 2048 rows 9.3 us, with pointers 11.8; a gate per head, 8 x 300 rows 18.6, with offsets 23.2)
    for (int i0 = 0; i0 < nb; i0 += 8) {
        const int left = nb - i0, first = CHANNELS ? i0 : 0;
        float4 x[8];
        float2 d[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < left) {
                x[i] = *reinterpret_cast<const float4*>(at + (first + i) * step);
                d[i] = dec[(first + i) * dstep];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < left) {
                *reinterpret_cast<float4*>(at + (first + i) * step) = carry;
                carry.x = decayed(d[i], carry.x, x[i].x);
                carry.y = decayed(d[i], carry.y, x[i].y);
                carry.z = decayed(d[i], carry.z, x[i].z);
                carry.w = decayed(d[i], carry.w, x[i].w);
            }
        if constexpr (!CHANNELS) {
            at += 8 * step;
            dec += 8 * dstep;
        }
    }
    st[0] = carry.x; st[1] = carry.y; st[2] = carry.z; st[3] = carry.w;
}

// Shared memory of memory_chunk_out: the queries' parts (per channel: times the decays since the chunk's start), 64 columns of
// the state in three parts, the decays since the chunk's start.
template <typename TQ, int DIM, bool CHANNELS>
struct OutPlan {
    using Z = Sizes<TQ, DIM>;
    static constexpr int QPARTS = CHANNELS ? 3 : Z::PARTS, COLS = 64;
    static constexpr int SP = COLS * 2 + 16, SMAT = DIM * SP;
    static constexpr int Q = 0, S = QPARTS * Z::MAT, P = S + 3 * SMAT, BYTES = P + (CHANNELS ? NS * DIM * 8 : CH * 4);
};

template <typename TQ, int DIM, bool CHANNELS>
__global__ void __launch_bounds__(OUT_THREADS, 2) memory_chunk_out_kernel(const ChunkArgs a) {
    using Z = Sizes<TQ, DIM>;
    using L = OutPlan<TQ, DIM, CHANNELS>;
    extern __shared__ __align__(16) char sm[];
    const int h = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int vdim = a.vdim;
    pdl_wait();
    const size_t unit = (size_t)blockIdx.y * a.H + h;
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    const float* S = a.local + unit * DIM * vdim;
    constexpr int NL = DIM * L::COLS / 4 / OUT_THREADS;          // float4 of a slice per thread
    float4 nx[NL];
    auto fetch = [&](int col0) {
#pragma unroll
        for (int e = 0; e < NL; ++e) {
            const int i = tid + e * OUT_THREADS, r = i / (L::COLS / 4), x = i % (L::COLS / 4);
            nx[e] = col0 + x * 4 < vdim ? *reinterpret_cast<const float4*>(S + (size_t)r * vdim + col0 + x * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);                                                    // (of scratch that nobody wrote, where there is no chunk)
    int row0 = 0, slot = -1;
    const int n = find_chunk(a, a.unit0 + blockIdx.y, lane, row0, slot);
    if (n <= 0 || slot < 0) return;
    float* P = reinterpret_cast<float*>(sm + L::P);
    if constexpr (CHANNELS) {
        double* Fs = reinterpret_cast<double*>(sm + L::P);
        constexpr int UNITS = DIM * NS / OUT_THREADS;            // (channel, sub-chunk) pairs of a thread
        float f[UNITS][SB];
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int i = tid + u * OUT_THREADS, ch = i % DIM, sub = i / DIM;
#pragma unroll
            for (int t = 0; t < SB; ++t)
                f[u][t] = sub * SB + t < n ? a.decay[(size_t)(row0 + sub * SB + t) * a.ldd + h * DIM + ch] : 1.f;
            double p = 1.0;
#pragma unroll
            for (int t = 0; t < SB; ++t) p *= (double)f[u][t];
            Fs[sub * DIM + ch] = p;
        }
        stage_rows<TQ, DIM, OUT_THREADS>((const TQ*)a.q + (size_t)row0 * a.ldq + h * DIM, a.ldq, n, sm + L::Q);
        __syncthreads();
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int i = tid + u * OUT_THREADS, ch = i % DIM, sub = i / DIM;
            double p = 1.0;
            for (int j = 0; j < sub; ++j) p *= Fs[j * DIM + ch];
#pragma unroll
            for (int t = 0; t < SB; ++t) {
                p *= (double)f[u][t];
                char* at = sm + L::Q + (sub * SB + t) * Z::P + ch * 2;
                store_split1(at, Z::MAT, bf_at(at) * (float)p);
            }
        }
    } else {
        stage_rows<TQ, DIM, OUT_THREADS>((const TQ*)a.q + (size_t)row0 * a.ldq + h * DIM, a.ldq, n, sm + L::Q);
        if (warp == 0) {                                         // decays since the chunk's start: two rows a lane, by doubling
            const int t = 2 * lane;
            const double d0 = t < n ? (double)a.decay[(size_t)(row0 + t) * a.ldd + h] : 1.0;
            const double d1 = t + 1 < n ? (double)a.decay[(size_t)(row0 + t + 1) * a.ldd + h] : 1.0;
            double d = d0 * d1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double x = __shfl_up_sync(0xffffffffu, d, o);
                if (lane >= o) d *= x;
            }
            const double up = __shfl_up_sync(0xffffffffu, d, 1);
            P[t] = (float)((lane ? up : 1.0) * d0);
            P[t + 1] = (float)d;
        }
    }
    const bool pairs = (a.vs & 1) == 0 && (a.ldo & 1) == 0;
    const int i = warp >> 1, cw = (warp & 1) * 32, g = lane >> 2, l2 = 2 * (lane & 3);
    const unsigned aq = a_row(base + L::Q + i * SB * Z::P, Z::P, lane);
    for (int col0 = 0; col0 < vdim; col0 += L::COLS) {
        if (col0) __syncthreads();                               // the slice before has been read
#pragma unroll
        for (int e = 0; e < NL; ++e) {
            const int x = tid + e * OUT_THREADS, r = x / (L::COLS / 4), y = x % (L::COLS / 4);
            char* at = sm + L::S + r * L::SP + y * 8;
            store_split(at, L::SMAT, nx[e].x, nx[e].y);
            store_split(at + 4, L::SMAT, nx[e].z, nx[e].w);
        }
        __syncthreads();
        if (col0 + L::COLS < vdim) fetch(col0 + L::COLS);
        float before[4][4];                                      // what the chunk's own rows gave
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = i * SB + g + r * 8, col = col0 + cw + nt * 8;
                const float* at = a.out + (size_t)(row0 + t) * a.ldo + (size_t)h * a.vs + col + l2;
                const bool live = t < n && col < vdim;
                float2 w = make_float2(0.f, 0.f);
                if (live) {
                    if (pairs) w = *reinterpret_cast<const float2*>(at);
                    else w = make_float2(at[0], at[1]);
                }
                before[nt][2 * r] = w.x;
                before[nt][2 * r + 1] = w.y;
            }
        Tile o[4];
#pragma unroll
        for (int ks = 0; ks < DIM / 16; ++ks) {
            uint32_t x[L::QPARTS][4], y[3][2][4];
#pragma unroll
            for (int p = 0; p < L::QPARTS; ++p) ldsm4(x[p], aq + p * Z::MAT + ks * 32);
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int u = 0; u < 2; ++u)
                    ldsm4t(y[p][u], a_row(base + L::S + p * L::SMAT + ks * 16 * L::SP + (cw + u * 16) * 2, L::SP, lane));
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int u = nt >> 1, w = 2 * (nt & 1);
                if constexpr (L::QPARTS == 1) o[nt].add3(x[0], y[0][u][w], y[0][u][w + 1], y[1][u][w], y[1][u][w + 1], y[2][u][w], y[2][u][w + 1]);
                else o[nt].add6(x[0], x[1], x[2], y[0][u][w], y[0][u][w + 1], y[1][u][w], y[1][u][w + 1], y[2][u][w], y[2][u][w + 1]);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = i * SB + g + r * 8;
            if (t >= n) continue;
            float f = a.q_scale;
            if constexpr (!CHANNELS) f *= P[t];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const int col = col0 + cw + nt * 8;
                if (col >= vdim) continue;
                float* at = a.out + (size_t)(row0 + t) * a.ldo + (size_t)h * a.vs + col + l2;
                const float x = before[nt][2 * r] + f * o[nt][2 * r], y = before[nt][2 * r + 1] + f * o[nt][2 * r + 1];
                if (pairs) *reinterpret_cast<float2*>(at) = make_float2(x, y);
                else {
                    at[0] = x;
                    at[1] = y;
                }
            }
        }
    }
    if constexpr (!CHANNELS) {
        if (a.vs > vdim) {                                       // n . q: four threads per row
            const int t = tid >> 2, part = tid & 3;
            const float* nv = a.local_n + unit * DIM;
            float x = 0.f;
            for (int ch = part; ch < DIM; ch += 4) {
                const char* at = sm + L::Q + t * Z::P + ch * 2;
                float qv = bf_at(at);
                if constexpr (Z::PARTS == 3) qv += bf_at(at + Z::MAT) + bf_at(at + 2 * Z::MAT);
                x += qv * nv[ch];
            }
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            x += __shfl_xor_sync(0xffffffffu, x, 2);
            if (part == 0 && t < n) {
                float* at = a.out + (size_t)(row0 + t) * a.ldo + (size_t)h * a.vs + vdim;
                *at = *at + a.q_scale * P[t] * x;
            }
        }
    }
}

template <typename TQ, int DIM, bool CHANNELS>
int launch(const ChunkArgs& a, cudaStream_t st) {
    using L = LocalPlan<TQ, DIM, CHANNELS>;
    using O = OutPlan<TQ, DIM, CHANNELS>;
    static OncePerDevice local_asked, out_asked;
    if (int rc = allow_shared(local_asked, memory_chunk_local_kernel<TQ, DIM, CHANNELS>, L::bytes(MAX_VDIM))) return rc;
    if (int rc = allow_shared(out_asked, memory_chunk_out_kernel<TQ, DIM, CHANNELS>, O::BYTES)) return rc;
    const dim3 grid(a.H, a.units);
    const int elements = DIM * (a.vdim / 4) + (a.vs > a.vdim ? DIM : 0);
    launch_pdl(memory_chunk_local_kernel<TQ, DIM, CHANNELS>, grid, dim3(LOCAL_THREADS), L::bytes(a.vdim), st, a);
    launch_pdl(memory_chunk_prefix_kernel<DIM, CHANNELS>, dim3((elements + 255) / 256, a.H, a.B), dim3(256), 0, st, a);
    launch_pdl(memory_chunk_out_kernel<TQ, DIM, CHANNELS>, grid, dim3(OUT_THREADS), O::BYTES, st, a);
    return (int)cudaGetLastError();
}

}  // namespace

// q, k: [rows, H * dim] of `qk_dtype` (float32 only with one decay per head), row pitch ldq; v: [rows, H * vdim] bfloat16, row
// pitch ldv; per_channel: decay[row * ldd + h * dim + channel], otherwise decay[row * ldd + h] (ldd = 0: the same in every row)
// and kw[row * ldw + h] (null: 1).  normaliser: vs = vdim + 1 state and output columns per head, the last one's value being 1
// (one decay per head only).  key_from_decay: the keys are 1 - decay, k is not read (per channel only).  Sequences of fewer than
// `least` rows are left alone.  The chunks of the others count through all sequences in order: this round takes unit0 .. unit0 +
// units - 1 (there may be fewer), and a step's rounds come in order.  local [units, H, dim, vdim], local_n [units, H, dim]
// (normaliser) and chunk_decay [units, H (, dim), 2] (on 8 bytes) are scratch.  dim 64 or 128, vdim a multiple of 8 up to 256;
// rows on 16 bytes.
QNN_API int qnn_memory_chunks(const void* q, const void* k, long long ldq, int qk_dtype, const void* v, long long ldv,
                              const float* decay, long long ldd, int per_channel, const float* kw, long long ldw, float q_scale,
                              int normaliser, int key_from_decay, const int* seq_row0, const int* seq_len, const int* slots,
                              float* state, long long state_stride, float* out, long long ldo, int B, int H, int dim, int vdim,
                              int least, int unit0, int units, float* local, float* local_n, float* chunk_decay, cudaStream_t st) {
    if (B <= 0 || units <= 0) return 0;
    if (H <= 0 || B > 65535 || units > 65535 || H > 65535 || unit0 < 0 || least < 1) return QNN_ERR_ARGUMENT;
    if (!seq_row0 || !seq_len || !slots || !state || !out || !local || !chunk_decay || (normaliser && !local_n)) return QNN_ERR_ARGUMENT;
    if ((dim != 64 && dim != 128) || vdim < 8 || vdim > MAX_VDIM || vdim % 8 != 0) return QNN_ERR_UNSUPPORTED;
    const int elt = qk_dtype == QNN_DT_BF16 ? 2 : 4;
    auto odd = [](const void* p) { return ((uintptr_t)p & 15) != 0; };
    if (odd(q) || (!key_from_decay && odd(k)) || odd(v) || ldq * elt % 16 != 0 || ldv % 8 != 0 || odd(local) || ((uintptr_t)chunk_decay & 7) != 0) return QNN_ERR_UNSUPPORTED;
    if (per_channel && (qk_dtype != QNN_DT_BF16 || normaliser || kw != nullptr || odd(decay) || ldd % 4 != 0)) return QNN_ERR_UNSUPPORTED;
    if (!per_channel && key_from_decay) return QNN_ERR_UNSUPPORTED;
    ChunkArgs a{q, k, ldq, (const bf16*)v, ldv, decay, ldd, kw, ldw, q_scale, seq_row0, seq_len, slots, B, least, out, ldo, state,
                state_stride, local, local_n, chunk_decay, unit0, units, H, vdim, vdim + (normaliser ? 1 : 0), key_from_decay};
    if (((uintptr_t)out & 7) != 0) return QNN_ERR_UNSUPPORTED;
    if (per_channel) return dim == 128 ? launch<bf16, 128, true>(a, st) : launch<bf16, 64, true>(a, st);
    if (qk_dtype == QNN_DT_BF16) return dim == 128 ? launch<bf16, 128, false>(a, st) : launch<bf16, 64, false>(a, st);
    return dim == 128 ? launch<float, 128, false>(a, st) : launch<float, 64, false>(a, st);
}
