// Whole-prompt matrix products on the 5th-generation tensor cores, two SMs per tile:
//     C[M, N] = A[M, K] * B[N, K]^T      bfloat16 in, float32 accumulation in tensor memory
// The same product and epilogues as gemm_tcgen05.cu; what differs is that a pair of CTAs (a
// thread-block cluster of two, on the two SMs of a TPC) computes a 256 x 256 tile with
// tcgen05.mma.cta_group::2.  Each CTA brings its own 128 rows of A and HALF of the B slab (128 of
// the 256 weight rows), so a CTA reads 32 KB from L2 per 64-deep slab instead of 48 KB for the same
// arithmetic; the single-CTA kernel is bound by exactly that traffic (its tensor pipe idles a quarter
// of the main loop), and the 32 KB stages leave room for 6 of them instead of 4.
//
//   * rank 0 of the pair is the leader: its lane issues every tcgen05.mma (M 256, N 256, K 16), reading
//     A and B from the shared memory of both CTAs and writing 128 accumulator rows into the tensor
//     memory of each;
//   * both CTAs run a TMA producer (cp.async.bulk.tensor with .cta_group::2, no multicast): the bytes of
//     both land on the LEADER's "full" barrier of the stage;
//   * tcgen05.commit.cta_group::2 with a CTA mask hands a stage back to both producers and, after the
//     last slab, an accumulator to the epilogue warps of both CTAs, each of which drains its own 128
//     rows; they return the accumulator with remote arrivals on the leader's barrier;
//   * the epilogue goes through shared memory (128 rows x 128 columns at a time) so that global memory
//     is written in whole 256-byte row pieces;
//   * tensor memory is allocated and freed with the .cta_group::2 forms by the same warp of both CTAs,
//     with cluster barriers after set-up and before the release.
// For the gated epilogue rank 0 loads the 128 gate rows and rank 1 the 128 matching up rows, so every
// accumulator row holds gate | up side by side, as in the single-CTA kernel.
//
// The plain product comes with tiles of 64, 96, .. 256 columns: its time is the rounds of tiles that the pairs take times one
// tile's walk over K, and a slab takes 0.16 us at 64 columns, 0.18 at 128, 0.24 at 192 and 0.30 at 256 (at 256 the tensor cores' time,
// below that of fetching: the 16 KB of A stay).  Measured (us, 256 columns / 128 / as chosen): of 2304 x 9216 256 rows 46.4 / 28.5 / 26.3 (64), 640
// rows 46.5 / 29.5 / 28.6 (96), 1280 rows 50.7 / 51.4 / 41.4 (192), 2809 rows 93.0 / 87.4 / 83.5 (192); of 4096 x 2304 640 rows 17.8 /
// 17.1 / 15.3 (192), 1280 rows 27.8 / 23.2 / 21.2 (160); of 1536 x 6144 2048 rows 36.4 / 35.1 / 28.9 (192).  With a short inner size the
// writing of a tile takes longer than its walk and hides the next one's, 2 us at 64 columns, 2.4 at 128, 3.7 at 256, and 3.5 already at 160: widths
// that are no multiple of 128 write pieces of rows that are shorter.  So the rule counts both (us, 256 columns / by the walk alone / as chosen:
// 8192 rows of 2048 x 512 20.7 / 22.2 / 20.7, of 2048 x 768 23.1 / 24.9 / 23.1, 4096 rows of 4096 x 256 17.3 / 20.0 / 17.3).  An element's
// sum runs over K in the same order whatever the tile, so the results are the same bit for bit.  (Sharing a tile's K among
// clusters of two or four pairs, summed through distributed shared memory in a fixed order, took 22 and 30 us for 256 and 640 rows of
// 2304 x 9216.  It is not in: it moves results by rounding, and with them ids that a model samples, where these are to stay the same.
// No precision speaks against it; the products of up to 128 rows share their K.)
//
// Every wait on an mbarrier is bounded (see gemm_tcgen05.cu); the two cluster barriers are reached by
// every thread of both CTAs on every path, in bounded time.
#include "common.cuh"
#include "tcgen05.cuh"

using namespace qnn;

#define EPI_NONE 0
#define EPI_GATED 2

namespace {

using namespace qnn::tc;
__device__ __forceinline__ void tmem_ld32(unsigned taddr, uint32_t (&r)[32]) { tmem_ld32_sync(taddr, r); }
inline int make_map(CUtensorMap* map, const void* base, long long rows, long long width, int box_rows) {
    return make_map_bf16(map, base, rows, width, box_rows, CU_TENSOR_MAP_L2_PROMOTION_L2_128B);
}

constexpr int BM = 128, BK = 64, UMMA_K = 16;        // BM: rows per CTA; the pair does 256
constexpr int A_BYTES = BM * BK * 2;                 // per CTA
constexpr int MAX_STAGES = 8;
template <int BN>                                    // columns of a pair's tile
struct Tile {
    static constexpr int B_BYTES = (BN / 2) * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;                // per CTA
    static constexpr int STAGES = BN >= 192 ? 6 : (BN >= 160 ? 7 : MAX_STAGES), RING_BYTES = STAGES * STAGE_BYTES;
    static constexpr int TMEM_COLS = BN <= 64 ? 64 : (BN <= 128 ? 128 : 256);                         // per accumulator: a power of two
    static_assert(BN % 32 == 0 && STAGE_BYTES % 1024 == 0, "the instruction's columns; the swizzle's 8 rows of 128 bytes");
    static_assert(RING_BYTES + BM * 128 * 2 + 1024 + 256 <= 232448, "a CTA's shared memory");
};
constexpr int STAGING_BYTES = BM * 128 * 2;          // the epilogue's 128 rows x 128 columns of bfloat16
constexpr int GEMM_THREADS = 192;
constexpr int SLAB_NS[7] = {160, 167, 175, 205, 235, 268, 300};             // time of a slab in tiles of 64, 96, .. 256 columns
constexpr int WRITE_NS[7] = {2000, 2400, 2400, 3500, 3600, 3700, 3700};      // of writing such a tile


// `bar` is a shared::cluster address: the leader's barrier, whichever CTA of the pair loads
__device__ __forceinline__ void tma_load_2d_pair(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void umma_bf16(unsigned tmem_d, uint64_t adesc, uint64_t bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives, once everything issued so far is done, on the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_pair(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}


struct __align__(8) Barriers {
    uint64_t full[MAX_STAGES];      // leader only: the slabs of both CTAs have landed (TMA bytes)
    uint64_t empty[MAX_STAGES];     // in each CTA: the MMAs that read the stage are done
    uint64_t acc_ready[2];      // in each CTA: an accumulator is complete
    uint64_t acc_free[2];       // leader only: the epilogues of both CTAs have read an accumulator
    uint32_t tmem_base;
    uint32_t failed;
};

__device__ __forceinline__ bool has_failed(Barriers* b) { return *reinterpret_cast<volatile uint32_t*>(&b->failed) != 0; }

// Persistent: a pair of CTAs per TPC walks over 256-row tiles t = pair, pair + pairs, ... (row tiles
// fastest, so the pairs that run together share their B slabs in L2).
template <int EPI, int BN>
__global__ void __launch_bounds__(GEMM_THREADS)
gemm_tcgen05_2cta_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         bf16* __restrict__ C, int M, int N, int K, int act, ActConsts actk, int* __restrict__ status) {
    static_assert(EPI == EPI_NONE || BN == 256, "a gated tile holds 128 gate and 128 up columns");
    constexpr int STAGES = Tile<BN>::STAGES, STAGE_BYTES = Tile<BN>::STAGE_BYTES, TMEM_COLS = Tile<BN>::TMEM_COLS;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* staging = smem + STAGES * STAGE_BYTES;
    Barriers* bars = reinterpret_cast<Barriers*>(staging + STAGING_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();                 // 0: leader
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int Nout = (EPI == EPI_GATED) ? N / 2 : N;
    constexpr int OUT_COLS = (EPI == EPI_GATED) ? BN / 2 : BN;          // output columns of a tile
    const int m_tiles = (M + 2 * BM - 1) / (2 * BM), n_tiles = (Nout + OUT_COLS - 1) / OUT_COLS;
    const int ntiles = m_tiles * n_tiles;
    const int nk = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&bars->acc_ready[a]), 1);
            mbar_init(smem_u32(&bars->acc_free[a]), 8);     // one arrival per epilogue warp of both CTAs
        }
        bars->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {   // the same warp of both CTAs allocates the pair's tensor memory, and frees it at the end
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&bars->tmem_base)), "r"(2 * TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();           // the peer's barriers exist before anything is sent to them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = bars->tmem_base;
    // Barriers and tensor memory are set up; only now wait for the kernels before this one (whose output
    // the loads below read), so that the set-up overlaps their tail.
    pdl_wait();

    if (warp == 0) {
        if (elect_one()) {
            // ---- producer (both CTAs) ---------------------------------------------------------
            int it = 0;                                    // slabs issued so far, over all tiles
            for (int tile = pair; tile < ntiles && !has_failed(bars); tile += pairs) {
                const int m0 = (tile % m_tiles) * (2 * BM) + (int)rank * BM;
                const int n0 = (tile / m_tiles) * OUT_COLS;
                // this CTA's half of the B slab: for the gated product the gate rows (rank 0) or the up rows (rank 1)
                const int brow = (EPI == EPI_GATED) ? (rank == 0 ? n0 : Nout + n0) : n0 + (int)rank * (BN / 2);
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait(smem_u32(&bars->empty[s]), ((it / STAGES) - 1) & 1)) {
                        atomicOr(status, 1);
                        bars->failed = 1;
                        break;
                    }
                    const unsigned full_local = smem_u32(&bars->full[s]);
                    const unsigned full_leader = map_to_rank(full_local, 0);
                    const unsigned a_dst = smem_u32(smem + s * STAGE_BYTES), b_dst = a_dst + A_BYTES;
                    if (rank == 0) mbar_expect_tx(full_local, 2 * STAGE_BYTES);
                    tma_load_2d_pair(a_dst, &map_a, full_leader, kb * BK, m0);
                    tma_load_2d_pair(b_dst, &map_b, full_leader, kb * BK, brow);
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // ---- tensor-core issue (leader) ----------------------------------------------------
            // instruction descriptor: D float32, A and B bfloat16, both K-major, N >> 3, M >> 4 (M = 256 over the pair)
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(BN >> 3) << 17) | ((unsigned)((2 * BM) >> 4) << 24);
            int it = 0, i = 0;                             // slabs consumed; tiles done by this pair
            for (int tile = pair; tile < ntiles && !has_failed(bars); tile += pairs, ++i) {
                const int a = i & 1;
                if (i >= 2 && !mbar_wait(smem_u32(&bars->acc_free[a]), ((i >> 1) - 1) & 1)) {
                    atomicOr(status, 8);
                    bars->failed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned acc = tmem + a * TMEM_COLS;
                bool ok = true;
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(smem_u32(&bars->full[s]), (it / STAGES) & 1)) {
                        atomicOr(status, 2);
                        bars->failed = 1;
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned a_addr = smem_u32(smem + s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        // 16 elements further along K = 32 bytes inside the 128-byte swizzled row
                        umma_bf16(acc, umma_desc(a_addr + k * UMMA_K * 2), umma_desc(b_addr + k * UMMA_K * 2), idesc,
                                  (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit_pair(smem_u32(&bars->empty[s]));     // the stage is free in both CTAs once these MMAs have read it
                }
                umma_commit_pair(smem_u32(&bars->acc_ready[a]));     // arrives in both CTAs when everything issued so far is done
                if (!ok) break;
            }
        }
    } else {
        // ---- epilogue (both CTAs): warps 2..5, each owns the 32 accumulator lanes (rows) of its quarter ----
        const int quarter = warp & 3;
        int i = 0;
        for (int tile = pair; tile < ntiles; tile += pairs, ++i) {
            const int a = i & 1;
            const int m0 = (tile % m_tiles) * (2 * BM) + (int)rank * BM, n0 = (tile / m_tiles) * OUT_COLS;
            if (!mbar_wait(smem_u32(&bars->acc_ready[a]), (i >> 1) & 1)) {
                atomicOr(status, 4);
                bars->failed = 1;
                break;
            }
            if (has_failed(bars)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m = m0 + quarter * 32 + lane;
            const unsigned lane_addr = tmem + a * TMEM_COLS + ((unsigned)(quarter * 32) << 16);
            if ((Nout & 7) == 0) {
                // Through shared memory, 128 columns at a time: each thread leaves its row as bfloat16
                // (16-byte chunks XOR-ed with the row number, so that neither side has bank conflicts), then
                // the warp writes its 32 rows to global memory two rows (2 x 256 bytes) per instruction.
                // A thread-per-row store straight from registers touches 32 lines per instruction and made
                // the epilogue 4.4 us of a 19 us product.
                unsigned char* mine = staging + quarter * (32 * 256);
#pragma unroll 1
                for (int h0 = 0; h0 < OUT_COLS; h0 += 128) {
                    const int part = min(OUT_COLS - h0, 128);
#pragma unroll 1
                    for (int c0 = h0; c0 < h0 + part; c0 += 32) {
                        uint32_t v[32];
                        tmem_ld32(lane_addr + c0, v);
                        float f[32];
                        if (EPI == EPI_GATED) {
                            uint32_t u[32];
                            tmem_ld32(lane_addr + BN / 2 + c0, u);
#pragma unroll
                            for (int j = 0; j < 32; ++j) f[j] = activate_fast(__uint_as_float(v[j]), act) * __uint_as_float(u[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
                            if (act >= QNN_ACT_ALONE) {      // an activation without a gate: act(A B^T)
#pragma unroll
                                for (int j = 0; j < 32; ++j) f[j] = activate_fast(f[j], act - QNN_ACT_ALONE, actk);
                            }
                        }
                        if (c0 + 32 >= OUT_COLS) {
                            // the last columns are in registers: hand the accumulator back to the leader
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&bars->acc_free[a]), 0));
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int ch = (c0 - h0) / 8 + j;
                            uint4 pk;
                            pk.x = pack_bf16(f[j * 8 + 0], f[j * 8 + 1]);
                            pk.y = pack_bf16(f[j * 8 + 2], f[j * 8 + 3]);
                            pk.z = pack_bf16(f[j * 8 + 4], f[j * 8 + 5]);
                            pk.w = pack_bf16(f[j * 8 + 6], f[j * 8 + 7]);
                            *reinterpret_cast<uint4*>(mine + lane * 256 + ((ch ^ (lane & 15)) << 4)) = pk;
                        }
                    }
                    __syncwarp();
#pragma unroll 4
                    for (int rr = 0; rr < 32; rr += 2) {
                        const int r = rr + (lane >> 4), pos = lane & 15;
                        const int row = m0 + quarter * 32 + r;
                        const int col = n0 + h0 + ((pos ^ (r & 15)) << 3);
                        const uint4 pk = *reinterpret_cast<const uint4*>(mine + r * 256 + (pos << 4));
                        const bool staged = OUT_COLS % 128 == 0 || (pos ^ (r & 15)) < part / 8;
                        if (staged && row < M && col < Nout) *reinterpret_cast<uint4*>(C + (size_t)row * Nout + col) = pk;
                    }
                    __syncwarp();
                }
                continue;
            }
#pragma unroll 1
            for (int c0 = 0; c0 < OUT_COLS; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(lane_addr + c0, v);
                float f[32];
                if (EPI == EPI_GATED) {
                    uint32_t u[32];
                    tmem_ld32(lane_addr + BN / 2 + c0, u);
#pragma unroll
                    for (int j = 0; j < 32; ++j) f[j] = activate_fast(__uint_as_float(v[j]), act) * __uint_as_float(u[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
                    if (act >= QNN_ACT_ALONE) {              // an activation without a gate: act(A B^T)
#pragma unroll
                        for (int j = 0; j < 32; ++j) f[j] = activate_fast(f[j], act - QNN_ACT_ALONE, actk);
                    }
                }
                if (c0 + 32 >= OUT_COLS) {
                    // the last columns are in registers: hand the accumulator back to the leader before storing them
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&bars->acc_free[a]), 0));
                }
                if (m < M) {
                    bf16* dst = C + (size_t)m * Nout + n0 + c0;
                    if (n0 + c0 + 32 <= Nout && ((Nout & 7) == 0)) {
#pragma unroll
                        for (int j = 0; j < 32; j += 8) Vec16<bf16>::store(dst + j, f + j);
                    } else {
                        for (int j = 0; j < 32; ++j)
                            if (n0 + c0 + j < Nout) dst[j] = __float2bfloat16_rn(f[j]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();           // neither CTA frees tensor memory, or leaves, while the other still uses the pair's
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TMEM_COLS) : "memory");
    }
}


typedef void (*Kernel)(CUtensorMap, CUtensorMap, bf16*, int, int, int, int, ActConsts, int*);

// Columns of a plain product's tile: the least time, of a round of tiles the longer of walking K and writing, of the last both;
// a narrower one where that is 2 % less (8192 rows of 6144 x 1536, a tie: 256 columns 102 us, 192 105).
int plain_tile_cols(long long M, long long N, long long K, int sm_count) {
    const long long m_tiles = (M + 2 * BM - 1) / (2 * BM), pairs = sm_count / 2 > 0 ? sm_count / 2 : 1;
    long long best = 0;
    int cols = 256;
    for (int c = 256; c >= 64; c -= 32) {
        const long long rounds = (m_tiles * ((N + c - 1) / c) + pairs - 1) / pairs;
        const long long walk = (K + BK - 1) / BK * SLAB_NS[c / 32 - 2], write = WRITE_NS[c / 32 - 2];
        const long long t = (rounds - 1) * (walk > write ? walk : write) + walk + write;
        if (c == 256 || t * 50 < best * 49) best = t, cols = c;
    }
    return cols;
}

}  // namespace

// The columns that qnn_gemm_tcgen05_2cta chooses for a plain product of this size on a device of so many SMs; ..._cols: of a long K.
QNN_API int qnn_gemm_tcgen05_2cta_width(int M, int N, int K, int sm_count) { return plain_tile_cols(M, N, K, sm_count); }
QNN_API int qnn_gemm_tcgen05_2cta_cols(int M, int N, int sm_count) { return plain_tile_cols(M, N, 1 << 24, sm_count); }

// The product of qnn_gemm_tcgen05 (same arguments, same meaning of `status`) computed by pairs of CTAs.
// Returns QNN_ERR_UNSUPPORTED when the device cannot hold a pair (the caller then uses the single-CTA
// kernel).  tile_cols: columns of a plain product's tile (64, 128 or 256), 0 to have them chosen.
QNN_API int qnn_gemm_tcgen05_2cta(const void* A, const void* B, void* C, int M, int N, int K, int epi, int act,
                                  float act_a, float act_b, int tile_cols, int* status, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || (K & 7) || ((((uintptr_t)A | (uintptr_t)B | (uintptr_t)C) & 15) != 0)) return QNN_ERR_UNSUPPORTED;
    if (epi != EPI_NONE && epi != EPI_GATED) return QNN_ERR_ARGUMENT;
    if (tile_cols != 0 && (epi != EPI_NONE || (tile_cols != 64 && tile_cols != 128 && tile_cols != 256))) return QNN_ERR_ARGUMENT;
    if (epi == EPI_GATED && (N & 1)) return QNN_ERR_ARGUMENT;
    const int Nout = epi == EPI_GATED ? N / 2 : N;
    const int sm_count = device_sms();
    const long long m_tiles = (M + 2 * BM - 1) / (2 * BM);
    const int cols = epi == EPI_GATED ? 128 : (tile_cols != 0 ? tile_cols : plain_tile_cols(M, N, K, sm_count));
    const long long ntiles = m_tiles * ((Nout + cols - 1) / cols);
    if (ntiles > 0x3fffffffLL) return QNN_ERR_UNSUPPORTED;
    CUtensorMap map_a, map_b;
    int rc = make_map(&map_a, A, M, K, BM);
    if (rc) return rc;
    rc = make_map(&map_b, B, N, K, epi == EPI_GATED ? 128 : cols / 2);
    if (rc) return rc;
    struct Form { Kernel kernel; int ring_bytes; };
    static const Form forms[8] = {        // gated, then plain by columns: 64, 96, .. 256
        {gemm_tcgen05_2cta_kernel<EPI_GATED, 256>, Tile<256>::RING_BYTES}, {gemm_tcgen05_2cta_kernel<EPI_NONE, 64>, Tile<64>::RING_BYTES},
        {gemm_tcgen05_2cta_kernel<EPI_NONE, 96>, Tile<96>::RING_BYTES},    {gemm_tcgen05_2cta_kernel<EPI_NONE, 128>, Tile<128>::RING_BYTES},
        {gemm_tcgen05_2cta_kernel<EPI_NONE, 160>, Tile<160>::RING_BYTES},  {gemm_tcgen05_2cta_kernel<EPI_NONE, 192>, Tile<192>::RING_BYTES},
        {gemm_tcgen05_2cta_kernel<EPI_NONE, 224>, Tile<224>::RING_BYTES},  {gemm_tcgen05_2cta_kernel<EPI_NONE, 256>, Tile<256>::RING_BYTES}};
    const int which = epi == EPI_GATED ? 0 : cols / 32 - 1;
    const Kernel kern = forms[which].kernel;
    const size_t smem = (size_t)forms[which].ring_bytes + STAGING_BYTES + sizeof(Barriers) + 1024;
    static OncePerDevice asked[8];
    static KnownPerDevice known[8];
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    if (const int err = allow_shared(asked[which], kern, smem)) return err;
    const int max_pairs = known[which].get(current_device(), 0, [&] {        // of this kernel that the device holds at once
        cfg.gridDim = dim3(2 * (sm_count / 2));
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
            (void)cudaGetLastError();
            return -1;
        }
        return n < sm_count / 2 ? n : sm_count / 2;
    });
    if (max_pairs < 0) return QNN_ERR_UNSUPPORTED;
    const int pairs = ntiles < max_pairs ? (int)ntiles : max_pairs;
    cfg.gridDim = dim3(2 * pairs);
    cfg.numAttrs = (qnn::pdl_enabled() && 2ll * pairs <= qnn::pdl_max_grid()) ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map_a, map_b, (bf16*)C, M, N, K, act, ActConsts{act_a, act_b}, status);
    return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
