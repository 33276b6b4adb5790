// Products of 8 bfloat16 rows with a few rows of weights, for the few outputs per row that feed float32 math (router logits, gates).
#pragma once
#include "common.cuh"

namespace qnn {

// dots[row][output] (rows `ldd` apart) of `rows` (1 to 8) rows x, ldx apart, with n rows w of `width`; float32, by all warps of the block.
// x, w and ldx lie on 16 bytes, width is a multiple of 8.  A sum is the one that a warp forms for one row and one output alone: lane l
// takes the pieces of eight l, l + 32, .. in order, one product after the other, and the lanes are added by a butterfly.  So a row has
// the same bits however many rows a step brings, whichever kernel forms it.
// A warp that forms one sum loads and unpacks both factors for every product; here it forms 4 x 4 of them, so that a factor serves four.
// (On the tensor cores, 16 at a time with the partial sums in 64 bits, 2048 rows of 2304 with 16 outputs take 6.4 us instead of 9.2, but
// with other bits than few rows have, so that a prompt's experts and gates depended on what shared its step; for few rows that form is the
// slower one, 8 rows of 1536 with 24 outputs 4.7 us instead of 2.3.)
// Two blocks of 256 threads share an SM (103 to 128 registers); 60 % of the issue slots are used, the rest waits for loads.  With room for
// three blocks (80 registers, the loads of one step fewer in flight) 2048 rows of 2304 with 16 outputs take 14.5 us.
constexpr int DOT_ROWS = 8, DOT_SIDE = 4;
__device__ __forceinline__ void row_dots(const bf16* x, long long ldx, int rows, const bf16* w, int n, int width, float* dots, int ldd) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    const int down = (rows + DOT_SIDE - 1) / DOT_SIDE, across = (n + DOT_SIDE - 1) / DOT_SIDE;
    for (int u = warp; u < down * across; u += nwarp) {
        const int r0 = u % down * DOT_SIDE, c0 = u / down * DOT_SIDE;
        const int nr = min(DOT_SIDE, rows - r0), nc = min(DOT_SIDE, n - c0);
        const bf16 *xr = x + (size_t)r0 * ldx, *wr = w + (size_t)c0 * width;
        float v[DOT_SIDE * DOT_SIDE];
#pragma unroll
        for (int i = 0; i < DOT_SIDE * DOT_SIDE; ++i) v[i] = 0.f;
#pragma unroll 2
        for (int k = lane * 8; k < width; k += 256) {
            Vec16<bf16> xv[DOT_SIDE], wv[DOT_SIDE];
#pragma unroll
            for (int r = 0; r < DOT_SIDE; ++r) {
                if (r < nr) xv[r].load(xr + (size_t)r * ldx + k);
                else xv[r].zero();
            }
#pragma unroll
            for (int c = 0; c < DOT_SIDE; ++c) {
                if (c < nc) wv[c].load(wr + (size_t)c * width + k);
                else wv[c].zero();
            }
            float xf[DOT_SIDE][8];
#pragma unroll
            for (int r = 0; r < DOT_SIDE; ++r) xv[r].unpack(xf[r]);
#pragma unroll
            for (int c = 0; c < DOT_SIDE; ++c) {
                float wf[8];
                wv[c].unpack(wf);
#pragma unroll
                for (int r = 0; r < DOT_SIDE; ++r)
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[r * DOT_SIDE + c] = fmaf(xf[r][j], wf[j], v[r * DOT_SIDE + c]);
            }
        }
        // warp_sum's butterfly for all 16 at once: at every distance a lane keeps half of what it holds, so 16 exchanges instead of 80
#pragma unroll
        for (int o = 16, half = 8; half > 0; o >>= 1, half >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < half; ++i) {
                const float keep = up ? v[i + half] : v[i], give = up ? v[i] : v[i + half];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        const int i = (lane >> 1 & 1) | (lane >> 2 & 1) << 1 | (lane >> 3 & 1) << 2 | (lane >> 4 & 1) << 3;   // which of the 16
        const int r = i / DOT_SIDE, c = i % DOT_SIDE;
        if (!(lane & 1) && r < nr && c < nc) dots[(r0 + r) * ldd + c0 + c] = v[0];
    }
    __syncthreads();
}

}  // namespace qnn
