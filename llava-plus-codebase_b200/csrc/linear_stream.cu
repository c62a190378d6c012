// Linears of a handful of rows (decode steps of 1..16 slots, tails of prompts) on bf16 weights: out[M, N] = A[M, K] W[N, K]^T with the fp32
// epilogue of linear_f32. A weight is used M times at most, so the kernel is a stream of weights and everything else stays out of its way:
//   * a CTA of 8 or 16 warps owns tiles of 16 output columns; its warps share a tile's K in units of 128, so that even the smallest matrix of a
//     model is spread over all SMs with its whole stream in flight, and the partial sums meet in shared memory in a fixed order;
//   * weights go from global memory straight into registers, 16 bytes per lane, in the order in which the tensor-core fragment wants them: the
//     sum over k may be taken in any order, so a lane's 8 consecutive k (of 32) are the fragment's k of two steps of 16 for A and B alike;
//   * two units per warp are in flight, across tile boundaries, and the first two are requested in front of the programmatic-dependent-launch
//     wait: weights depend on nothing, so they travel while the kernel in front finishes.
// 2..16 rows: mma.sync m16n8k16 (weights are the 16-row operand, the rows of A the 8 columns; 9..16 rows take two column tiles): tcgen05 wants
// 128 rows of A or a 128-row weight tile per CTA, which cuts these matrices into too few pieces. One row: the same stream on the FMA pipe.
// A four-layer model of width 2048 (weights 0.49 GB a step), one decode step: 8 slots 420 -> 274 us (before: a cast and the 128-row tile GEMM,
// 17-31 us a product; here 9), one slot 285 -> 256 us (before: one warp or a few per column). With the gated unit of a feed-forward inside its
// first product: 48 steps 12.23 -> 12.03 ms (one slot; before: one warp per output), 14.81 -> 14.53 (8 slots; before: a product and a launch of its own).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace b2 {
namespace {

constexpr int LS_UNIT = 128, LS_N = 16;

__device__ __forceinline__ void mma_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: column tiles of 8 rows of A (0: one row on the FMA pipe). A16: A lies there as bf16 rows of pitch K. GLU: a tile is 8 outputs of a gated unit,
// rows 0..7 their gate weights and 8..15 their up weights. An SM holds 16 warps: one CTA of 16, or two of 8.
template <int NT, bool A16, bool GLU, int LS_WARPS>
__global__ void __launch_bounds__(LS_WARPS * 32, 16 / LS_WARPS) linear_stream_kernel(LinearArgs a) {
    constexpr int COLS = NT == 0 ? 1 : 8 * NT, OUTS = GLU ? LS_N / 2 : LS_N;   // outputs per tile
    __shared__ float red[LS_WARPS][LS_N][COLS + (NT == 0 ? 0 : 1)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, kq = (lane & 3) * 8;
    const int units = (a.K + LS_UNIT - 1) / LS_UNIT, upw = (units + LS_WARPS - 1) / LS_WARPS;   // units per warp and tile
    const int tiles = (a.N + OUTS - 1) / OUTS, mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int steps = mine * upw;
    const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(a.W);

    uint4 w[2][4][2];
    auto load_w = [&](int s, uint4 (&u)[4][2]) {   // step s: tile s / upw of this CTA, unit (s % upw) * LS_WARPS + warp
        const int n0 = ((int)blockIdx.x + (s / upw) * (int)gridDim.x) * OUTS, k0 = ((s % upw) * LS_WARPS + warp) * LS_UNIT + kq;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + row + (GLU ? 0 : 8 * h);
            const __nv_bfloat16* p = W + (size_t)(n < a.N ? n + (GLU ? h * a.N : 0) : 0) * a.ldw + k0;
#pragma unroll
            for (int c = 0; c < 4; ++c) u[c][h] = s < steps && n < a.N && k0 + 32 * c < a.K ? ld_stream_16(p + 32 * c) : make_uint4(0, 0, 0, 0);
        }
    };
    load_w(0, w[0]);
    load_w(1, w[1]);
    pdl_trigger();
    pdl_wait();   // A, and the output when it is added to, come from the kernels in front

    float acc[NT == 0 ? 1 : NT][4];
#pragma unroll
    for (int t = 0; t < (NT == 0 ? 1 : NT); ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
    auto step = [&](int s, const uint4 (&u)[4][2]) {
        const int k0 = ((s % upw) * LS_WARPS + warp) * LS_UNIT + kq;
        if (NT == 0) {
            float x[4][8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool in = k0 + 32 * c < a.K;
                const float4 p = in ? *reinterpret_cast<const float4*>(a.A + k0 + 32 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 q = in ? *reinterpret_cast<const float4*>(a.A + k0 + 32 * c + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[c][0] = p.x; x[c][1] = p.y; x[c][2] = p.z; x[c][3] = p.w; x[c][4] = q.x; x[c][5] = q.y; x[c][6] = q.z; x[c][7] = q.w;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (a.round_a) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[c][i] = round_bf16(x[c][i]);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t v[4] = {u[c][h].x, u[c][h].y, u[c][h].z, u[c][h].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc[0][2 * h] = fmaf(x[c][2 * i], bf16_lo(v[i]), acc[0][2 * h]);
                        acc[0][2 * h + 1] = fmaf(x[c][2 * i + 1], bf16_hi(v[i]), acc[0][2 * h + 1]);
                    }
                }
            }
        } else {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int m = t * 8 + row;
                uint4 x[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    x[c] = make_uint4(0, 0, 0, 0);
                    if (m < a.M && k0 + 32 * c < a.K) {
                        if (A16) {
                            x[c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.A16) + (size_t)m * a.K + k0 + 32 * c);
                        } else {
                            const float* p = a.A + (size_t)m * a.lda + k0 + 32 * c;
                            const float4 f = *reinterpret_cast<const float4*>(p), g = *reinterpret_cast<const float4*>(p + 4);
                            x[c] = make_uint4(pack_bf16(f.x, f.y), pack_bf16(f.z, f.w), pack_bf16(g.x, g.y), pack_bf16(g.z, g.w));
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    mma_16x8x16(acc[t], u[c][0].x, u[c][1].x, u[c][0].y, u[c][1].y, x[c].x, x[c].y);
                    mma_16x8x16(acc[t], u[c][0].z, u[c][1].z, u[c][0].w, u[c][1].w, x[c].z, x[c].w);
                }
            }
        }
    };
    auto finish = [&](int s) {   // the last unit of a tile: the warps' sums meet, every thread writes some outputs
        if (s % upw != upw - 1) return;
        const int n0 = ((int)blockIdx.x + (s / upw) * (int)gridDim.x) * OUTS;
        __syncthreads();   // the previous tile's sums have been read
        if (NT == 0) {
            float v0 = acc[0][0] + acc[0][1], v1 = acc[0][2] + acc[0][3];
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1); v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 1); v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
            if ((lane & 3) == 0) { red[warp][row][0] = v0; red[warp][row + 8][0] = v1; }
        } else {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int c = t * 8 + (lane & 3) * 2;
                red[warp][row][c] = acc[t][0]; red[warp][row][c + 1] = acc[t][1];
                red[warp][row + 8][c] = acc[t][2]; red[warp][row + 8][c + 1] = acc[t][3];
            }
        }
#pragma unroll
        for (int t = 0; t < (NT == 0 ? 1 : NT); ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
        __syncthreads();
        const int i = threadIdx.x % OUTS, m = threadIdx.x / OUTS, n = n0 + i;
        if (m < a.M && m < COLS && n < a.N) {
            float v = 0.f;
#pragma unroll
            for (int q = 0; q < LS_WARPS; ++q) v += red[q][i][m];
            if constexpr (GLU) {
                float u = 0.f;
#pragma unroll
                for (int q = 0; q < LS_WARPS; ++q) u += red[q][i + OUTS][m];
                v = glu_act(v, u, a.glu);
                if (a.out16 != nullptr) reinterpret_cast<__nv_bfloat16*>(a.out16)[(size_t)m * a.ld_out + n] = __float2bfloat16_rn(v);
                else a.out[(size_t)m * a.ld_out + n] = v;
            } else linear_store(a.out + (size_t)m * a.ld_out + n, v, a.bias, n, a.act, a.alpha, a.accumulate);
        }
    };
    for (int s = 0; s < steps; s += 2) {
        step(s, w[0]);
        load_w(s + 2, w[0]);
        finish(s);
        if (s + 1 < steps) {
            step(s + 1, w[1]);
            load_w(s + 3, w[1]);
            finish(s + 1);
        }
    }
}

template <int NT, bool A16, bool GLU>
int launch_stream(const LinearArgs& a, cudaStream_t st) {
    const int outs = GLU ? LS_N / 2 : LS_N, tiles = (a.N + outs - 1) / outs, units = (a.K + LS_UNIT - 1) / LS_UNIT;
    // Two CTAs of 8 warps on an SM, or one of 16: the shorter one of the longest chains that a warp walks, in half units of weights. The end of a tile
    // (two barriers, the warps' sums) takes about half a unit's time, with more than 8 rows a whole one's; in a long stream of tiles whose last units
    // leave some of 8 warps idle (a head of 32000 outputs, K = 1536: 12 units), 16 warps were the faster form all the same. us a step, always 8 warps /
    // the shorter chain of units alone / this: four mixed layers of width 2048, one slot 205 / 197 / 194, 16 slots 271 / 265 / 258; of 1280, one slot 170 / 156 /
    // 154; of 3072, 8 slots 303 / 310 / 303; gated linear attention of 1536, 3 slots 80 / 73 / 71, 16 slots 121 / 125 / 116; window attention of 4096, 16 slots
    // 202 / 212 / 200.
    const int end = NT == 2 ? 2 : tiles >= 8 * num_sms() && units % 8 != 0 ? 0 : 1;
    const auto chain = [&](int ctas, int warps) { return ((tiles + ctas - 1) / ctas) * (2 * ((units + warps - 1) / warps) + end); };
    if (chain(num_sms(), 16) <= chain(2 * num_sms(), 8)) B2_CUDA_CHECK(launch_pdl(linear_stream_kernel<NT, A16, GLU, 16>, dim3(std::min(tiles, num_sms())), dim3(512), 0, st, a));
    else B2_CUDA_CHECK(launch_pdl(linear_stream_kernel<NT, A16, GLU, 8>, dim3(std::min(tiles, 2 * num_sms())), dim3(256), 0, st, a));
    B2_LAUNCH_CHECK();
    return 0;
}
}  // namespace

bool linear_streams(const LinearArgs& a) {
    return a.w_dtype == DT_BF16 && a.M >= 1 && a.M <= LINEAR_STREAM_MAX && a.K % 8 == 0 && a.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(a.W) & 15) == 0 &&
           a.norm.alpha == nullptr && (a.M == 1 || a.round_a) &&
           (a.M > 1 && a.A16 != nullptr ? (reinterpret_cast<uintptr_t>(a.A16) & 15) == 0 : a.A != nullptr && (a.M == 1 || a.lda % 4 == 0) && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0);
}

template <bool GLU>
static int stream_rows(const LinearArgs& a, cudaStream_t st) {
    if (a.M == 1) return launch_stream<0, false, GLU>(a, st);
    if (a.M <= 8) return a.A16 != nullptr ? launch_stream<1, true, GLU>(a, st) : launch_stream<1, false, GLU>(a, st);
    return a.A16 != nullptr ? launch_stream<2, true, GLU>(a, st) : launch_stream<2, false, GLU>(a, st);
}

int linear_stream_f32(const LinearArgs& a, cudaStream_t st) { return a.gated ? stream_rows<true>(a, st) : stream_rows<false>(a, st); }

}  // namespace b2
