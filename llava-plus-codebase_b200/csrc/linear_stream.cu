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

// What a launch computes: a product; a gated unit (a tile is 8 outputs, rows 0..7 their gate weights and 8..15 their up weights); a product `a` and a gated
// unit `b` of the same rows of A, side by side (the tiles of a, then those of b); the sum of two products on the same outputs (the units of a, then
// those of b; a's epilogue).
enum { LS_ONE = 0, LS_GLU = 1, LS_SIDE = 2, LS_SUM = 3 };

// NT: column tiles of 8 rows of A (0: one row on the FMA pipe). A16: A lies there as bf16 rows of pitch K (LS_SUM: looked up for each product).
// An SM holds 16 warps: one CTA of 16, or two of 8.
// RMS (one row): A passes a weighted RMS norm into shared memory on its way in, in every CTA: 8 KB read 148 times, beside weights that are on their way, for
// a launch of 2 us. (More rows would be 64 KB and more a CTA.)
template <int NT, bool A16, int FORM, bool RMS, int LS_WARPS>
__device__ __forceinline__ void linear_stream_body(const LinearArgs& a, const LinearArgs& b) {
    constexpr int COLS = NT == 0 ? 1 : 8 * NT;
    __shared__ float red[LS_WARPS][LS_N][COLS + (NT == 0 ? 0 : 1)];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, kq = (lane & 3) * 8;
    const int units0 = (a.K + LS_UNIT - 1) / LS_UNIT, units = units0 + (FORM == LS_SUM ? (b.K + LS_UNIT - 1) / LS_UNIT : 0);
    const int upw = (units + LS_WARPS - 1) / LS_WARPS;   // units per warp and tile
    constexpr int OUTS = FORM == LS_GLU ? LS_N / 2 : LS_N;   // outputs per tile of a
    const int tiles0 = (a.N + OUTS - 1) / OUTS, tiles = tiles0 + (FORM == LS_SIDE ? (b.N + LS_N / 2 - 1) / (LS_N / 2) : 0);
    const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int steps = mine * upw;

    uint4 w[2][4][2];
    auto load_w = [&](int s, uint4 (&u)[4][2]) {   // step s: tile s / upw of this CTA, unit (s % upw) * LS_WARPS + warp
        int tile = (int)blockIdx.x + (s / upw) * (int)gridDim.x, unit = (s % upw) * LS_WARPS + warp;
        const bool second = FORM == LS_SIDE ? tile >= tiles0 : FORM == LS_SUM && unit >= units0;
        const bool pairs = FORM == LS_GLU || (FORM == LS_SIDE && second);
        if (FORM == LS_SIDE && second) tile -= tiles0;
        if (FORM == LS_SUM && second) unit -= units0;
        const LinearArgs& p = second ? b : a;
        const int N = p.N, K = p.K, n0 = tile * (pairs ? LS_N / 2 : LS_N), k0 = unit * LS_UNIT + kq;
        const int64_t ldw = p.ldw;
        const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.W);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + row + (pairs ? 0 : 8 * h);
            const __nv_bfloat16* q = W + (size_t)(n < N ? n + (pairs ? h * N : 0) : 0) * ldw + k0;
#pragma unroll
            for (int c = 0; c < 4; ++c) u[c][h] = s < steps && n < N && k0 + 32 * c < K ? ld_stream_16(q + 32 * c) : make_uint4(0, 0, 0, 0);
        }
    };
    load_w(0, w[0]);
    load_w(1, w[1]);
    pdl_trigger();
    pdl_wait();   // A, and the output when it is added to, come from the kernels in front

    __shared__ __align__(16) float normed[RMS ? LINEAR_RMS_MAX_K : 4];
    if constexpr (RMS) {
        constexpr int U = LINEAR_RMS_MAX_K / 4 / (LS_WARPS * 32);
        float4 x[U], g[U];
        float q = 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = (threadIdx.x + u * LS_WARPS * 32) * 4;
            x[u] = c < a.K ? *reinterpret_cast<const float4*>(a.A + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            g[u] = c < a.K ? *reinterpret_cast<const float4*>(a.rms_w + c) : x[u];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) { q = fmaf(x[u].x, x[u].x, q); q = fmaf(x[u].y, x[u].y, q); q = fmaf(x[u].z, x[u].z, q); q = fmaf(x[u].w, x[u].w, q); }
        q = warp_sum(q);
        if (lane == 0) red[warp][0][0] = q;
        __syncthreads();
        q = warp_sum(lane < LS_WARPS ? red[lane][0][0] : 0.f);
        const float mul = 1.f / sqrtf(q / (float)a.K + a.rms_eps);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = (threadIdx.x + u * LS_WARPS * 32) * 4;
            float4 v = make_float4(x[u].x * mul * g[u].x, x[u].y * mul * g[u].y, x[u].z * mul * g[u].z, x[u].w * mul * g[u].w);
            if (a.round_a) v = make_float4(round_bf16(v.x), round_bf16(v.y), round_bf16(v.z), round_bf16(v.w));
            if (c < a.K) *reinterpret_cast<float4*>(normed + c) = v;
        }
        __syncthreads();
    }

    float acc[NT == 0 ? 1 : NT][4];
#pragma unroll
    for (int t = 0; t < (NT == 0 ? 1 : NT); ++t)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = 0.f;
    auto step = [&](int s, const uint4 (&u)[4][2]) {
        int unit = (s % upw) * LS_WARPS + warp;
        const bool second = FORM == LS_SUM && unit >= units0;
        if (second) unit -= units0;
        const LinearArgs& p = second ? b : a;
        const int k0 = unit * LS_UNIT + kq, K = p.K;
        const float* A = RMS ? normed : p.A;
        if (NT == 0) {
            float x[4][8];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool in = k0 + 32 * c < K;
                const float4 f = in ? *reinterpret_cast<const float4*>(A + k0 + 32 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 g = in ? *reinterpret_cast<const float4*>(A + k0 + 32 * c + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[c][0] = f.x; x[c][1] = f.y; x[c][2] = f.z; x[c][3] = f.w; x[c][4] = g.x; x[c][5] = g.y; x[c][6] = g.z; x[c][7] = g.w;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (a.round_a && !RMS) {
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
            const bool as16 = FORM == LS_SUM ? p.A16 != nullptr : A16;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int m = t * 8 + row;
                uint4 x[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    x[c] = make_uint4(0, 0, 0, 0);
                    if (m < a.M && k0 + 32 * c < K) {
                        if (as16) {
                            x[c] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.A16) + (size_t)m * K + k0 + 32 * c);
                        } else {
                            const float* r = A + (size_t)m * p.lda + k0 + 32 * c;
                            const float4 f = *reinterpret_cast<const float4*>(r), g = *reinterpret_cast<const float4*>(r + 4);
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
        const int tile = (int)blockIdx.x + (s / upw) * (int)gridDim.x;
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
        const bool pairs = FORM == LS_GLU || (FORM == LS_SIDE && tile >= tiles0);
        if (pairs) {
            const LinearArgs& p = FORM == LS_SIDE ? b : a;
            constexpr int H = LS_N / 2;
            const int i = threadIdx.x % H, m = threadIdx.x / H, n = (FORM == LS_SIDE ? tile - tiles0 : tile) * H + i;
            if (m < p.M && m < COLS && n < p.N) {
                float v = 0.f, u = 0.f;
#pragma unroll
                for (int q = 0; q < LS_WARPS; ++q) v += red[q][i][m];
#pragma unroll
                for (int q = 0; q < LS_WARPS; ++q) u += red[q][i + H][m];
                v = glu_act(v, u, p.glu);
                if (p.out16 != nullptr) reinterpret_cast<__nv_bfloat16*>(p.out16)[(size_t)m * p.ld_out + n] = __float2bfloat16_rn(v);
                else p.out[(size_t)m * p.ld_out + n] = v;
            }
        } else {
            const int i = threadIdx.x % LS_N, m = threadIdx.x / LS_N, n = tile * LS_N + i;
            if (m < a.M && m < COLS && n < a.N) {
                float v = 0.f;
#pragma unroll
                for (int q = 0; q < LS_WARPS; ++q) v += red[q][i][m];
                linear_store(a.out + (size_t)m * a.ld_out + n, v, a.bias, n, a.act, a.alpha, a.accumulate);
            }
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

template <int NT, bool A16, bool GLU, bool RMS, int LS_WARPS>
__global__ void __launch_bounds__(LS_WARPS * 32, 16 / LS_WARPS) linear_stream_kernel(LinearArgs a) {
    linear_stream_body<NT, A16, GLU ? LS_GLU : LS_ONE, RMS, LS_WARPS>(a, a);
}
template <int NT, bool A16, int FORM, bool RMS, int LS_WARPS>
__global__ void __launch_bounds__(LS_WARPS * 32, 16 / LS_WARPS) linear_stream_two_kernel(LinearArgs a, LinearArgs b) {
    linear_stream_body<NT, A16, FORM, RMS, LS_WARPS>(a, b);
}

// Whether a launch of `tiles` tiles of `units` units runs as one CTA of 16 warps an SM, not two of 8
template <int NT>
bool wide_ctas(int tiles, int units) {
    // Two CTAs of 8 warps on an SM, or one of 16: the shorter one of the longest chains that a warp walks, in half units of weights. The end of a tile
    // (two barriers, the warps' sums) takes about half a unit's time, with more than 8 rows a whole one's; in a long stream of tiles whose last units
    // leave some of 8 warps idle (a head of 32000 outputs, K = 1536: 12 units), 16 warps were the faster form all the same. us a step, always 8 warps /
    // the shorter chain of units alone / this: four mixed layers of width 2048, one slot 205 / 197 / 194, 16 slots 271 / 265 / 258; of 1280, one slot 170 / 156 /
    // 154; of 3072, 8 slots 303 / 310 / 303; gated linear attention of 1536, 3 slots 80 / 73 / 71, 16 slots 121 / 125 / 116; window attention of 4096, 16 slots
    // 202 / 212 / 200.
    const int end = NT == 2 ? 2 : tiles >= 8 * num_sms() && units % 8 != 0 ? 0 : 1;
    const auto chain = [&](int ctas, int warps) { return ((tiles + ctas - 1) / ctas) * (2 * ((units + warps - 1) / warps) + end); };
    return chain(num_sms(), 16) <= chain(2 * num_sms(), 8);
}

template <int NT, bool A16, bool GLU, bool RMS = false>
int launch_stream(const LinearArgs& a, cudaStream_t st) {
    const int outs = GLU ? LS_N / 2 : LS_N, tiles = (a.N + outs - 1) / outs;
    if (wide_ctas<NT>(tiles, (a.K + LS_UNIT - 1) / LS_UNIT)) B2_CUDA_CHECK(launch_pdl(linear_stream_kernel<NT, A16, GLU, RMS, 16>, dim3(std::min(tiles, num_sms())), dim3(512), 0, st, a));
    else B2_CUDA_CHECK(launch_pdl(linear_stream_kernel<NT, A16, GLU, RMS, 8>, dim3(std::min(tiles, 2 * num_sms())), dim3(256), 0, st, a));
    B2_LAUNCH_CHECK();
    return 0;
}
template <int NT, bool A16, int FORM, bool RMS = false>
int launch_two(const LinearArgs& a, const LinearArgs& b, cudaStream_t st) {
    const int tiles = (a.N + LS_N - 1) / LS_N + (FORM == LS_SIDE ? (b.N + LS_N / 2 - 1) / (LS_N / 2) : 0);
    // A product and a gated unit side by side have tiles in plenty (3.6 rounds of two CTAs an SM at width 1024, 1024 outputs and a unit of 2560) and run as two
    // CTAs of 8 warps, whose ends of tiles fall between each other's. us a layer in a chain of 3 to 12, 8 / 16 warps: gated linear attention of width 1024, 2 slots
    // 19.8 / 22.6, of 2048, one slot 36.8 / 38.7, 8 slots 39.9 / 40.3, of 2304, 4 slots 45.2 / 48.0; window attention of 2560, one slot 45.6 / 48.4, of 4096, 16
    // slots 101 / 103; of 135 measured (widths 1024 to 4096, 1 to 16 slots) 16 warps were ahead by more than 1 % in 3, by 2.4 % at most (1536, 4 slots 30.1 / 29.4).
    if constexpr (FORM == LS_SUM) {
        if (wide_ctas<NT>(tiles, (a.K + LS_UNIT - 1) / LS_UNIT + (b.K + LS_UNIT - 1) / LS_UNIT)) {
            B2_CUDA_CHECK(launch_pdl(linear_stream_two_kernel<NT, A16, FORM, RMS, 16>, dim3(std::min(tiles, num_sms())), dim3(512), 0, st, a, b));
            B2_LAUNCH_CHECK();
            return 0;
        }
    }
    B2_CUDA_CHECK(launch_pdl(linear_stream_two_kernel<NT, A16, FORM, RMS, 8>, dim3(std::min(tiles, 2 * num_sms())), dim3(256), 0, st, a, b));
    B2_LAUNCH_CHECK();
    return 0;
}
}  // namespace

bool linear_streams(const LinearArgs& a) {
    return a.w_dtype == DT_BF16 && a.M >= 1 && a.M <= LINEAR_STREAM_MAX && a.K % 8 == 0 && a.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(a.W) & 15) == 0 &&
           a.norm.alpha == nullptr && (a.M == 1 || a.round_a) &&
           (a.rms_w == nullptr || (a.M == 1 && a.K <= LINEAR_RMS_MAX_K && (reinterpret_cast<uintptr_t>(a.rms_w) & 15) == 0)) &&
           (a.M > 1 && a.A16 != nullptr ? (reinterpret_cast<uintptr_t>(a.A16) & 15) == 0 : a.A != nullptr && (a.M == 1 || a.lda % 4 == 0) && (reinterpret_cast<uintptr_t>(a.A) & 15) == 0);
}

template <bool GLU>
static int stream_rows(const LinearArgs& a, cudaStream_t st) {
    if (a.M == 1) return launch_stream<0, false, GLU>(a, st);
    if (a.M <= 8) return a.A16 != nullptr ? launch_stream<1, true, GLU>(a, st) : launch_stream<1, false, GLU>(a, st);
    return a.A16 != nullptr ? launch_stream<2, true, GLU>(a, st) : launch_stream<2, false, GLU>(a, st);
}

bool linear_stream_norms(const LinearArgs& a) { return a.rms_w != nullptr && !a.gated && linear_streams(a); }

int linear_stream_side_f32(const LinearArgs& a, const LinearArgs& b, cudaStream_t st) {
    B2_CHECK_ARG(linear_streams(a) && linear_streams(b) && !a.gated && b.gated && a.M == b.M && a.K == b.K && a.A == b.A && a.A16 == b.A16 && a.lda == b.lda && a.round_a == b.round_a && a.rms_w == b.rms_w,
                 "linear_stream_side: two products that do not share their rows");
    if (a.M == 1) return a.rms_w != nullptr ? launch_two<0, false, LS_SIDE, true>(a, b, st) : launch_two<0, false, LS_SIDE>(a, b, st);
    if (a.M <= 8) return a.A16 != nullptr ? launch_two<1, true, LS_SIDE>(a, b, st) : launch_two<1, false, LS_SIDE>(a, b, st);
    return a.A16 != nullptr ? launch_two<2, true, LS_SIDE>(a, b, st) : launch_two<2, false, LS_SIDE>(a, b, st);
}

int linear_stream_sum_f32(const LinearArgs& a, const LinearArgs& b, cudaStream_t st) {
    B2_CHECK_ARG(linear_streams(a) && linear_streams(b) && !a.gated && !b.gated && a.M == b.M && a.N == b.N && a.round_a == b.round_a && a.rms_w == nullptr && b.rms_w == nullptr, "linear_stream_sum: two products of other sizes");
    if (a.M == 1) return launch_two<0, false, LS_SUM>(a, b, st);
    return a.M <= 8 ? launch_two<1, false, LS_SUM>(a, b, st) : launch_two<2, false, LS_SUM>(a, b, st);
}

int linear_stream_f32(const LinearArgs& a, cudaStream_t st) {
    B2_CHECK_ARG(a.rms_w == nullptr || linear_stream_norms(a), "linear_stream: a norm that this product does not take");
    if (a.rms_w != nullptr) return launch_stream<0, false, false, true>(a, st);
    return a.gated ? stream_rows<true>(a, st) : stream_rows<false>(a, st);
}

}  // namespace b2
