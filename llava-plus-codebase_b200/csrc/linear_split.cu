// Linears in true fp32 for portions of a prompt, on the tensor cores: out[M, N] = alpha act(A[M, K] W[N, K]^T + bias) (+ out), all fp32, with both
// operands as three bf16 parts and six products of each pair (split.cuh). The tensor core cuts its fp32 sums off after every step of 16, so an
// accumulator spans one block of 64 of K only; the blocks are added up in fp32 registers.
//   1. split_rows_kernel writes the parts of A and of W (per call: the weights stay fp32 in memory, and a pass over them is short beside the product);
//      a W whose parts exceed the scratch goes in blocks of rows;
//   2. linear_split_kernel: one tile of 128 x BN per CTA, warp 0 TMA producer (a stage: the three parts of 64 columns of A and W), warp 1 MMA
//      issuer, warps 2..9 take every block's accumulator out of TMEM (two of them, so that the next block's products run meanwhile).
// What bounds it: the stream of parts into the SM (96 KB per block at BN = 128 against 1536 clk of products), then too few tiles at small N.
// 600 rows, 13 products of a state-space + RWKV pair of width 1024 (33 GFLOP): 2512 us on linear_tiled_kernel -> 413 us and 86 us of cutting; the
// pair's error against 64 bits falls from 1.4e-6 to 3.6e-7.
#include <cuda.h>

#include <algorithm>

#include "kernels.h"
#include "split.cuh"

namespace b2 {

int make_tmap_parts(CUtensorMap* map, const void* ptr, int pitch, int64_t rows, int planes, int box_rows);

namespace {

constexpr int LX_M = 128, LX_K = 64, LX_THREADS = 320;

template <int BN>
struct LxCfg {
    static constexpr int A_BYTES = 3 * LX_M * 128, B_BYTES = 3 * BN * 128, STAGE = A_BYTES + B_BYTES, STAGES = BN == 128 ? 2 : 3;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 128;
};

// rows of fp32 -> [part][rows][pitch] bf16, entries past K zero
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ in, int64_t ld, int rows, int K, int pitch, __nv_bfloat16* __restrict__ out, int vec) {
    pdl_enter();
    const int chunks = pitch >> 3;
    const int64_t total = (int64_t)rows * chunks, plane = (int64_t)rows * pitch;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
        const int64_t r = e / chunks;
        const int c = (int)(e - r * chunks) * 8;
        float x[8];
        load8(in + r * ld, c, K, vec != 0, x);
        uint4 h, m, l;
        split8(x, h, m, l);
        __nv_bfloat16* o = out + r * pitch + c;
        *reinterpret_cast<uint4*>(o) = h;
        *reinterpret_cast<uint4*>(o + plane) = m;
        *reinterpret_cast<uint4*>(o + 2 * plane) = l;
    }
}

__device__ __noinline__ float lx_act(float v, int act) { return epi_post_act(v, act); }

// Outputs [n0, n1) of one row in plain fp32, for a row with an operand that has no parts (split.cuh). A sum that has become NaN stays one. (Its
// arguments are values: by reference to the kernel's parameter block the whole kernel reads that block through memory, 2 us a launch: 600 rows
// through a state-space + RWKV pair of width 1024 846 -> 873 us.)
__device__ __noinline__ void lx_plain(const float* x, const float* w, int64_t ldw, int K, float* o, const float* bias, int n0, int n1, int act, float alpha, int accumulate) {
    for (int n = n0; n < n1; ++n) {
        float acc = 0.f;
        for (int k = 0; k < K && acc == acc; ++k) acc = fmaf(x[k], w[(size_t)n * ldw + k], acc);
        linear_store(o + n, acc, bias, n, act, alpha, accumulate);
    }
}

template <int BN>
__global__ void __launch_bounds__(LX_THREADS, 1) linear_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, LinearArgs a) {
    using Cfg = LxCfg<BN>;
    constexpr int CH = BN / 2;   // columns per epilogue thread
    extern __shared__ uint8_t lx_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lx_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE);
    uint64_t *full = bars, *empty = bars + Cfg::STAGES, *acc_full = bars + 2 * Cfg::STAGES /*[2]*/, *acc_empty = acc_full + 2 /*[2]*/;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int num_m = (a.M + LX_M - 1) / LX_M, m0 = (int)(blockIdx.x % num_m) * LX_M, n0 = (int)(blockIdx.x / num_m) * BN;
    const int blocks = (a.K + LX_K - 1) / LX_K;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_w);
        for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 2 * BN); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *tmem_slot;
    pdl_trigger_small();   // (behind the allocation: see tmem_alloc)
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            for (int b = 0; b < blocks; ++b) {
                mbar_wait(&empty[stage], phase ^ 1);
                uint8_t* d = smem + stage * Cfg::STAGE;
                mbar_arrive_expect_tx(&full[stage], Cfg::STAGE);
                for (int p = 0; p < 3; ++p) tma_load_3d(d + p * LX_M * 128, &tm_a, &full[stage], b * LX_K, m0, p);
                for (int p = 0; p < 3; ++p) tma_load_3d(d + Cfg::A_BYTES + p * BN * 128, &tm_w, &full[stage], b * LX_K, n0, p);
                if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // walked by the whole warp, an elected lane issues (elect_one, common.cuh): 600 rows through a state-space and an attention layer of width 1024
        // (13 of these Linears) 818 us, 772
        const bool leader = elect_one();
        constexpr uint32_t idesc = make_idesc_bf16_f32(LX_M, BN);
        int stage = 0;
        uint32_t phase = 0;
        for (int b = 0; b < blocks; ++b) {
            mbar_wait(&acc_empty[b & 1], ((b >> 1) & 1) ^ 1);
            mbar_wait(&full[stage], phase);
            tc_fence_after();
            const uint32_t s = smem_u32(smem + stage * Cfg::STAGE);
            const uint64_t da = make_sw128_kmajor_desc(s), db = make_sw128_kmajor_desc(s + Cfg::A_BYTES);
#pragma unroll 1
            for (int i = 0; i < 6; ++i) {
                const uint32_t pa = (SPLIT_A >> (2 * i)) & 3u, pb = (SPLIT_B >> (2 * i)) & 3u;
                if (leader)
#pragma unroll
                    for (int k = 0; k < LX_K / 16; ++k)
                        umma_bf16(tm + (b & 1) * BN, da + (pa * (LX_M * 8) + 2 * k), db + (pb * (BN * 8) + 2 * k), idesc, (i | k) != 0 ? 1u : 0u);
            }
            if (leader) {
                umma_commit(&empty[stage]);
                umma_commit(&acc_full[b & 1]);
            }
            __syncwarp();
            if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2, m = m0 + q * 32 + lane;
        float acc[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) acc[i] = 0.f;
        for (int b = 0; b < blocks; ++b) {
            mbar_wait(&acc_full[b & 1], (b >> 1) & 1);
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < CH / 32; ++c) {
                uint32_t v[32];
                __syncwarp();
                tmem_ld_32x32(tm + (static_cast<uint32_t>(q * 32) << 16) + (b & 1) * BN + half * CH + c * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[c * 32 + i] += __uint_as_float(v[i]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b & 1]);
        }
        bool plain = false;
#pragma unroll
        for (int i = 0; i < CH; ++i) plain |= acc[i] != acc[i];
        if (m < a.M && plain) {
            lx_plain(a.A + (size_t)m * a.lda, reinterpret_cast<const float*>(a.W), a.ldw, a.K, a.out + (size_t)m * a.ld_out, a.bias, n0 + half * CH, min(n0 + (half + 1) * CH, a.N), a.act, a.alpha,
                     a.accumulate);
        } else if (m < a.M) {
            const int c0 = n0 + half * CH;
            float* o = a.out + (size_t)m * a.ld_out + c0;
            const bool vec = a.ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
#pragma unroll
            for (int c = 0; c < CH; c += 4) {
                float y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    y[i] = acc[c + i] + (a.bias != nullptr && c0 + c + i < a.N ? a.bias[c0 + c + i] : 0.f);
                    if (a.act != 0) y[i] = lx_act(y[i], a.act);
                    y[i] *= a.alpha;
                }
                if (vec && c0 + c + 4 <= a.N) {
                    if (a.accumulate) {
                        const float4 p = *reinterpret_cast<const float4*>(o + c);
                        y[0] += p.x; y[1] += p.y; y[2] += p.z; y[3] += p.w;
                    }
                    *reinterpret_cast<float4*>(o + c) = make_float4(y[0], y[1], y[2], y[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (c0 + c + i < a.N) o[c + i] = a.accumulate ? o[c + i] + y[i] : y[i];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tm, 2 * BN); }
}

int split_rows(const float* in, int64_t ld, int rows, int K, int pitch, __nv_bfloat16* out, cudaStream_t st) {
    const int vec = ld % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    const int64_t blocks = ((int64_t)rows * (pitch / 8) + 255) / 256;
    launch_pdl(split_rows_kernel, dim3((unsigned)std::min<int64_t>(blocks, 8 * num_sms())), dim3(256), 0, st, in, ld, rows, K, pitch, out, vec);
    B2_LAUNCH_CHECK();
    return 0;
}

template <int BN>
int launch_split_linear(const LinearArgs& a, const __nv_bfloat16* pa, const __nv_bfloat16* pw, int pitch, cudaStream_t st) {
    CUtensorMap ta, tw;
    B2_TRY(make_tmap_parts(&ta, pa, pitch, a.M, 3, LX_M));
    B2_TRY(make_tmap_parts(&tw, pw, pitch, a.N, 3, BN));
    B2_CUDA_CHECK(cudaFuncSetAttribute(linear_split_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, LxCfg<BN>::SMEM));
    launch_pdl(linear_split_kernel<BN>, dim3(((a.M + LX_M - 1) / LX_M) * ((a.N + BN - 1) / BN)), dim3(LX_THREADS), LxCfg<BN>::SMEM, st, ta, tw, a);
    B2_LAUNCH_CHECK();
    return 0;
}

int pitch_of(int K) { return (K + 7) / 8 * 8; }
}  // namespace

size_t linear_split_bytes(int rows, int K) { return (size_t)6 * rows * pitch_of(K); }

bool linear_splits(const LinearArgs& a) {
    return a.w_dtype == DT_F32 && !a.round_a && a.norm.alpha == nullptr && a.parts != nullptr && a.M >= LINEAR_SPLIT_MIN_ROWS &&
           linear_split_bytes(a.M, a.K) + linear_split_bytes(std::min(a.N, 128), a.K) <= a.parts_bytes;
}

int linear_split_f32(const LinearArgs& a, cudaStream_t st) {
    const int pitch = pitch_of(a.K);
    __nv_bfloat16* pa = reinterpret_cast<__nv_bfloat16*>(a.parts);
    __nv_bfloat16* pw = pa + (size_t)3 * a.M * pitch;
    B2_TRY(split_rows(a.A, a.lda, a.M, a.K, pitch, pa, st));
    // as many rows of W at a time as the scratch holds, in whole tiles
    const int64_t fit = (int64_t)((a.parts_bytes - linear_split_bytes(a.M, a.K)) / linear_split_bytes(1, a.K));
    const int step = fit >= a.N ? a.N : (int)(fit / 128 * 128);
    for (int n0 = 0; n0 < a.N; n0 += step) {
        LinearArgs b = a;
        b.N = std::min(step, a.N - n0);
        b.out = a.out + n0;
        if (a.bias != nullptr) b.bias = a.bias + n0;
        b.W = reinterpret_cast<const float*>(a.W) + (size_t)n0 * a.ldw;
        B2_TRY(split_rows(reinterpret_cast<const float*>(b.W), a.ldw, b.N, a.K, pitch, pw, st));
        const int num_m = (b.M + LX_M - 1) / LX_M;
        // tiles of 128 columns read A half as often; narrower ones where they would leave SMs idle
        const bool wide = num_m * ((b.N + 127) / 128) > num_sms() / 2;
        B2_TRY(wide ? launch_split_linear<128>(b, pa, pw, pitch, st) : launch_split_linear<64>(b, pa, pw, pitch, st));
    }
    return 0;
}

}  // namespace b2
