// Linears in true fp32 for portions of a prompt, on the tensor cores: out[M, N] = alpha act(A[M, K] W[N, K]^T + bias) (+ out), all fp32, with both
// operands as bf16 parts (split.cuh): A in three, W in three and six products of each pair, or, where every value of W is a bf16 one (the weights of a
// bf16 checkpoint, looked at when the model is finalized), W as it is and the three products that are not zero: the same sums. The tensor core cuts
// its fp32 sums off after every step of 16, so an accumulator spans one block of 64 of K only; the blocks are added up in fp32 registers.
//   1. split_rows_kernel writes the parts of A, and of a W of three parts, per call: a W whose parts exceed the scratch goes in blocks of rows;
//   2. linear_split_kernel: one tile of 128 x BN per CTA, or per cluster whose CTAs share out K; warp 0 TMA producer (a stage: the parts of 64 columns of
//      A and W), warp 1 MMA issuer, warps 2..9 take every block's accumulator out of TMEM (four of them, two at BN = 256). The sums pass through
//      shared memory, the cluster's meet there, and leave in whole rows.
// What bounds it: the stream of parts into the SM, some 40 B a clock (64 KB a block at BN = 128 with W in one part, 768 clk of products). Splitting A
// inside the kernel (32 KB a block) was slower: 8 warps convert a block of 128 x 64 in 1300 clk (600 x 1024 x 4096: 60 us, the parts by TMA 41, K over
// a cluster 24).
// 600 rows, 13 products of a state-space + RWKV pair of width 1024 (33 GFLOP): 2512 us on linear_tiled_kernel -> 413 us and 86 us of cutting on tiles of
// 64 and 128 columns, six products and one CTA a tile; the whole call 764 -> 576 us with W in one part, tiles of up to 256 columns and clusters. The pair's
// error against 64 bits: 1.4e-6, 3.6e-7 on the tensor cores.
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "kernels.h"
#include "split.cuh"

namespace b2 {

int make_tmap_parts(CUtensorMap* map, const void* ptr, int pitch, int64_t rows, int planes, int box_rows);

namespace {

constexpr int LX_M = 128, LX_K = 64, LX_THREADS = 320, LX_MAX_CLUSTER = 8;

// WP: parts of W (3, or 1: W holds bf16 values)
template <int BN, int WP>
struct LxCfg {
    static constexpr int A_BYTES = 3 * LX_M * 128, B_BYTES = WP * BN * 128, STAGE = A_BYTES + B_BYTES, STAGES = STAGE > 72 * 1024 ? 2 : STAGE > 56 * 1024 ? 3 : 4;
    static constexpr int ACCS = BN == 256 ? 2 : 4;                     // accumulators in TMEM
    static constexpr int PITCH = BN + 4;                               // floats between rows of the tile of sums, which takes the ring's place
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static_assert(LX_M * PITCH * 4 <= STAGES * STAGE, "the sums fit into the ring");
};

// rows of fp32 -> [part][rows][pitch] bf16, entries past K zero
__global__ void __launch_bounds__(256) split_rows_kernel(const float* in, int64_t ld, int rows, int K, int pitch, __nv_bfloat16* __restrict__ out, int vec) {
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

__device__ __forceinline__ float4 lx_ld_remote4(const float* p, int rank) {
    uint32_t at;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// grid: tiles x S, clusters of S CTAs that share out the blocks of K, `per` each
template <int BN, int WP>
__global__ void __launch_bounds__(LX_THREADS, 1) linear_split_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, LinearArgs a, int S, int per) {
    using Cfg = LxCfg<BN, WP>;
    constexpr int CH = BN / 2;   // columns per epilogue thread
    extern __shared__ uint8_t lx_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lx_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE);
    uint64_t *full = bars, *empty = bars + Cfg::STAGES, *acc_full = bars + 2 * Cfg::STAGES, *acc_empty = acc_full + Cfg::ACCS;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + Cfg::ACCS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)blockIdx.x % S, tile = (int)blockIdx.x / S;
    const int num_m = (a.M + LX_M - 1) / LX_M, m0 = tile % num_m * LX_M, n0 = tile / num_m * BN;
    const int k_blocks = (a.K + LX_K - 1) / LX_K, b0 = rank * per, blocks = min(per, k_blocks - b0);

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_a);
        tma_prefetch_desc(&tm_w);
        for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int i = 0; i < Cfg::ACCS; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, Cfg::ACCS * BN); tmem_relinquish(); }
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
                for (int p = 0; p < 3; ++p) tma_load_3d(d + p * LX_M * 128, &tm_a, &full[stage], (b0 + b) * LX_K, m0, p);
                for (int p = 0; p < WP; ++p) tma_load_3d(d + Cfg::A_BYTES + p * BN * 128, &tm_w, &full[stage], (b0 + b) * LX_K, n0, p);
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
            const int ac = b % Cfg::ACCS;
            mbar_wait(&acc_empty[ac], ((b / Cfg::ACCS) & 1) ^ 1);
            mbar_wait(&full[stage], phase);
            tc_fence_after();
            const uint32_t s = smem_u32(smem + stage * Cfg::STAGE);
            const uint64_t da = make_sw128_kmajor_desc(s), db = make_sw128_kmajor_desc(s + Cfg::A_BYTES);
            if (leader) {
#pragma unroll
                for (int i = 0; i < (WP == 1 ? 3 : 6); ++i) {   // (W's one part: lo, mid, hi of A in turn)
                    const uint32_t pa = WP == 1 ? 2 - i : (SPLIT_A >> (2 * i)) & 3u, pb = WP == 1 ? 0 : (SPLIT_B >> (2 * i)) & 3u;
#pragma unroll
                    for (int k = 0; k < LX_K / 16; ++k)
                        umma_bf16(tm + ac * BN, da + (pa * (LX_M * 8) + 2 * k), db + (pb * (BN * 8) + 2 * k), idesc, (i | k) != 0 ? 1u : 0u);
                }
                umma_commit(&empty[stage]);
                umma_commit(&acc_full[ac]);
            }
            __syncwarp();
            if (++stage == Cfg::STAGES) { stage = 0; phase ^= 1; }
        }
    } else {
        const int q = warp & 3, half = (warp - 2) >> 2;
        float acc[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) acc[i] = 0.f;
        for (int b = 0; b < blocks; ++b) {
            const int ac = b % Cfg::ACCS;
            mbar_wait(&acc_full[ac], (b / Cfg::ACCS) & 1);
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < CH / 32; ++c) {
                uint32_t v[32];
                __syncwarp();
                tmem_ld_32x32(tm + (static_cast<uint32_t>(q * 32) << 16) + ac * BN + half * CH + c * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[c * 32 + i] += __uint_as_float(v[i]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[ac]);
        }
        // (the last products are done, so nothing reads the ring any more and no copy is on its way)
        float* row = reinterpret_cast<float*>(smem) + (q * 32 + lane) * Cfg::PITCH + half * CH;
#pragma unroll
        for (int i = 0; i < CH; i += 4) *reinterpret_cast<float4*>(row + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    }
    tc_fence_before();
    if (S > 1) cluster_sync();
    else __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tm, Cfg::ACCS * BN); }
    // The sums of the cluster, in the order of K, leave in whole rows: rows rank, rank + S, ... are this CTA's
    const bool vec = a.ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0;
    const float* sums = reinterpret_cast<const float*>(smem);
    for (int e = threadIdx.x; e < (LX_M - rank + S - 1) / S * (BN / 4); e += LX_THREADS) {
        const int r = rank + e / (BN / 4) * S, c = e % (BN / 4) * 4, m = m0 + r, n = n0 + c;
        if (m >= a.M || n >= a.N) continue;
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (S == 1) {
            f = *reinterpret_cast<const float4*>(sums + r * Cfg::PITCH + c);
        } else {
            for (int s = 0; s < S; ++s) {
                const float4 g = lx_ld_remote4(sums + r * Cfg::PITCH + c, s);
                f.x += g.x; f.y += g.y; f.z += g.z; f.w += g.w;
            }
        }
        float* o = a.out + (size_t)m * a.ld_out + n;
        float y[4] = {f.x, f.y, f.z, f.w};
        if (f.x != f.x || f.y != f.y || f.z != f.z || f.w != f.w) {
            lx_plain(a.A + (size_t)m * a.lda, reinterpret_cast<const float*>(a.W), a.ldw, a.K, a.out + (size_t)m * a.ld_out, a.bias, n, min(n + 4, a.N), a.act, a.alpha, a.accumulate);
            continue;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            y[i] += a.bias != nullptr && n + i < a.N ? a.bias[n + i] : 0.f;
            if (a.act != 0) y[i] = lx_act(y[i], a.act);
            y[i] *= a.alpha;
        }
        if (vec && n + 4 <= a.N) {
            if (a.accumulate) {
                const float4 p = *reinterpret_cast<const float4*>(o);
                y[0] += p.x; y[1] += p.y; y[2] += p.z; y[3] += p.w;
            }
            *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n + i < a.N) o[i] = a.accumulate ? o[i] + y[i] : y[i];
        }
    }
    if (S > 1) cluster_sync();   // no tile goes away while another CTA reads it
}

int split_rows(const float* in, int64_t ld, int rows, int K, int pitch, __nv_bfloat16* out, cudaStream_t st) {
    const int vec = ld % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0;
    const int64_t blocks = ((int64_t)rows * (pitch / 8) + 255) / 256;
    launch_pdl(split_rows_kernel, dim3((unsigned)std::min<int64_t>(blocks, 8 * num_sms())), dim3(256), 0, st, in, ld, rows, K, pitch, out, vec);
    B2_LAUNCH_CHECK();
    return 0;
}

template <int BN, int WP>
int launch_split_linear(const LinearArgs& a, const __nv_bfloat16* pa, const __nv_bfloat16* w, int pitch, int pitch_w, int S, cudaStream_t st) {
    CUtensorMap ta, tw;
    B2_TRY(make_tmap_parts(&ta, pa, pitch, a.M, 3, LX_M));
    B2_TRY(make_tmap_parts(&tw, w, pitch_w, a.N, WP, BN));
    B2_CUDA_CHECK(cudaFuncSetAttribute(linear_split_kernel<BN, WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, LxCfg<BN, WP>::SMEM));
    const int blocks = (a.K + LX_K - 1) / LX_K, per = (blocks + S - 1) / S;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(((a.M + LX_M - 1) / LX_M) * ((a.N + BN - 1) / BN) * S); cfg.blockDim = dim3(LX_THREADS); cfg.dynamicSmemBytes = LxCfg<BN, WP>::SMEM; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = S; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = S > 1 ? 2 : 1;
    B2_CUDA_CHECK(cudaLaunchKernelEx(&cfg, linear_split_kernel<BN, WP>, ta, tw, a, S, per));
    B2_LAUNCH_CHECK();
    return 0;
}
// Clusters of S CTAs, one CTA an SM, that the device holds at once: what its GPCs' sizes leave
int clusters_held(int S) {
    static std::atomic<int> held[16][LX_MAX_CLUSTER + 1];
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 16) return std::max(1, num_sms() / (2 * S));
    n = held[dev][S].load(std::memory_order_relaxed);
    if (n > 0) return n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S); cfg.blockDim = dim3(LX_THREADS); cfg.dynamicSmemBytes = LxCfg<128, 1>::SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = S; attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(linear_split_kernel<128, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, LxCfg<128, 1>::SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, linear_split_kernel<128, 1>, &cfg) != cudaSuccess || n < 1) {
        cudaGetLastError();
        n = std::max(1, num_sms() / (2 * S));
    }
    held[dev][S].store(n, std::memory_order_relaxed);
    return n;
}

// Tiles of 64, 128 or (W in one part) 256 columns, K in one piece or shared out over a cluster of up to 8 CTAs: whichever is done first. Clocks of a CTA: a
// block of K is bound by its bytes, some 40 a clock (56 KB at 64 columns with W in one part: 1216 measured, 64 KB at 128: 1500, 80 KB at 256: 2025) or by
// its products (48, 64, 128 clk each); what a tile costs beside them grows with its columns, a cluster adds its barriers and the reads of its tiles. Wide
// tiles read A less often, a cut K fills the SMs. us with the parts of A made, rows x outputs x K, W in one part, 64 columns uncut / the rule's / the best
// of all 24 forms: 600 x 1024 x 1024 15.2 / 14.1 / 14.1; x 4096 41.0 / 23.8 / 23.8; 600 x 4096 x 1024 38.0 / 27.1 / 27.1; 600 x 6176 x 1024 50.2 / 27.9 /
// 27.9; 600 x 64 x 1024 14.5 / 8.3 / 8.3; 64 x 1024 x 1024 13.5 / 7.9 / 7.9; 300 x 1536 x 1536 18.8 / 14.9 / 14.7; 1200 x 2048 x 2048 64.4 / 41.3 / 41.3;
// 40 x 4096 x 1024 13.2 / 9.8 / 9.0. W in three parts: 600 x 1024 x 4096 66.5 / 39.9 / 39.9.
template <int WP>
int launch_tiles(const LinearArgs& a, const __nv_bfloat16* pa, const __nv_bfloat16* w, int pitch, int pitch_w, cudaStream_t st) {
    const int num_m = (a.M + LX_M - 1) / LX_M, blocks = (a.K + LX_K - 1) / LX_K;
    int best_bn = 64, best_s = 1;
    int64_t best = INT64_MAX;
    for (int bn = 64; bn <= (WP == 1 ? 256 : 128); bn *= 2) {
        const int tiles = num_m * ((a.N + bn - 1) / bn);
        const int block = std::max((WP == 1 ? 12 : 24) * std::max(48, bn / 2), (3 * LX_M + WP * bn) * 128 / 40);
        for (int S = 1; S <= LX_MAX_CLUSTER && S <= blocks; ++S) {
            const int per = (blocks + S - 1) / S, held = S == 1 ? num_sms() : clusters_held(S);
            if ((S - 1) * per >= blocks) continue;   // (a CTA without blocks)
            const int64_t clk = (int64_t)((tiles + held - 1) / held) * ((int64_t)per * block + 2500 + 36 * bn + (S > 1 ? 1500 + 30 * std::min(bn, 128) + 300 * S : 0));
            if (clk < best) { best = clk; best_bn = bn; best_s = S; }
        }
    }
    if (WP == 1 && best_bn == 256) return launch_split_linear<WP == 1 ? 256 : 128, WP>(a, pa, w, pitch, pitch_w, best_s, st);
    return best_bn == 128 ? launch_split_linear<128, WP>(a, pa, w, pitch, pitch_w, best_s, st) : launch_split_linear<64, WP>(a, pa, w, pitch, pitch_w, best_s, st);
}

int pitch_of(int K) { return (K + 7) / 8 * 8; }

__global__ void __launch_bounds__(256) bf16_values_kernel(const Fp32Matrix* __restrict__ list, int* __restrict__ other) {
    const Fp32Matrix m = list[blockIdx.y];
    int bad = 0;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < m.fours; i += (int64_t)gridDim.x * 256) {
        const uint4 v = m.w[i];
        bad |= ((v.x | v.y | v.z | v.w) & 0xffffu) != 0;
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) other[blockIdx.y] = 1;
}
__global__ void __launch_bounds__(256) high_halves_kernel(const Fp32Matrix* __restrict__ list) {
    const Fp32Matrix m = list[blockIdx.y];
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < m.fours; i += (int64_t)gridDim.x * 256) {
        const uint4 v = m.w[i];
        m.out[i] = make_uint2(v.x >> 16 | (v.y & 0xffff0000u), v.z >> 16 | (v.w & 0xffff0000u));
    }
}
}  // namespace

size_t linear_split_bytes(int rows, int K) { return (size_t)6 * rows * pitch_of(K); }

bool linear_splits(const LinearArgs& a) {
    return a.w_dtype == DT_F32 && !a.round_a && a.norm.alpha == nullptr && a.parts != nullptr && a.M >= LINEAR_SPLIT_MIN_ROWS &&
           linear_split_bytes(a.M, a.K) + (a.W16 != nullptr ? 0 : linear_split_bytes(std::min(a.N, 128), a.K)) <= a.parts_bytes;
}

int linear_split_f32(const LinearArgs& a, cudaStream_t st) {
    const int pitch = pitch_of(a.K);
    __nv_bfloat16* pa = reinterpret_cast<__nv_bfloat16*>(a.parts);
    __nv_bfloat16* pw = pa + (size_t)3 * a.M * pitch;
    B2_TRY(split_rows(a.A, a.lda, a.M, a.K, pitch, pa, st));
    if (a.W16 != nullptr) return launch_tiles<1>(a, pa, reinterpret_cast<const __nv_bfloat16*>(a.W16), pitch, a.K, st);
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
        B2_TRY(launch_tiles<3>(b, pa, pw, pitch, pitch, st));
    }
    return 0;
}

int bf16_values(const Fp32Matrix* list, int n, int* other, cudaStream_t st) {
    B2_CHECK_ARG(list && other && n >= 1 && n <= 65535, "bf16_values: 1..65535 matrices");
    bf16_values_kernel<<<dim3(2 * num_sms(), n), 256, 0, st>>>(list, other);
    B2_LAUNCH_CHECK();
    return 0;
}
int high_halves(const Fp32Matrix* list, int n, cudaStream_t st) {
    B2_CHECK_ARG(list && n >= 1 && n <= 65535, "high_halves: 1..65535 matrices");
    high_halves_kernel<<<dim3(2 * num_sms(), n), 256, 0, st>>>(list);
    B2_LAUNCH_CHECK();
    return 0;
}

}  // namespace b2
