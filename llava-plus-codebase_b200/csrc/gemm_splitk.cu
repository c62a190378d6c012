// bf16 GEMM whose K is cut over the CTAs of a cluster: C[M,N] = epilogue(A[M,K] · W[N,K]^T) for shapes whose output tiles do not fill the SMs
// (short prompts, one to four pictures). The plain kernel (gemm_tcgen05.cu) then walks a long K on a few SMs, bound by what ONE SM can take
// out of L2; here S = 2 to 4 CTAs of a cluster take a slice of K each, with the same TMA ring and tcgen05 products, and their partial tiles meet
// in distributed shared memory: every CTA puts its accumulator into its drained ring, the cluster synchronises, and CTA r adds up its 1/S of
// the columns from all S rings in rank order (deterministic, fp32) and runs the epilogue for them. No workspace, no second launch.
// M = 64, N = 2048, K = 5120: 23.0 us on 32 SMs -> 11.4 us on 128; N = 4096, K = 11008: 46.4 -> 21.6 us.
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace b2 {

int make_tmap_bf16(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows);

namespace {

constexpr int KS_BM = 128, KS_BK = 64, KS_THREADS = 320, KS_A = KS_BM * KS_BK * 2;

template <int BN>
struct KsCfg {
    static constexpr int STAGE = KS_A + BN * KS_BK * 2, STAGES = BN == 256 ? 4 : BN == 128 ? 6 : 8, SMEM = STAGES * STAGE + 1024 + 256;
    static_assert(KS_BM * BN * 4 <= STAGES * STAGE, "the partial tile lies in the drained ring");
};

struct KsEpi {
    const __nv_bfloat16 *bias, *residual;
    void* out;
    int ld_out, ld_res, out_fp32, post, accumulate;
    float alpha;
    int a_bytes;           // of A per k-block: gemm_a_rows(M) rows
    int w_early;           // GemmArgs
};

__device__ __forceinline__ uint32_t ks_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ float4 ks_ld_remote(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}

template <int BN, int ACT>
__global__ void __launch_bounds__(KS_THREADS, 1) gemm_splitk_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                                                                    int M, int N, int K, int S, KsEpi ep) {
    using Cfg = KsCfg<BN>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t ks_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ks_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE);
    uint64_t *full = bars, *empty = bars + STAGES, *done = bars + 2 * STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)ks_rank(), tile = blockIdx.x / S, num_m = (M + KS_BM - 1) / KS_BM;
    const int m0 = (tile % num_m) * KS_BM, n0 = (tile / num_m) * BN;
    const int num_kb = (K + KS_BK - 1) / KS_BK, kb0 = num_kb * rank / S, kb1 = num_kb * (rank + 1) / S;   // at least one: S <= num_kb

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(done, 1);
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, BN); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_trigger();
    if (warp == 0) {
        if (lane == 0) {
            // the weight halves of the first stages travel in front of the programmatic-dependent-launch wait (unless the kernel in front may be
            // writing W: w_early), A follows behind it
            const int pre = ep.w_early == 0 ? 0 : kb1 - kb0 < STAGES ? kb1 - kb0 : STAGES;
            for (int i = 0; i < pre; ++i) {
                mbar_arrive_expect_tx(&full[i], ep.a_bytes + BN * KS_BK * 2);
                tma_load_2d(smem + i * Cfg::STAGE + KS_A, &tmap_b, &full[i], (kb0 + i) * KS_BK, n0, kEvictNormal);
            }
            pdl_wait();
            int stage = 0;
            uint32_t phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                uint8_t* sa = smem + stage * Cfg::STAGE;
                if (kb - kb0 >= pre) {
                    mbar_wait(&empty[stage], phase ^ 1);
                    mbar_arrive_expect_tx(&full[stage], ep.a_bytes + BN * KS_BK * 2);
                    tma_load_2d(sa + KS_A, &tmap_b, &full[stage], kb * KS_BK, n0, kEvictNormal);
                }
                tma_load_2d(sa, &tmap_a, &full[stage], kb * KS_BK, m0, kEvictNormal);
                if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        constexpr uint32_t idesc = make_idesc_bf16_f32(KS_BM, BN);
        int stage = 0;
        uint32_t phase = 0, ready = 0;
        for (int kb = kb0; kb < kb1; ++kb) {
            if (!ready) mbar_wait(&full[stage], phase);
            const int next = stage + 1 == STAGES ? 0 : stage + 1;
            const uint32_t next_phase = next == 0 ? phase ^ 1 : phase;
            ready = __all_sync(0xffffffffu, kb + 1 < kb1 ? mbar_try_wait(&full[next], next_phase) : 0u);
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE);
            const uint64_t da = make_sw128_kmajor_desc(sa), db = make_sw128_kmajor_desc(sa + KS_A);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < KS_BK / 16; ++k) umma_bf16(tmem, da + 2 * k, db + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
                umma_commit(&empty[stage]);
                if (kb == kb1 - 1) umma_commit(done);
            }
            __syncwarp();
            stage = next;
            phase = next_phase;
        }
    } else {
        // the accumulator into the drained ring (every load has landed and every product has read it when `done` completes): [4 columns][128 rows]
        const int q = warp & 3, half = (warp - 2) >> 2, row = q * 32 + lane;
        mbar_wait(done, 0);
        tc_fence_after();
        float4* part = reinterpret_cast<float4*>(smem);
#pragma unroll 1
        for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
            uint32_t v[32];
            __syncwarp();
            tmem_ld_32x32(tmem + (static_cast<uint32_t>(q * 32) << 16) + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                part[(c * 8 + i) * KS_BM + row] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
        }
        tc_fence_before();
    }
    cluster_sync();
    if (warp >= 2) {
        pdl_wait();   // residual and output may be written by the kernels in front
        const int t = threadIdx.x - 64, row = t & 127, g1 = BN / 8 * (rank + 1) / S;   // 8-column groups of this CTA's share
        const uint32_t base = smem_u32(smem);
        for (int c8 = BN / 8 * rank / S + (t >> 7); c8 < g1 && m0 + row < M; c8 += 2) {   // group of 8 columns inside the tile
            float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s < S; ++s) {
                const float4 u = ks_ld_remote(base + (uint32_t)((2 * c8) * KS_BM + row) * 16, s), w = ks_ld_remote(base + (uint32_t)((2 * c8 + 1) * KS_BM + row) * 16, s);
                x[0] += u.x; x[1] += u.y; x[2] += u.z; x[3] += u.w; x[4] += w.x; x[5] += w.y; x[6] += w.z; x[7] += w.w;
            }
            const int m = m0 + row, n = n0 + c8 * 8;
            if (n >= N) continue;
            if (ep.bias != nullptr) {
                const uint4 b = *reinterpret_cast<const uint4*>(ep.bias + n);
                x[0] += bf16_lo(b.x); x[1] += bf16_hi(b.x); x[2] += bf16_lo(b.y); x[3] += bf16_hi(b.y);
                x[4] += bf16_lo(b.z); x[5] += bf16_hi(b.z); x[6] += bf16_lo(b.w); x[7] += bf16_hi(b.w);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                if (ACT == ACT_QUICK_GELU) x[e] = __fdividef(x[e], 1.0f + __expf(-1.702f * x[e]));
                if (ACT == ACT_GELU_ERF) x[e] = 0.5f * x[e] * (1.0f + erff(x[e] * 0.70710678118654752440f));
            }
            if (ep.residual != nullptr) {
                const uint4 r = *reinterpret_cast<const uint4*>(ep.residual + (size_t)m * ep.ld_res + n);
                x[0] += bf16_lo(r.x); x[1] += bf16_hi(r.x); x[2] += bf16_lo(r.y); x[3] += bf16_hi(r.y);
                x[4] += bf16_lo(r.z); x[5] += bf16_hi(r.z); x[6] += bf16_lo(r.w); x[7] += bf16_hi(r.w);
            }
            if (ep.out_fp32) {
                float* op = reinterpret_cast<float*>(ep.out) + (size_t)m * ep.ld_out + n;
                if (ep.post != 0 || ep.accumulate != 0 || ep.alpha != 1.f) epi_post8(x, op, ep.post, ep.alpha, ep.accumulate);
                *reinterpret_cast<float4*>(op) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(op + 4) = make_float4(x[4], x[5], x[6], x[7]);
            } else {
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)m * ep.ld_out + n) =
                    make_uint4(pack_bf16(x[0], x[1]), pack_bf16(x[2], x[3]), pack_bf16(x[4], x[5]), pack_bf16(x[6], x[7]));
            }
        }
    }
    cluster_sync();   // no ring goes away while another CTA reads it
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, BN); }
}

template <int BN, int ACT>
int launch_splitk(const GemmArgs& g, int S, const KsEpi& ep, cudaStream_t st) {
    CUtensorMap ta, tb;
    B2_TRY(make_tmap_bf16(&ta, g.A, g.M, g.K, g.lda, gemm_a_rows(g.M)));
    B2_TRY(make_tmap_bf16(&tb, g.W, g.N, g.K, g.ldw, BN));
    auto kernel = gemm_splitk_kernel<BN, ACT>;
    B2_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KsCfg<BN>::SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S * ((g.M + KS_BM - 1) / KS_BM) * ((g.N + BN - 1) / BN)); cfg.blockDim = dim3(KS_THREADS); cfg.dynamicSmemBytes = KsCfg<BN>::SMEM; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    cfg.attrs = attr; cfg.numAttrs = 2;
    B2_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, ta, tb, g.M, g.N, g.K, S, ep));
    B2_LAUNCH_CHECK();
    return 0;
}
template <int BN>
int splitk_act(const GemmArgs& g, int S, const KsEpi& ep, cudaStream_t st) {
    if (g.act == ACT_QUICK_GELU) return launch_splitk<BN, ACT_QUICK_GELU>(g, S, ep, st);
    if (g.act == ACT_GELU_ERF) return launch_splitk<BN, ACT_GELU_ERF>(g, S, ep, st);
    return launch_splitk<BN, ACT_NONE>(g, S, ep, st);
}
}  // namespace

int gemm_bf16_splitk(const GemmArgs& g, int bn, int S, cudaStream_t st) {
    B2_CHECK_ARG((bn == 64 || bn == 128 || bn == 256) && S >= 2 && S <= 4 && S <= (g.K + KS_BK - 1) / KS_BK && g.tile_group == nullptr, "gemm(split K): bad plan bn=%d S=%d K=%d", bn, S, g.K);
    // (a gated unit's output has half the product's columns: without its epilogue here, the plain one would write past every row)
    B2_CHECK_ARG(g.act == ACT_NONE || g.act == ACT_QUICK_GELU || g.act == ACT_GELU_ERF, "gemm(split K): activation %d has no epilogue here", g.act);
    KsEpi ep;
    ep.a_bytes = gemm_a_rows(g.M) * KS_BK * 2;
    ep.w_early = g.w_early;
    ep.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias); ep.residual = reinterpret_cast<const __nv_bfloat16*>(g.residual);
    ep.out = g.out; ep.ld_out = g.ld_out; ep.ld_res = g.ld_res; ep.out_fp32 = g.out_fp32;
    ep.post = g.out_fp32 ? g.post : 0; ep.alpha = g.out_fp32 ? g.alpha : 1.f; ep.accumulate = g.out_fp32 ? g.accumulate : 0;
    return bn == 64 ? splitk_act<64>(g, S, ep, st) : bn == 128 ? splitk_act<128>(g, S, ep, st) : splitk_act<256>(g, S, ep, st);
}

}  // namespace b2
