// CTA-pair (cta_group::2) bf16 GEMM for the big-M launches (ViT at B >= 16, LLaMA prefill at B >= 8):
//     C[M,N] = epilogue(A[M,K] · W[N,K]^T)          one 256 x 256 output tile per CTA PAIR
//
// Selected by gemm_bf16's cost model (gemm_tcgen05.cu) wherever its pair tiles fill their waves
// (tests/test_ops_gpu.py::test_gemm_2cta_*), measured in profiles/r2b_gemm_sweep.json.
//
// Why: the 1-CTA kernel (gemm_tcgen05.cu) reads 96 B/clk of operands from shared memory at its best tile (128x256) — every
// CTA stages the whole 256-row B tile — and tops out at 75-90 % of cuBLAS on these shapes (profiles/r1e_gemm_sweep_bn192.json).
// In a CTA pair each CTA stages HALF of the B tile (128 of the 256 W rows) plus its own 128 A rows, and one
// tcgen05.mma.cta_group::2 (M = 256) issued by the leader CTA drives the tensor cores of both SMs against the union of the two
// shared memories: 64 B/clk per SM, and half the L2->SM traffic for B.
//
// Protocol (ranks 0 = leader, 1 = peer; the two CTAs of a cluster land on the two SMs of a TPC):
//   TMA producer (1 thread per CTA)   waits its own empty[s]; the leader arms ITS full[s] with the bytes of BOTH CTAs; both CTAs
//                                     issue cp.async.bulk.tensor...cta_group::2 whose mbarrier operand is the LEADER's full[s]
//   MMA issuer   (1 thread, leader)   waits full[s] and tmem_empty[a]; 4 x tcgen05.mma.cta_group::2.kind::f16 (256x256x16) per
//                                     k-block; tcgen05.commit ... multicast::cluster (mask 0b11) onto empty[s] / tmem_full[a] of
//                                     both CTAs
//   epilogue     (8 warps per CTA)    each CTA drains its own 128 TMEM lanes (its 128 rows of the tile) with the same fused
//                                     epilogues as the 1-CTA kernel, then arrives on the LEADER's tmem_empty[a] (remote arrive
//                                     from the peer)
#include <cuda.h>
#include <math.h>

#include "common.cuh"
#include "kernels.h"
#include "tile_store.cuh"

namespace b2 {

int make_tmap_bf16(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_rows);

namespace {

constexpr int P_BM = 128;            // rows of A / of W staged per CTA
constexpr int P_TM = 2 * P_BM;       // pair tile M
constexpr int P_TN = 2 * P_BM;       // pair tile N
constexpr int P_BK = 64;
constexpr int P_THREADS = 320;       // warp 0: TMA, warp 1: MMA (leader only), warps 2..9: epilogue
constexpr int P_EPI_WARPS = 8;
constexpr int P_TILE_BYTES = P_BM * P_BK * 2;      // 16 KB
constexpr int P_STAGE_BYTES = 2 * P_TILE_BYTES;    // A half + B half per CTA
constexpr int P_STAGES = 6;
constexpr int P_TMEM_COLS = 512;                   // two 256-column accumulator stages
constexpr int P_BOX = 128;                         // bytes of a row of an epilogue warp's box (tile_store.cuh)
constexpr int P_BOX_BYTES = P_EPI_WARPS * 32 * P_BOX;
constexpr int P_SMEM = P_STAGES * P_STAGE_BYTES + P_BOX_BYTES + 1024 + 256;
static_assert(P_SMEM <= 227 * 1024, "shared memory of one CTA");

struct PairEpi {
    const __nv_bfloat16* bias;
    const __nv_bfloat16* residual;
    void* out;
    int ld_out, ld_res, out_fp32;
    int post = 0;          // fp32 output only: LIN_* activation, scale, accumulate onto the output
    float alpha = 1.f;
    int accumulate = 0;
    // ACT_ROPE_QKV
    const uint32_t* rope_tab;
    __nv_bfloat16* kcache;
    __nv_bfloat16* vcache;
    int rope_S, rope_H, rope_Smax;
    GluAct glu;            // ACT_GLU
    int w_early;           // GemmArgs
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of `local_smem_addr` (a shared::cta address of THIS CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_rank(uint32_t local_smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-SM TMA load: destination in this CTA's shared memory, completion bytes on an mbarrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_2sm(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int32_t c0, int32_t c1,
                                                uint64_t cache_hint) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "l"(cache_hint)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_2sm(uint32_t* smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2sm(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_2sm(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive (once all MMAs issued so far have retired) on the barrier at this shared-memory offset in BOTH CTAs of the pair
__device__ __forceinline__ void umma_commit_2sm(uint64_t* bar) {
    const uint16_t mask = 0b11;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "h"(mask)
                 : "memory");
}

__device__ __forceinline__ float p_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
// q*cos + rotate_half(q)*sin with bf16 rounding of each product and of the sum (attention.cu rope_apply: same expression)
__device__ __forceinline__ float p_rope(float x, float partner_signed, float c, float s) {
    return round_bf16(round_bf16(x * c) + round_bf16(partner_signed * s));
}

template <int ACT, bool F32>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(P_THREADS, 1)
gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const __grid_constant__ CUtensorMap tmap_out, int M, int N, int K, PairEpi ep) {
    extern __shared__ uint8_t p_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p_smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* boxes = smem + P_STAGES * P_STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(boxes + P_BOX_BYTES);
    uint64_t* full_bar = bars;                        // [P_STAGES]   used in the leader
    uint64_t* empty_bar = bars + P_STAGES;            // [P_STAGES]   one per CTA
    uint64_t* tmem_full = bars + 2 * P_STAGES;        // [2]          one per CTA
    uint64_t* tmem_empty = bars + 2 * P_STAGES + 2;   // [2]          used in the leader
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * P_STAGES + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;

    const int num_m = (M + P_TM - 1) / P_TM;
    const int num_n = (N + P_TN - 1) / P_TN;
    const int num_tiles = num_m * num_n;
    const int num_kb = (K + P_BK - 1) / P_BK;
    constexpr int GM = 4;  // pair-tile m-blocks per raster group
    auto tile_coords = [&](int t, int& m_blk, int& n_blk) {
        const int per_group = GM * num_n;
        const int group = t / per_group;
        const int first_m = group * GM;
        const int gsize = min(GM, num_m - first_m);
        const int within = t - group * per_group;
        m_blk = first_m + within % gsize;
        n_blk = within / gsize;
    };

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        if constexpr (ACT != ACT_ROPE_QKV && !F32) tma_prefetch_desc(&tmap_out);
        for (int s = 0; s < P_STAGES; ++s) {
            mbar_init(&full_bar[s], 1);    // the leader producer's arrive.expect_tx (+ the TMA bytes of both CTAs)
            mbar_init(&empty_bar[s], 1);   // one multicast tcgen05.commit per use
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&tmem_full[a], 1);                   // one multicast tcgen05.commit
            mbar_init(&tmem_empty[a], 2 * P_EPI_WARPS);    // every epilogue warp of BOTH CTAs
        }
        fence_barrier_init();
    }
    // The allocation below is the pair's: both CTAs must be there, and one may start long before the other (without this barrier prompts of 512 rows at the 7B width,
    // whose pair kernels come in while the last CTAs of tile GEMMs leave, stood still for good within 300 of them; none of 14400 did with it)
    cluster_sync();
    if (warp == 1) tmem_alloc_2sm(tmem_slot, P_TMEM_COLS);  // collective over the pair: one warp in each CTA
    tc_fence_before();
    cluster_sync();  // barriers initialised and TMEM allocated in both CTAs before anyone signals across
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_trigger();   // the set-up above and (w_early) the first weights below overlap the upstream kernel's tail; A / residual are its outputs

    if (warp == 0) {
        if (lane == 0) {
            // ===================== TMA producer (both CTAs) =====================
            // b_row: this CTA's 128 rows of W (half of the N tile; ACT_GLU: 64 of gate, 64 of up)
            auto load_b = [&](uint8_t* sb, uint32_t leader_full, int kb, int b_row) {
                if constexpr (ACT == ACT_GLU) {
                    tma_load_2d_2sm(sb, &tmap_b, leader_full, kb * P_BK, b_row / 2, kEvictNormal);
                    tma_load_2d_2sm(sb + P_TILE_BYTES / 2, &tmap_b, leader_full, kb * P_BK, N / 2 + b_row / 2, kEvictNormal);
                } else {
                    tma_load_2d_2sm(sb, &tmap_b, leader_full, kb * P_BK, b_row, kEvictNormal);
                }
            };
            // the weight halves of the first stages travel in front of the programmatic-dependent-launch wait (unless the kernel in front may be
            // writing W: w_early), A follows behind it
            int pre = 0;
            if (ep.w_early != 0 && pair < num_tiles) {
                int m_blk, n_blk;
                tile_coords(pair, m_blk, n_blk);
                for (; pre < num_kb && pre < P_STAGES; ++pre) {
                    if (leader) mbar_arrive_expect_tx(&full_bar[pre], 2 * P_STAGE_BYTES);
                    load_b(smem + pre * P_STAGE_BYTES + P_TILE_BYTES, mapa_rank(smem_u32(&full_bar[pre]), 0), pre, n_blk * P_TN + (int)rank * P_BM);
                }
            }
            pdl_wait();
            int stage = 0, seen = 0;
            uint32_t phase = 0;
            for (int t = pair; t < num_tiles; t += num_pairs) {
                int m_blk, n_blk;
                tile_coords(t, m_blk, n_blk);
                const int a_row = m_blk * P_TM + (int)rank * P_BM;  // this CTA's 128 rows of A
                for (int kb = 0; kb < num_kb; ++kb, ++seen) {
                    uint8_t* sa = smem + stage * P_STAGE_BYTES;
                    const uint32_t leader_full = mapa_rank(smem_u32(&full_bar[stage]), 0);
                    if (seen >= pre) {
                        mbar_wait(&empty_bar[stage], phase ^ 1);
                        if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * P_STAGE_BYTES);
                        load_b(sa + P_TILE_BYTES, leader_full, kb, n_blk * P_TN + (int)rank * P_BM);
                    }
                    tma_load_2d_2sm(sa, &tmap_a, leader_full, kb * P_BK, a_row, kEvictNormal);
                    if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (leader && lane == 0) {
            // ===================== MMA issuer (leader CTA only) =====================
            constexpr uint32_t idesc = make_idesc_bf16_f32(P_TM, P_TN);
            int stage = 0;
            uint32_t phase = 0;
            int local = 0;
            for (int t = pair; t < num_tiles; t += num_pairs, ++local) {
                const int as = local & 1;
                mbar_wait(&tmem_empty[as], ((local >> 1) & 1) ^ 1);
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + as * P_TN;
                for (int kb = 0; kb < num_kb; ++kb) {
                    mbar_wait(&full_bar[stage], phase);
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + stage * P_STAGE_BYTES);
                    const uint64_t da = make_sw128_kmajor_desc(sa);
                    const uint64_t db = make_sw128_kmajor_desc(sa + P_TILE_BYTES);
#pragma unroll
                    for (int k = 0; k < P_BK / 16; ++k)
                        umma_bf16_2sm(tmem_d, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
                    umma_commit_2sm(&empty_bar[stage]);
                    if (kb == num_kb - 1) umma_commit_2sm(&tmem_full[as]);
                    if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else {
        // ===================== epilogue warps 2..9 (both CTAs: own 128 rows of the pair tile) =====================
        pdl_wait();   // residual / out may be read or written by the upstream kernel
        const int q = warp & 3;
        const int half = (warp - 2) >> 2;
        int local = 0;
        for (int t = pair; t < num_tiles; t += num_pairs, ++local) {
            int m_blk, n_blk;
            tile_coords(t, m_blk, n_blk);
            const int as = local & 1;
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * P_TN + half * 128;
            const int row0 = m_blk * P_TM + (int)rank * P_BM + q * 32;
            uint8_t* buf = boxes + (warp - 2) * 32 * P_BOX;
            auto ready = [&] { mbar_wait(&tmem_full[as], (local >> 1) & 1); tc_fence_after(); };
            auto drained = [&] {   // this warp has read its part of accumulator stage `as`: tell the leader's MMA issuer
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(mapa_rank(smem_u32(&tmem_empty[as]), 0));
            };
            if constexpr (ACT == ACT_SWIGLU || ACT == ACT_GLU) {   // 64 gate columns, then 64 up columns of the same outputs
                const TileBox<P_BOX> box{&tmap_out, buf, lane, row0, M, N / 2};
                store_glu_tile<P_BOX, 64, ACT == ACT_GLU ? 8 : 32>(box, taddr, n_blk * (P_TN / 2) + half * 64, ready, drained, [&](float g, float u) {
                    if constexpr (ACT == ACT_GLU) return glu_act(g, u, ep.glu);
                    else return p_silu(g) * u;
                });
            } else if constexpr (ACT == ACT_ROPE_QKV) {
                // This warp's half of the pair tile is the 128 columns of ONE head of q, k or v (hidden % 256 == 0, head_dim 128).
                // Element i of the head rotates with element i + 64: columns j.. and 64 + j.. are read together, 8 at a time.
                // Rows of q and rows of the caches lie at pitches of their own (and a tile may hold rows of two prompts), so the box leaves by
                // ordinary stores: four lanes on 64 bytes of a row.
                const int row = row0 + lane;
                const int col_base = n_blk * P_TN + half * 128;
                const int hdim = ep.rope_H * 128;
                const int part = col_base / hdim;  // 0 = q, 1 = k, 2 = v
                const int head = (col_base - part * hdim) >> 7;
                const uint4* tab = reinterpret_cast<const uint4*>(ep.rope_tab + (size_t)(row % ep.rope_S) * 64);  // 16 x 16 B: 64 (cos, sin) pairs
                ready();
#pragma unroll 1
                for (int j = 0; j < 8; ++j) {
                    uint32_t lo[8], hi[8];
                    __syncwarp();
                    tmem_ld_cols(taddr + j * 8, lo);
                    tmem_ld_cols(taddr + 64 + j * 8, hi);
                    tmem_ld_wait();
                    if (j == 7) drained();
                    float ol[8], oh[8];
                    uint32_t csw[8];
                    if (part < 2) {
                        const uint4 t0 = __ldg(tab + j * 2), t1 = __ldg(tab + j * 2 + 1);
                        csw[0] = t0.x; csw[1] = t0.y; csw[2] = t0.z; csw[3] = t0.w;
                        csw[4] = t1.x; csw[5] = t1.y; csw[6] = t1.z; csw[7] = t1.w;
                    }
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float xl = round_bf16(__uint_as_float(lo[e]));  // the projection as bf16, like the unfused path
                        const float xh = round_bf16(__uint_as_float(hi[e]));
                        if (part < 2) {
                            const float cs_c = bf16_lo(csw[e]), cs_s = bf16_hi(csw[e]);
                            ol[e] = p_rope(xl, -xh, cs_c, cs_s);
                            oh[e] = p_rope(xh, xl, cs_c, cs_s);
                        } else {
                            ol[e] = xl; oh[e] = xh;
                        }
                    }
                    *box_slot<P_BOX>(buf, lane, j & 3) = make_uint4(pack_bf16(ol[0], ol[1]), pack_bf16(ol[2], ol[3]), pack_bf16(ol[4], ol[5]), pack_bf16(ol[6], ol[7]));
                    *box_slot<P_BOX>(buf, lane, 4 + (j & 3)) = make_uint4(pack_bf16(oh[0], oh[1]), pack_bf16(oh[2], oh[3]), pack_bf16(oh[4], oh[5]), pack_bf16(oh[6], oh[7]));
                    if ((j & 3) != 3) continue;
                    __syncwarp();
                    const int piece = lane & 7, at = (piece < 4 ? 0 : 64) + (j >> 2) * 32 + (piece & 3) * 8;
#pragma unroll 4
                    for (int i = 0; i < 8; ++i) {
                        const int r = i * 4 + (lane >> 3), orow = row0 + r;
                        if (!(orow < M && col_base < N)) continue;
                        __nv_bfloat16* dst;
                        if (part == 0) {
                            dst = reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)orow * ep.ld_out + col_base;
                        } else {
                            const int b = orow / ep.rope_S, t2 = orow - b * ep.rope_S;
                            dst = (part == 1 ? ep.kcache : ep.vcache) + (((size_t)b * ep.rope_H + head) * ep.rope_Smax + t2) * 128;
                        }
                        *reinterpret_cast<uint4*>(dst + at) = *box_slot<P_BOX>(buf, r, piece);
                    }
                }
            } else {
                const TileBox<P_BOX> box{&tmap_out, buf, lane, row0, M, N};
                store_tile<ACT, P_BOX, 128, F32>(box, taddr, n_blk * P_TN + half * 128, ep, ready, drained);
            }
        }
        if (lane == 0) bulk_wait_all();
    }

    tc_fence_before();
    cluster_sync();  // no CTA may free TMEM / exit while its partner can still signal into its shared memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_2sm(tmem_base, P_TMEM_COLS);
    }
}

template <int ACT, bool F32 = false>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, const PairEpi& ep, cudaStream_t stream) {
    static bool attr_set = false;
    auto kern = gemm_bf16_2cta_kernel<ACT, F32>;
    if (!attr_set) {
        B2_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM));
        attr_set = true;
    }
    CUtensorMap to = {};
    if (ACT != ACT_ROPE_QKV && !F32) B2_TRY(make_tmap_out(&to, ep.out, M, ACT == ACT_SWIGLU || ACT == ACT_GLU ? N / 2 : N, ep.ld_out, P_BOX));
    const int tiles = ((M + P_TM - 1) / P_TM) * ((N + P_TN - 1) / P_TN);
    const int max_pairs = num_sms() / 2;
    const int pairs = tiles < max_pairs ? tiles : max_pairs;
    B2_CUDA_CHECK(launch_pdl(kern, dim3(2 * pairs), dim3(P_THREADS), (size_t)P_SMEM, stream, ta, tb, to, M, N, K, ep));  // cluster dims (2,1,1) are a kernel attribute
    B2_LAUNCH_CHECK();
    return 0;
}

}  // namespace

// Same contract as gemm_bf16 (kernels.h). SwiGLU needs N % 128 == 0.
int gemm_bf16_2cta(const GemmArgs& g, cudaStream_t stream) {
    B2_CHECK_ARG(g.M > 0 && g.N > 0 && g.K > 0, "gemm_2cta: empty problem M=%d N=%d K=%d", g.M, g.N, g.K);
    B2_CHECK_ARG(g.K % 8 == 0 && g.N % 8 == 0, "gemm_2cta: K and N must be multiples of 8 (K=%d N=%d)", g.K, g.N);
    B2_CHECK_ARG(g.act != ACT_SWIGLU || (g.N % 128 == 0 && !g.out_fp32 && g.bias == nullptr && g.residual == nullptr),
                 "gemm_2cta: swiglu needs N %% 128 == 0, no bias/residual, bf16 output");
    B2_CHECK_ARG(g.act != ACT_GLU || (g.N % 16 == 0 && !g.out_fp32 && g.bias == nullptr && g.residual == nullptr),
                 "gemm_2cta: glu needs N %% 16 == 0, no bias/residual, bf16 output");
    B2_CHECK_ARG((reinterpret_cast<uintptr_t>(g.out) & 15) == 0 && (g.ld_out % 8) == 0, "gemm_2cta: out alignment");
    B2_CHECK_ARG(g.residual == nullptr || ((reinterpret_cast<uintptr_t>(g.residual) & 15) == 0 && (g.ld_res % 8) == 0),
                 "gemm_2cta: residual alignment");
    CUtensorMap ta, tb;
    B2_TRY(make_tmap_bf16(&ta, g.A, g.M, g.K, g.lda, P_BM));
    B2_TRY(make_tmap_bf16(&tb, g.W, g.N, g.K, g.ldw, g.act == ACT_GLU ? P_BM / 2 : P_BM));
    PairEpi ep;
    ep.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias);
    ep.residual = reinterpret_cast<const __nv_bfloat16*>(g.residual);
    ep.out = g.out; ep.ld_out = g.ld_out; ep.ld_res = g.ld_res; ep.out_fp32 = g.out_fp32;
    ep.post = g.out_fp32 ? g.post : 0; ep.alpha = g.out_fp32 ? g.alpha : 1.f; ep.accumulate = g.out_fp32 ? g.accumulate : 0;
    ep.rope_tab = reinterpret_cast<const uint32_t*>(g.rope.table);
    ep.kcache = reinterpret_cast<__nv_bfloat16*>(g.rope.kcache); ep.vcache = reinterpret_cast<__nv_bfloat16*>(g.rope.vcache);
    ep.rope_S = g.rope.S; ep.rope_H = g.rope.H; ep.rope_Smax = g.rope.Smax;
    ep.glu = g.glu;
    ep.w_early = g.w_early;
    if (g.act == ACT_ROPE_QKV) {
        B2_CHECK_ARG(g.rope.table && g.rope.kcache && g.rope.vcache && g.rope.S > 0 && g.rope.H > 0 && g.rope.Smax >= g.rope.S,
                     "gemm_2cta(rope_qkv): rope arguments missing");
        B2_CHECK_ARG(g.N == 3 * g.rope.H * 128 && (g.rope.H * 128) % 256 == 0 && g.M % g.rope.S == 0 && !g.out_fp32 &&
                         g.bias == nullptr && g.residual == nullptr,
                     "gemm_2cta(rope_qkv): needs N = 3*H*128 with H*128 %% 256 == 0, M = B*S, bf16 output, no bias/residual");
    }
    switch (g.act) {
        case ACT_NONE: return ep.out_fp32 ? launch_pair<ACT_NONE, true>(ta, tb, g.M, g.N, g.K, ep, stream) : launch_pair<ACT_NONE>(ta, tb, g.M, g.N, g.K, ep, stream);
        case ACT_QUICK_GELU: return ep.out_fp32 ? launch_pair<ACT_QUICK_GELU, true>(ta, tb, g.M, g.N, g.K, ep, stream) : launch_pair<ACT_QUICK_GELU>(ta, tb, g.M, g.N, g.K, ep, stream);
        case ACT_GELU_ERF: return ep.out_fp32 ? launch_pair<ACT_GELU_ERF, true>(ta, tb, g.M, g.N, g.K, ep, stream) : launch_pair<ACT_GELU_ERF>(ta, tb, g.M, g.N, g.K, ep, stream);
        case ACT_SWIGLU: return launch_pair<ACT_SWIGLU>(ta, tb, g.M, g.N, g.K, ep, stream);
        case ACT_GLU: return launch_pair<ACT_GLU>(ta, tb, g.M, g.N, g.K, ep, stream);
        case ACT_ROPE_QKV: return launch_pair<ACT_ROPE_QKV>(ta, tb, g.M, g.N, g.K, ep, stream);
        default: break;
    }
    set_error("gemm_2cta: unsupported activation %d", g.act);
    return -1;
}

}  // namespace b2
