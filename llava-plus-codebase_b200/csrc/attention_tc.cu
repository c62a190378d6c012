// tcgen05 flash attention for prefill / ViT (sm_100a): S = Q·K^T and O += P·V on the 5th-gen tensor cores with
// TMEM accumulators, TMA-fed operands, fp32 online softmax by one thread per query row.
//
// Replaces the eager attention of the reference's HF path, which materialises the [B,H,S,S] score matrix
// (transformers modeling_llama.py:199-221 eager_attention_forward; modeling_clip.py:261-279).
//
// CTA = one (batch, head, 128-query tile), 192 threads, TWO CTAs per SM (256 TMEM columns each; two groups of softmax warps: 320, one, 512):
//   warp 0 / lane 0 : TMA producer — Q once, then K_t / V_t tiles of 64 keys into rings (4-D tensor maps over the strided [b, t, h, d]
//                     views: the same kernel reads the fused qkv activation buffer of the ViT and the [B, H, Smax, 128] KV cache
//                     of the decoder)
//   warp 1          : MMA issuer — S_t = Q K_t^T  (UMMA 128x64xD, both operands K-major, SWIZZLE_128B), into one of two TMEM buffers
//                                  O += P_t V_t (UMMA 128xDx64; P from TMEM, V straight from its [keys, d] tile as an MN-major operand)
//   warps 2..5 (..9): softmax — thread r owns query row r: tcgen05.ld the S row, scale/mask, running max / sum, P = exp2(s - m) as bf16
//                     back into TMEM over the score row it came from; O in TMEM is rescaled only when a row's max grew by more
//                     than 2^8 (lazy rescale: P and l keep using the stale max, which cancels in O / l), finally O / l -> global.
// S_(t+1) is there before softmax t ends, and S_(t+2) is issued when O_t has read P_t out of its buffer: the softmax warps never wait for a
// product of their own tile. They are what bounds the kernel (at d = 64 the special-function unit alone needs 1024 clk for 128 x 128 exponentials,
// the products 640). Before: tiles of 128 keys, one score buffer, P through shared memory, every tile a chain of product, softmax and product.
// A CTA alone on its SM is bound by the latency of a tile (1310 clk of which the exponentials' unit needs 512), so there two groups of four softmax warps
// take the tiles in turn, each with buffers, an O, a maximum and a sum of its own, which meet in the epilogue (launch rule at the end).
// Measured, before -> now: [B, S, H, d] = [1, 577, 16, 64] 18.4 -> 11.9 -> 8.9 us (two groups), [32, 577, 16, 64] 214 -> 104 us (204 -> 419 TFLOP/s),
// causal [1, 704, 32, 128] 32.9 -> 15.0 us, [4, 2048, 32, 128] 441 -> 172 us (797 TFLOP/s of the 0.5 S^2 that is visible).
#include <cuda.h>
#include <math.h>
#include <stdlib.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace b2 {
namespace {

constexpr int TC_BM = 128;  // queries per CTA
constexpr int TC_BN = 64;   // keys per tile

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]),
        "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]),
        "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// MUFU.EX2 without exp2f's denormal-range fix-up (inputs here are <= 8, results feed a bf16 / an fp32 sum)
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// smem descriptor for an MN-major bf16 operand tile stored as rows of 128 bytes (64 elements along MN) indexed by k,
// SWIZZLE_128B: atoms of 8 k-rows x 128 B; SBO = 1024 B between k-atoms, LBO = bytes between 64-wide MN slabs.
__device__ __forceinline__ uint64_t make_sw128_mnmajor_desc(uint32_t smem_addr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr >> 4) & 0x3FFF);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
// kind::f16 instruction descriptor: A K-major, B K-major (b_mn = 0) or MN-major (b_mn = 1); bf16 x bf16 -> fp32
__host__ __device__ constexpr uint32_t make_idesc(uint32_t m, uint32_t n, uint32_t b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// D (+)= A B with A [128 x 16] in TMEM (two bf16 of a row per column) and B by descriptor
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

struct FlashTcParams {
    const int32_t* seq_lens;
    __nv_bfloat16* o;
    int64_t o_bs, o_ts, o_hs;
    int S;
    float scale_log2;
};

template <int D, int WGS>
struct TcCfg {
    static constexpr int Q_BYTES = TC_BM * D * 2, TILE = TC_BN * D * 2, STAGES = WGS == 2 ? 4 : D == 64 ? 3 : 2;   // of K and of V each
    static constexpr int SMEM = Q_BYTES + 2 * STAGES * TILE + 1024 /*align*/ + 256 /*barriers*/ + (WGS == 2 ? 2 * TC_BM * 8 : 0) /*maxima and sums of both groups*/;
};

template <int D, bool CAUSAL, int WGS>
__global__ void __launch_bounds__(64 + 128 * WGS, 3 - WGS)
flash_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, FlashTcParams p) {
    using Cfg = TcCfg<D, WGS>;
    constexpr int SLABS = D / 64, STAGES = Cfg::STAGES;   // 64-wide (128 B) slabs of the head dim
    constexpr int Q_SLAB = TC_BM * 128, KV_SLAB = TC_BN * 128;
    constexpr int NBUF = 2 * WGS, TMEM_COLS = 256 * WGS, TM_O = NBUF * TC_BN;   // S_t / P_t: columns [64 (t % NBUF), + 64), then O of each group of warps

    extern __shared__ uint8_t tc_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + Cfg::Q_BYTES;
    uint8_t* sV = sK + STAGES * Cfg::TILE;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + STAGES * Cfg::TILE);
    uint64_t *q_full = bars, *s_full = bars + 1, *p_full = s_full + NBUF, *o_done = p_full + NBUF /*[WGS]*/, *o_last = o_done + WGS;
    uint64_t *k_full = o_last + WGS, *k_empty = k_full + STAGES, *v_full = k_empty + STAGES, *v_empty = v_full + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(v_empty + STAGES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // causal: the query tiles with the most keys go first
    const int q0 = (CAUSAL ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z) * TC_BM;
    const int head = blockIdx.x, b = blockIdx.y;
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        mbar_init(q_full, 1);
        for (int s = 0; s < NBUF; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 4);  // one arrive per softmax warp of the group; one a buffer, as P_(t+1) may be announced before anyone waited for P_t
        }
        for (int w = 0; w < WGS; ++w) {
            mbar_init(&o_done[w], 1);
            mbar_init(&o_last[w], 1);
        }
        for (int s = 0; s < 4 * STAGES; ++s) mbar_init(&k_full[s], 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *tmem_slot;
    pdl_trigger();  // (behind the allocation: see tmem_alloc)
    pdl_wait();  // q/k/v (and seq_lens) are outputs of upstream kernels (programmatic dependent launch)
    const int len = p.seq_lens != nullptr ? p.seq_lens[b] : p.S;
    const int kv_end = CAUSAL ? min(len, q0 + TC_BM) : len;
    const int T = (max(kv_end, 0) + TC_BN - 1) / TC_BN;  // 0: a request without keys, whose rows are zeros
    // the last tile has 16 keys or fewer (a class token behind 24 x 24 patches): a lone CTA computes no more than those, and nothing in warps without a query. (In
    // CTAs that share their SM both only cost: 16 pictures 53.3 -> 53.8 us, causal [1, 2000, 32, 64] 33.5 -> 34.7, [1, 100, 32, 128] 6.2 -> 6.6.)
    const bool stub = WGS == 2 && kv_end - (T - 1) * TC_BN <= 16;

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer: K runs NBUF tiles ahead of V, as the scores do ----------------
            mbar_arrive_expect_tx(q_full, Cfg::Q_BYTES);
            for (int sl = 0; sl < SLABS; ++sl) {
                tma_load_4d(sQ + sl * Q_SLAB, &tm_q, q_full, sl * 64, q0, head, b);
                tma_load_4d(sQ + sl * Q_SLAB + KV_SLAB, &tm_q, q_full, sl * 64, q0 + TC_BN, head, b);
            }
            for (int t = 0; t < T + NBUF; ++t) {
                if (t < T) {
                    const int s = t % STAGES;
                    mbar_wait(&k_empty[s], ((t / STAGES) & 1) ^ 1);
                    mbar_arrive_expect_tx(&k_full[s], Cfg::TILE);
                    for (int sl = 0; sl < SLABS; ++sl) tma_load_4d(sK + s * Cfg::TILE + sl * KV_SLAB, &tm_k, &k_full[s], sl * 64, t * TC_BN, head, b);
                }
                if (t >= NBUF) {
                    const int u = t - NBUF, s = u % STAGES;
                    mbar_wait(&v_empty[s], ((u / STAGES) & 1) ^ 1);
                    mbar_arrive_expect_tx(&v_full[s], Cfg::TILE);
                    for (int sl = 0; sl < SLABS; ++sl) tma_load_4d(sV + s * Cfg::TILE + sl * KV_SLAB, &tm_v, &v_full[s], sl * 64, u * TC_BN, head, b);
                }
            }
        }
    } else if (warp == 1) {
        {
            // ---------------- MMA issuer: walked by the whole warp, an elected lane issues (elect_one, common.cuh) ----------------
            const bool leader = elect_one();
            constexpr uint32_t idesc_s = make_idesc(TC_BM, TC_BN, 0), idesc_o = make_idesc(TC_BM, D, 1);
            const uint64_t q_desc = make_sw128_kmajor_desc(smem_u32(sQ));
            auto scores = [&](int t) {   // S_t: K-loop over the head dim in steps of 16 (32 B inside a 128 B swizzle row; slabs of 64)
                const int s = t % STAGES;
                mbar_wait(&k_full[s], (t / STAGES) & 1);
                tc_fence_after();
                const uint64_t k_desc = make_sw128_kmajor_desc(smem_u32(sK + s * Cfg::TILE));
                if (leader)
#pragma unroll
                for (int k = 0; k < D / 16; ++k)
                    umma_bf16(tm + (t % NBUF) * TC_BN, q_desc + ((k >> 2) * (Q_SLAB >> 4) + (k & 3) * 2), k_desc + ((k >> 2) * (KV_SLAB >> 4) + (k & 3) * 2), idesc_s,
                              k != 0 ? 1u : 0u);
                if (leader) {
                    umma_commit(&k_empty[s]);
                    umma_commit(&s_full[t % NBUF]);
                }
                __syncwarp();
            };
            mbar_wait(q_full, 0);
#pragma unroll 1
            for (int t = -NBUF; t < T; ++t) {
                if (t >= 0) {   // O += P_t V_t once the softmax warps have written P_t (and rescaled O)
                    const int s = t % STAGES, w = t % WGS;
                    mbar_wait(&v_full[s], (t / STAGES) & 1);
                    mbar_wait(&p_full[t % NBUF], (t / NBUF) & 1);
                    tc_fence_after();
                    const uint64_t v_desc = make_sw128_mnmajor_desc(smem_u32(sV + s * Cfg::TILE), KV_SLAB);
                    if (leader)
#pragma unroll
                    for (int k = 0; k < TC_BN / 16; ++k)   // 16 key rows of 128 B per step
                        if (k == 0 || t + 1 < T || !stub) umma_ts(tm + TM_O + w * D, tm + (t % NBUF) * TC_BN + k * 8, v_desc + k * 128, idesc_o, (t >= WGS || k != 0) ? 1u : 0u);
                    if (leader) umma_commit(&v_empty[s]);
                    // the last product has a barrier of its own: its waiters may come while the one before is still under way, and would
                    // take the parity of the one before that for theirs
                    if (leader) umma_commit(t + WGS < T ? &o_done[w] : &o_last[w]);
                    __syncwarp();
                    if (t + NBUF < T) mbar_wait(&o_done[w], (t / WGS) & 1);   // S_(t+NBUF) takes the buffer that P_t was read from
                }
                if (t + NBUF < T) scores(t + NBUF);
            }
        }
    } else {
        // ---------------- softmax / correction / epilogue: thread r <-> query row q0 + r ----------------
        const int quad = warp & 3, w = WGS == 2 ? (warp - 2) >> 2 : 0;   // group w: tiles w, w + WGS, ... and an O, a maximum and a sum of its own
        const int r = quad * 32 + lane;
        const int qrow = q0 + r;
        const uint32_t lanes = tm + (static_cast<uint32_t>(quad * 32) << 16), tm_o = lanes + TM_O + w * D;
        float m_run = -INFINITY, l_run = 0.f;
        auto softmax = [&](int t, auto cols) {   // of the first COLS keys of tile t
            constexpr int COLS = decltype(cols)::value;
            const int key0 = t * TC_BN;
            const uint32_t buf = lanes + (t % NBUF) * TC_BN;
            uint32_t v[COLS];
            __syncwarp();
            if constexpr (COLS == 64) {
                tmem_ld_32x32(buf, reinterpret_cast<uint32_t(&)[32]>(v[0]));
                tmem_ld_32x32(buf + 32, reinterpret_cast<uint32_t(&)[32]>(v[32]));
            } else {
                tmem_ld_cols(buf, v);
            }
            tmem_ld_wait();
            // interior tiles need no per-key mask (CTA-uniform test: every key valid for every query row of this CTA)
            if (!(key0 + COLS <= len && (!CAUSAL || key0 + COLS - 1 <= q0))) {
                const int last = (CAUSAL ? min(len - 1, qrow) : len - 1) - key0;   // last visible key of the tile
#pragma unroll
                for (int i = 0; i < COLS; ++i)
                    if (i > last) v[i] = __float_as_uint(-INFINITY);
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int i = 0; i < COLS; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(v[i]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;  // scale > 0: max commutes with the scaling (-inf stays -inf)
            // lazy rescale: keep the stale max while the new one is < 2^8 above it (P <= 256: exact enough in bf16 / fp32;
            // the stale max cancels in O / l)
            const bool grow = mx > m_run + 8.0f;  // also true on the first valid tile (m_run = -inf)
            const float m_new = grow ? mx : m_run;
            const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            const float corr = grow ? exp2f(m_run - m_use) : 1.0f;  // m_run = -inf -> 0
            if (t >= WGS && __any_sync(0xffffffffu, corr != 1.0f)) {   // rescale the running output (in TMEM) once the previous P·V has landed
                mbar_wait(&o_done[w], (t / WGS - 1) & 1);
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < D / 32; ++c) {
                    uint32_t o[32];
                    __syncwarp();
                    tmem_ld_32x32(tm_o + c * 32, o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                    tmem_st_32x32(tm_o + c * 32, o);
                }
            }
            l_run *= corr;
            m_run = m_new;
            float rs[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t pk[COLS / 2];
#pragma unroll
            for (int i = 0; i < COLS; i += 2) {
                const float p0 = ex2_approx(fmaf(__uint_as_float(v[i]), p.scale_log2, -m_use));   // -inf -> +0
                const float p1 = ex2_approx(fmaf(__uint_as_float(v[i + 1]), p.scale_log2, -m_use));
                rs[(i >> 1) & 3] += p0 + p1;
                pk[i >> 1] = pack_bf16(p0, p1);
            }
            l_run += (rs[0] + rs[1]) + (rs[2] + rs[3]);
            __syncwarp();
            if constexpr (COLS == 64) tmem_st_32x32(buf, pk);   // over the scores of this row
            else tmem_st_32x8(buf, pk);
            tmem_st_wait();
        };
        const bool idle = WGS == 2 && q0 + quad * 32 >= p.S;   // no query in this warp's rows: nothing of O is read there
        for (int t = w; t < T; t += WGS) {
            mbar_wait(&s_full[t % NBUF], (t / NBUF) & 1);
            tc_fence_after();
            if (!idle) {
                if (stub && t + 1 == T) softmax(t, std::integral_constant<int, 16>());
                else softmax(t, std::integral_constant<int, 64>());
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[t % NBUF]);
        }
        // ---- epilogue: O / l (no key: no product to wait for, and nothing of O to read) ----
        float corr[WGS];   // of each group's O, 1 / l included
        if constexpr (WGS == 2) {
            float2* ml = reinterpret_cast<float2*>(tmem_slot + 2);
            ml[w * TC_BM + r] = make_float2(m_run, l_run);
            __syncwarp();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float2 a = ml[r], c = ml[TC_BM + r];
            const float m = fmaxf(a.x, c.x);
            corr[0] = a.x == -INFINITY ? 0.f : exp2f(a.x - m);
            corr[1] = c.x == -INFINITY ? 0.f : exp2f(c.x - m);
            const float l = a.y * corr[0] + c.y * corr[1], inv = l > 0.f ? 1.f / l : 0.f;
            corr[0] *= inv;
            corr[1] *= inv;
        } else {
            corr[0] = l_run > 0.f ? 1.f / l_run : 0.f;
        }
        for (int i = 0; i < WGS; ++i)
            if (T > i) mbar_wait(&o_last[i], 0);
        tc_fence_after();
        __nv_bfloat16* orow = p.o + b * p.o_bs + (int64_t)qrow * p.o_ts + head * p.o_hs;
#pragma unroll
        for (int i = 0; i < D / 32 / WGS; ++i) {   // two groups: half of the columns each
            const int c = w * (D / 32 / WGS) + i;
            float x[32];
            uint32_t v[32];
            __syncwarp();
            tmem_ld_32x32(lanes + TM_O + c * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] = T == 0 ? 0.f : __uint_as_float(v[j]) * corr[0];
            if (WGS == 2 && T > 1) {
                tmem_ld_32x32(lanes + TM_O + D + c * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; ++j) x[j] = fmaf(__uint_as_float(v[j]), corr[WGS - 1], x[j]);
            }
            if (qrow < p.S) {
#pragma unroll
                for (int j = 0; j < 32; j += 8)
                    *reinterpret_cast<uint4*>(orow + c * 32 + j) = make_uint4(pack_bf16(x[j], x[j + 1]), pack_bf16(x[j + 2], x[j + 3]), pack_bf16(x[j + 4], x[j + 5]), pack_bf16(x[j + 6], x[j + 7]));
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tm, TMEM_COLS);
    }
}

// ------------------------------------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                    CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                    CUtensorMapFloatOOBfill);

// 4-D view (d, t, h, b) of a bf16 tensor with element strides (1, ts, hs, bs); box = [64, 64, 1, 1], SWIZZLE_128B
int make_tmap_4d(CUtensorMap* map, const void* ptr, int D, int S, int H, int B, int64_t ts, int64_t hs, int64_t bs) {
    static PFN_encodeTiled fn = nullptr;
    if (fn == nullptr) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess || f == nullptr) {
            set_error("cuTensorMapEncodeTiled entry point unavailable");
            return -2;
        }
        fn = reinterpret_cast<PFN_encodeTiled>(f);
    }
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) != 0 || (ts * 2) % 16 != 0 || (hs * 2) % 16 != 0 || (bs * 2) % 16 != 0) {
        set_error("flash_attn(tc): operands must be 16B aligned with 16B-multiple strides");
        return -1;
    }
    cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {(cuuint64_t)(ts * 2), (cuuint64_t)(hs * 2), (cuuint64_t)(bs * 2)};
    cuuint32_t box[4] = {64, (cuuint32_t)TC_BN, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled(4d) failed (%d): D=%d S=%d H=%d B=%d ts=%lld hs=%lld bs=%lld", (int)r, D, S, H,
                  B, (long long)ts, (long long)hs, (long long)bs);
        return -2;
    }
    return 0;
}

template <int D, bool CAUSAL, int WGS>
int launch_tc(const FlashArgs& a, cudaStream_t stream) {
    CUtensorMap tq, tk, tv;
    B2_TRY(make_tmap_4d(&tq, a.q, D, a.S, a.H, a.B, a.q_ts, a.q_hs, a.q_bs));
    B2_TRY(make_tmap_4d(&tk, a.k, D, a.S, a.H, a.B, a.k_ts, a.k_hs, a.k_bs));
    B2_TRY(make_tmap_4d(&tv, a.v, D, a.S, a.H, a.B, a.v_ts, a.v_hs, a.v_bs));
    FlashTcParams p;
    p.seq_lens = a.seq_lens;
    p.o = reinterpret_cast<__nv_bfloat16*>(a.o);
    p.o_bs = a.o_bs; p.o_ts = a.o_ts; p.o_hs = a.o_hs;
    p.S = a.S;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    constexpr int smem = TcCfg<D, WGS>::SMEM;
    auto kern = flash_tc_kernel<D, CAUSAL, WGS>;
    B2_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid(a.H, a.B, (a.S + TC_BM - 1) / TC_BM);
    B2_CUDA_CHECK(launch_pdl(kern, grid, dim3(64 + 128 * WGS), (size_t)smem, stream, tq, tk, tv, p));
    B2_LAUNCH_CHECK();
    return 0;
}

}  // namespace

int flash_attn_tc_bf16(const FlashArgs& a, cudaStream_t stream) {
    B2_CHECK_ARG(a.D == 64 || a.D == 128, "flash_attn(tc): head_dim must be 64 or 128 (got %d)", a.D);
    B2_CHECK_ARG((a.o_ts % 8) == 0 && (a.o_hs % 8) == 0 && (a.o_bs % 8) == 0 && (reinterpret_cast<uintptr_t>(a.o) & 15) == 0,
                 "flash_attn(tc): output must be 16B aligned with 16B-multiple strides");
    // at most one CTA an SM, and three tiles of keys or more: two groups of softmax warps take the tiles in turn. One group / two, us: [1, 577, 16, 64]
    // 12.0 / 8.9, [1, 1024, 16, 64] 17.8 / 12.7, causal [1, 300, 32, 64] 7.4 / 6.2 (two tiles: 4.7 / 4.4; two such CTAs do not fit an SM: [2, 577, 16, 64] 12.9 / 15.8).
    const bool two = (long long)a.H * a.B * ((a.S + TC_BM - 1) / TC_BM) <= num_sms() && a.S > 2 * TC_BN;
    if (a.D == 64) {
        if (two) return a.causal ? launch_tc<64, true, 2>(a, stream) : launch_tc<64, false, 2>(a, stream);
        return a.causal ? launch_tc<64, true, 1>(a, stream) : launch_tc<64, false, 1>(a, stream);
    }
    if (two) return a.causal ? launch_tc<128, true, 2>(a, stream) : launch_tc<128, false, 2>(a, stream);
    return a.causal ? launch_tc<128, true, 1>(a, stream) : launch_tc<128, false, 1>(a, stream);
}

}  // namespace b2
