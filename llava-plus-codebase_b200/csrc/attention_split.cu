// fp32 attention of a prompt portion on the tensor cores (sm_100a): the same softmax attention over an fp32 cache as
// attn_tile_kernel (attention_bias.cu) with every fp32 operand carried as THREE bf16 parts.
//
// x = hi + mid + lo (bf16 each, round to nearest: 24 significant bits, fp32's exponent range, so no scaling and no loss; what has no parts is
// done over in plain fp32, attn_plain below), and a product
// of two such operands is the six products hi*hi, hi*mid, mid*hi, hi*lo, lo*hi, mid*mid on tcgen05 (kind::f16) with fp32 accumulation;
// the three that are left out lie below 2^-25 of |q| |k|. The tensor core TRUNCATES its fp32 sum after every step of 16 (measured: sums of K
// bf16 products of random sign are off by 1.2e-7 of the result at K = 128 and 1.0e-6 at K = 1024, a serial fp32 chain by 0.7e-7 and
// 2.5e-7; 0.65e-7 against 0.51e-7 at K = 64), so what it adds up is kept short: the small products go first, every 64 entries of the head
// have an accumulator of their own, and the weighted sum of values leaves TMEM after every key tile and is added up in fp32 registers. Scores, bias, soft-cap, mask, maximum, exponential, denominator: fp32 on the
// CUDA cores, as before.
//
// What bounds it: the products (12 of a tile where bf16 attention has 2) and their issue; with them issued by an elected lane of the whole warp instead of by
// one lane's loop, window 129 -> 106 us, tensor pipe active 38.7 -> 48.4 % (profiles/split_attention_scan_ncu.txt). Then the chain of a tile through the
// softmax warps, and CTAs whose rows see few keys beside CTAs whose rows see many. 2048 rows, 16 heads of 128 on 4 key/value heads: window of 1024 + 4
// kept positions 1061 -> 104 us (attn_tile_kernel -> this), no window, 1536 rows on 16 key/value heads 947 -> 80 us; cutting the keys and values: 4 us of
// that call.
// Error of one fp32 layer against 64 bits, old -> new: 5.0e-7 -> 4.7e-7 at 17 rows, 7.1e-7 -> 5.9e-7 at 333, 8.6e-7 -> 6.5e-7 at 2048.
//   1. attn_split_kv_kernel cuts the visible keys and values of the call into parts once (they are read by every query tile);
//   2. attn_split_kernel: CTA = 128 (row, head) pairs of ONE key/value head (rows x the group's query heads, so that a key tile serves
//      all of them), warp 0 TMA producer, warp 1 MMA issuer, warps 2.. softmax: two or four threads per pair, each its share of a tile's
//      keys and of the value columns. S is double-buffered in TMEM: S(t+1) runs while softmax(t) does, O(t) while softmax(t+1) does. P goes to TMEM
//      as the A operand of the second product.
// Key tiles of 64 for key sizes up to 128; the 192 sizes (latent attention with a rotated part) leave room for 32.
#include <cuda.h>
#include <math.h>

#include "kernels.h"
#include "split.cuh"

namespace b2 {

// [planes][rows][pitch] bf16, box = [1][box_rows][64], SWIZZLE_128B (bf16 parts; linear_split.cu uses it too)
int make_tmap_parts(CUtensorMap* map, const void* ptr, int pitch, int64_t nkeys, int planes, int box_rows) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(f) : nullptr;
    }();
    if (fn == nullptr) { set_error("cuTensorMapEncodeTiled entry point unavailable"); return -2; }
    const cuuint64_t dims[3] = {(cuuint64_t)pitch, (cuuint64_t)nkeys, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)nkeys * pitch * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1}, one[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled(parts) failed (%d): %d x %lld x %d", (int)r, pitch, (long long)nkeys, planes); return -2; }
    return 0;
}

namespace {

constexpr int SP_M = 128, SP_SLAB_Q = SP_M * 128, FEW_KEYS = 256;

__device__ __forceinline__ int split_first(int pos, int kind, int size) {   // first position a row at `pos` sees (kept first positions aside)
    if (kind == MASK_WINDOW) return max(0, pos - size + 1);
    if (kind == MASK_CHUNK) return pos / size * size;
    return 0;
}

struct SplitSrc {          // rows of one operand: element (head, key, d) at base + head * hs + key * ks + d
    const float* base;
    int64_t hs, ks;
    int heads, n, pitch;   // entries of a row, pitch of a row of parts (multiple of 8)
    __nv_bfloat16* out;    // [head][part][index][pitch]
    int vec;
};
// index -> key: the kept first positions (nA of them), then the positions from `first` on
__global__ void __launch_bounds__(256) attn_split_kv_kernel(SplitSrc k, SplitSrc v, int nkeys, int nA, int first) {
    pdl_enter();
    const SplitSrc s = blockIdx.y == 0 ? k : v;
    const int chunks = s.pitch >> 3;
    const int64_t total = (int64_t)s.heads * nkeys * chunks;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
        const int c = (int)(e % chunks);
        const int64_t r = e / chunks;
        const int i = (int)(r % nkeys), h = (int)(r / nkeys);
        const int key = i < nA ? i : first + (i - nA);
        float x[8];
        load8(s.base + h * s.hs + key * s.ks, c * 8, s.n, s.vec, x);
        uint4 p0, p1, p2;
        split8(x, p0, p1, p2);
        __nv_bfloat16* o = s.out + ((int64_t)h * 3 * nkeys + i) * s.pitch + c * 8;
        const int64_t part = (int64_t)nkeys * s.pitch;
        *reinterpret_cast<uint4*>(o) = p0;
        *reinterpret_cast<uint4*>(o + part) = p1;
        *reinterpret_cast<uint4*>(o + 2 * part) = p2;
    }
}

// D (+)= A B with A [128 x 16] in TMEM (two bf16 of a row per column) and B by descriptor
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t t, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t t, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tmem_st_done() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
template <int SOFT>
__device__ __forceinline__ void softmax_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * SOFT) : "memory"); }

// MN-major operand of 128-byte rows (64 entries of the row per slab), SWIZZLE_128B; lbo: bytes between the slabs
__device__ __forceinline__ uint64_t make_mn_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}

struct SplitParams {
    BiasAttnArgs a;
    int QT, HG;            // query rows and query heads per CTA (QT * HG <= 128)
    int nA0, first0;       // the index -> key map of the parts
};

template <int DKS, int DVS, int KT>
struct SplitCfg {
    static constexpr int Q_BYTES = 3 * DKS * SP_SLAB_Q, K_BYTES = 3 * DKS * KT * 128, V_BYTES = 3 * DVS * KT * 128;
    static constexpr int SMEM = Q_BYTES + K_BYTES + V_BYTES + 8 * SP_M * 4 + 128 + 1024;
    static constexpr int TM_P = 2 * DKS * KT, TM_O = TM_P + 3 * KT / 2;   // TMEM columns: S [2][DKS][KT], P [3][KT / 2], O
    static_assert(TM_O + 64 * DVS <= 512, "TMEM");
};

// out of line, once in the code: unrolled into the loops below (with the products' loops unrolled too) they made the kernel wait for
// instructions: 220 us against 129 us for 2048 rows of 16 heads of 128 with a window of 1024
__device__ __noinline__ float soft_cap(float v, float cap) { return cap * tanhf(v / cap); }
__device__ __noinline__ float sigmoid_times(float gate, float v) { return v / (1.f + expf(-gate)); }

__device__ __forceinline__ float plain_score(const BiasAttnArgs& a, const float* q, const float* k, int head, int dist) {
    float s = 0.f;
    for (int d = 0; d < a.dk; ++d) s = fmaf(q[d], k[d], s);
    s *= a.scale;
    if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
    if (a.rel != nullptr) s += a.rel[(size_t)a.bucket_of[dist] * a.H + head];
    return s;
}
// Value columns [d0, d1) of one (row, head) in plain fp32, for a row that saw an operand without parts (split.cuh): maximum, denominator, then 16
// columns at a time. Keys that the row does not see have no part in it. Once the denominator, or all 16 columns, are NaN they stay so.
__device__ __noinline__ void attn_plain(const SplitParams& p, int row, int head, int pos, int d0, int d1) {
    const BiasAttnArgs& a = p.a;
    const int g = head / p.HG, Gv = a.Gv > 0 ? a.Gv : a.G, gv = g % Gv;
    const bool mat = a.kv_row_stride > 0;
    const float* K = mat ? a.kcache + (size_t)g * a.dk : a.kcache + ((size_t)a.slot * a.G + g) * a.Smax * a.dk;
    const float* V = mat ? a.vcache + (size_t)gv * a.dv : a.vcache + ((size_t)a.slot * Gv + gv) * a.Smax * a.dv;
    const size_t ks = mat ? (size_t)a.kv_row_stride : (size_t)a.dk, vs = mat ? (size_t)a.kv_row_stride_v : (size_t)a.dv;
    const float* q = a.q + (size_t)row * a.ldq + (size_t)head * a.dk;
    const int first = split_first(pos, a.mask_kind, a.mask_size), kept = min(a.mask_kind == MASK_WINDOW ? a.mask_keep : 0, first);
    auto next = [&](int j) { return j + 1 == kept ? first : j + 1; };   // visible keys: [0, kept) and [first, pos]
    const int start = kept > 0 ? 0 : first;
    float m = -INFINITY, l = 0.f;
    for (int j = start; j <= pos; j = next(j)) m = fmaxf(m, plain_score(a, q, K + j * ks, head, pos - j));
    const float m_use = m == -INFINITY ? 0.f : m;
    for (int j = start; j <= pos && l == l; j = next(j)) l += expf(plain_score(a, q, K + j * ks, head, pos - j) - m_use);
    float inv = 1.f / l;
    if (a.sink != nullptr || a.sink_fixed) {
        const float sk = a.sink != nullptr ? a.sink[head] : a.sink_value, mf = fmaxf(m, sk), c0 = expf(m - mf);
        inv = c0 / fmaf(l, c0, expf(sk - mf));
    }
    if (a.head_gate != nullptr) inv /= 1.f + expf(-a.head_gate[(size_t)row * a.ldg + head]);
    const float* cg = a.chan_gate != nullptr ? a.chan_gate + (size_t)row * a.ldg + (size_t)head * (a.chan_step ? a.dv : 1) : nullptr;
    const size_t at = (size_t)row * a.ldo + (size_t)head * a.dv;
    for (int d = d0; d < d1; d += 16) {
        float o[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) o[c] = 0.f;
        bool live = inv == inv;
        for (int j = start; j <= pos && live; j = next(j)) {
            const float w = expf(plain_score(a, q, K + j * ks, head, pos - j) - m_use);
            live = false;
#pragma unroll
            for (int c = 0; c < 16; ++c)
                if (d + c < d1) {
                    o[c] = fmaf(w, V[j * vs + d + c], o[c]);
                    live |= o[c] == o[c];
                }
        }
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            if (d + c >= d1) continue;
            float y = o[c] * inv;
            if (cg != nullptr) y = sigmoid_times(cg[(d + c) * a.chan_step], y);
            if (a.out16 != nullptr) reinterpret_cast<__nv_bfloat16*>(a.out16)[at + d + c] = __float2bfloat16_rn(y);
            else a.out[at + d + c] = y;
        }
    }
}

template <int DKS, int DVS, int KT, bool EXTRA, int SOFT, bool ONE = false>   // EXTRA: soft-cap or distance bias; SOFT: softmax warps, 8 or 16; ONE: one channel gate a head
__global__ void __launch_bounds__(64 + 32 * SOFT, 1) attn_split_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                                                                   const __grid_constant__ SplitParams p) {
    using Cfg = SplitCfg<DKS, DVS, KT>;
    constexpr int SP_THREADS = 64 + 32 * SOFT, SHARES = SOFT / 4;             // softmax threads of a pair
    constexpr int KH = KT / 2, KQ = KT / SHARES, CQ = 64 * DVS / SHARES;       // TMEM columns of a part of P; keys of a tile and value columns of one of them
    extern __shared__ uint8_t sp_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sp_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t* sQ = smem;                          // [part][slab][128 pairs][128 B]
    uint8_t* sK = sQ + Cfg::Q_BYTES;             // [part][slab][KT keys][128 B]
    uint8_t* sV = sK + Cfg::K_BYTES;             // [part][slab][KT keys][128 B]
    float* s_red = reinterpret_cast<float*>(sV + Cfg::V_BYTES);   // [tile parity][share][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(s_red + 8 * SP_M);
    uint64_t *k_full = bars, *k_empty = bars + 1, *v_full = bars + 2, *v_empty = bars + 3, *s_full = bars + 4 /*[2]*/, *p_full = bars + 6, *o_full = bars + 7;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);

    const BiasAttnArgs& a = p.a;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, HG = p.HG;
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        for (int i = 0; i < 8; ++i) mbar_init(&bars[i], i == 6 ? SOFT : 1);   // p_full: one arrive per softmax warp
        fence_barrier_init();
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *tmem_slot;
    pdl_trigger_small();   // (behind the allocation: see tmem_alloc)
    pdl_wait();

    // the query tiles with the most keys go first
    const int nq = (a.rows + p.QT - 1) / p.QT, qt = nq - 1 - (int)(blockIdx.x / a.G), g = blockIdx.x % a.G;
    const int gv = a.Gv > 0 ? g % a.Gv : g;
    const int r0 = qt * p.QT, nrows = min(p.QT, a.rows - r0), P = nrows * HG;
    const int minpos = a.row_pos[r0], maxpos = a.row_pos[r0 + nrows - 1];   // consecutive positions of one slot
    const int first = split_first(minpos, a.mask_kind, a.mask_size), maxfirst = split_first(maxpos, a.mask_kind, a.mask_size);
    const int keep = a.mask_kind == MASK_WINDOW ? a.mask_keep : 0;
    // visible keys: [0, nA) (kept first positions in front of the earliest window) and [first, maxpos], in tiles of KT
    const int nA = min(keep, first), tilesA = (nA + KT - 1) / KT, T = tilesA + (maxpos + 1 - first + KT - 1) / KT;
    auto tile_start = [&](int t) { return t < tilesA ? t * KT : first + (t - tilesA) * KT; };

    auto load_tile = [&](const CUtensorMap* map, uint8_t* dst, uint64_t* bar, int t, int head, int slabs, int bytes) {
        const int j0 = tile_start(t), i0 = j0 < p.nA0 ? j0 : j0 - p.first0 + p.nA0;
        mbar_arrive_expect_tx(bar, bytes);
        for (int part = 0; part < 3; ++part)
            for (int s = 0; s < slabs; ++s) tma_load_3d(dst + (part * slabs + s) * KT * 128, map, bar, s * 64, i0, head * 3 + part);
    };
    if (threadIdx.x == 0) {   // the first tiles travel while the queries are cut
        load_tile(&tm_k, sK, k_full, 0, g, DKS, Cfg::K_BYTES);
        load_tile(&tm_v, sV, v_full, 0, gv, DVS, Cfg::V_BYTES);
    }
    {   // queries: pair = row * HG + head; parts into the swizzled K-major operand tiles, idle pairs and entries past dk as zeros
        const bool vec = a.dk % 4 == 0 && a.ldq % 4 == 0 && (reinterpret_cast<uintptr_t>(a.q) & 15) == 0;
        constexpr int U = SOFT == 8 ? 4 : 2, TASKS = SP_M * DKS * 8;   // a task is 8 entries of a pair; a thread has the loads of U in flight
        for (int e0 = threadIdx.x; e0 < TASKS; e0 += SP_THREADS * U) {
            float x[U][8];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * SP_THREADS, pair = e / (DKS * 8), c = e % (DKS * 8);
                if (pair < P) load8(a.q + (size_t)(r0 + pair / HG) * a.ldq + (size_t)(g * HG + pair % HG) * a.dk, c * 8, a.dk, vec, x[u]);
                else
#pragma unroll
                    for (int i = 0; i < 8; ++i) x[u][i] = 0.f;
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = e0 + u * SP_THREADS, pair = e / (DKS * 8), c = e % (DKS * 8);
                if (e >= TASKS) break;
                uint4 h, m, l;
                split8(x[u], h, m, l);
                uint8_t* d = sQ + (c >> 3) * SP_SLAB_Q + pair * 128 + (((c & 7) ^ (pair & 7)) << 4);
                *reinterpret_cast<uint4*>(d) = h;
                *reinterpret_cast<uint4*>(d + DKS * SP_SLAB_Q) = m;
                *reinterpret_cast<uint4*>(d + 2 * DKS * SP_SLAB_Q) = l;
            }
        }
    }
    fence_proxy_async();
    __syncthreads();

    if (warp == 0) {
        if (lane == 0) {
            // K runs one tile ahead of V, as the scores do: K(t+1) replaces K(t) as soon as S(t) is done, while O(t-1) is computed
            for (int t = 0; t < T; ++t) {
                if (t + 1 < T) {
                    mbar_wait(k_empty, t & 1);
                    load_tile(&tm_k, sK, k_full, t + 1, g, DKS, Cfg::K_BYTES);
                }
                if (t > 0) {
                    mbar_wait(v_empty, (t - 1) & 1);
                    load_tile(&tm_v, sV, v_full, t, gv, DVS, Cfg::V_BYTES);
                }
            }
        }
    } else if (warp == 1) {
        {
            // walked by the whole warp, an elected lane issues (elect_one, common.cuh); the loops stay rolled: the kernel's roles share the instruction cache
            const bool leader = elect_one();
            constexpr uint32_t idesc_s = make_idesc_bf16_f32(SP_M, KT), idesc_o = make_idesc_bf16_f32(SP_M, 64 * DVS) | (1u << 16);
            const uint64_t q_desc = make_sw128_kmajor_desc(smem_u32(sQ)), k_desc = make_sw128_kmajor_desc(smem_u32(sK)), v_desc = make_mn_desc(smem_u32(sV), KT * 128);
#pragma unroll 1
            for (int t = -1; t < T; ++t) {
                if (t + 1 < T) {   // S(t+1); its buffer was read before P(t-1) was announced
                    mbar_wait(k_full, (t + 1) & 1);
                    tc_fence_after();
                    const uint32_t d0 = tm + ((t + 1) & 1) * DKS * KT;
#pragma unroll 1
                    for (int i = 0; i < 6; ++i) {
                        const uint32_t pa = (SPLIT_A >> (2 * i)) & 3u, pb = (SPLIT_B >> (2 * i)) & 3u;
                        if (leader)
#pragma unroll
                        for (int s = 0; s < DKS; ++s)   // a slab of 64 entries of the head has an accumulator of its own
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                umma_bf16(d0 + s * KT, q_desc + ((pa * DKS + s) * (SP_SLAB_Q >> 4) + 2 * k), k_desc + ((pb * DKS + s) * (KT * 8) + 2 * k), idesc_s,
                                          (i | k) != 0 ? 1u : 0u);
                    }
                    if (leader) {
                        umma_commit(k_empty);
                        umma_commit(&s_full[(t + 1) & 1]);
                    }
                    __syncwarp();
                }
                if (t >= 0) {   // O(t)
                    mbar_wait(v_full, t & 1);
                    mbar_wait(p_full, t & 1);
                    tc_fence_after();
#pragma unroll 1
                    for (int i = 0; i < 6; ++i) {
                        const uint32_t pa = (SPLIT_A >> (2 * i)) & 3u, pb = (SPLIT_B >> (2 * i)) & 3u;
                        if (leader)
#pragma unroll
                        for (int k = 0; k < KT / 16; ++k)
                            umma_ts(tm + Cfg::TM_O, tm + Cfg::TM_P + pa * KH + k * 8, v_desc + (pb * (DVS * KT * 8) + k * 128), idesc_o, (i | k) != 0 ? 1u : 0u);
                    }
                    if (leader) {
                        umma_commit(v_empty);
                        umma_commit(o_full);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        const int quad = warp & 3, share = (warp - 2) >> 2, pair = quad * 32 + lane;
        const uint32_t lanes = tm + (static_cast<uint32_t>(quad * 32) << 16);
        const bool live = pair < P;
        const int row = r0 + (live ? pair / HG : 0), head = g * HG + (live ? pair % HG : 0);
        const int pos = live ? minpos + pair / HG : -1, pfirst = split_first(max(pos, 0), a.mask_kind, a.mask_size);
        float m = -INFINITY, l = 0.f, corr = 1.f, o[CQ];
#pragma unroll
        for (int c = 0; c < CQ; ++c) o[c] = 0.f;
        auto join = [&](int t) {   // O(t), in the measure of the maximum that P(t) had
            mbar_wait(o_full, t & 1);
            tc_fence_after();
            constexpr int W = CQ < 32 ? CQ : 32;
#pragma unroll
            for (int c = 0; c < CQ; c += W) {
                uint32_t v[W];
                __syncwarp();
                tmem_ld_cols(lanes + Cfg::TM_O + share * CQ + c, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < W; ++i) o[c + i] = fmaf(o[c + i], corr, __uint_as_float(v[i]));
            }
            tc_fence_before();
        };
        for (int t = 0; t < T; ++t) {
            const int j0 = tile_start(t), jh = j0 + share * KQ;
            const int nk = min(KT, (t < tilesA ? nA : maxpos + 1) - j0);
            const bool full = nk == KT && j0 + KT <= minpos + 1 && (t < tilesA || j0 >= maxfirst);   // every pair sees every key of the tile
            float s[KQ];
            mbar_wait(&s_full[t & 1], (t >> 1) & 1);
            tc_fence_after();
            __syncwarp();
#pragma unroll
            for (int sl = 0; sl < DKS; ++sl) {
                uint32_t u[KQ];
                tmem_ld_cols(lanes + ((t & 1) * DKS + sl) * KT + share * KQ, u);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < KQ; ++i) s[i] = sl == 0 ? __uint_as_float(u[i]) : s[i] + __uint_as_float(u[i]);
            }
            tc_fence_before();
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < KQ; ++i) {
                s[i] *= a.scale;
                if (EXTRA && a.softcap > 0.f) s[i] = soft_cap(s[i], a.softcap);
            }
            if (EXTRA && a.rel != nullptr) {   // all of the tile's rows of the bias table, then all of its entries
                int b[KQ];
#pragma unroll
                for (int i = 0; i < KQ; ++i) b[i] = a.bucket_of[max(pos - jh - i, 0)];
#pragma unroll
                for (int i = 0; i < KQ; ++i) s[i] += a.rel[(size_t)b[i] * a.H + head];
            }
            if (!full) {
                const int hi = min(pos, j0 + nk - 1) - jh, lo = pfirst - jh, kept = keep - jh;
#pragma unroll
                for (int i = 0; i < KQ; ++i)
                    if (!(i <= hi && (i >= lo || i < kept))) s[i] = -INFINITY;
            }
#pragma unroll
            for (int i = 0; i < KQ; ++i) mx = fmaxf(mx, s[i]);
            float* red = s_red + (t & 1) * 4 * SP_M;
            red[share * SP_M + pair] = mx;
            softmax_sync<SOFT>();
#pragma unroll
            for (int i = 0; i < SHARES; ++i) mx = fmaxf(mx, red[i * SP_M + pair]);
            const float m_new = fmaxf(m, mx), m_use = m_new == -INFINITY ? 0.f : m_new, c_new = expf(m - m_use);   // (m = -inf: 0)
            m = m_new;
            float sum = 0.f;
            uint32_t part[3][KQ / 2];
#pragma unroll
            for (int i = 0; i < KQ; i += 2) {
                const float p0 = expf(s[i] - m_use), p1 = expf(s[i + 1] - m_use);
                sum += p0 + p1;
                split3(p0, p1, part[0][i / 2], part[1][i / 2], part[2][i / 2]);
            }
            l = fmaf(l, c_new, sum);
            if (t > 0) join(t - 1);   // (P's buffer is free after that, too)
            corr = c_new;
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                if constexpr (KQ == 8) tmem_st4(lanes + Cfg::TM_P + q * KH + share * (KQ / 2), part[q]);
#pragma unroll
                for (int c = 0; c < KQ / 16; ++c) tmem_st8(lanes + Cfg::TM_P + q * KH + share * (KQ / 2) + c * 8, &part[q][c * 8]);
            }
            tmem_st_done();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        join(T - 1);
        float* red = s_red + (T & 1) * 4 * SP_M;
        red[share * SP_M + pair] = l;
        softmax_sync<SOFT>();
        l = red[pair] + red[SP_M + pair];
        if constexpr (SHARES == 4) l += red[2 * SP_M + pair] + red[3 * SP_M + pair];
        bool plain = l != l;
#pragma unroll
        for (int c = 0; c < CQ; ++c) plain |= o[c] != o[c];
        if (live && plain) {
            attn_plain(p, row, head, pos, share * CQ, min((share + 1) * CQ, a.dv));
        } else if (live) {
            float inv = 1.f / l;
            if (a.sink != nullptr || a.sink_fixed) {   // the sink joins the denominator once, under the common maximum
                const float sk = a.sink != nullptr ? a.sink[head] : a.sink_value, mf = fmaxf(m, sk), c0 = expf(m - mf);
                inv = c0 / fmaf(l, c0, expf(sk - mf));
            }
            if (a.head_gate != nullptr) inv /= 1.f + expf(-a.head_gate[(size_t)row * a.ldg + head]);
            const int d0 = share * CQ;
            const float* cg = a.chan_gate != nullptr ? a.chan_gate + (size_t)row * a.ldg + (size_t)head * (a.chan_step ? a.dv : 1) : nullptr;
            if constexpr (ONE) {
                const float den = 1.f + expf(-cg[0]);
#pragma unroll
                for (int c = 0; c < CQ; ++c) o[c] = o[c] * inv / den;
            }
            const size_t at = (size_t)row * a.ldo + (size_t)head * a.dv;
            const bool vec = a.dv % 4 == 0 && a.ldo % 4 == 0 &&
                             (a.out16 != nullptr ? (reinterpret_cast<uintptr_t>(a.out16) & 7) == 0 : (reinterpret_cast<uintptr_t>(a.out) & 15) == 0);
#pragma unroll
            for (int c = 0; c < CQ; c += 4) {
                float y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int d = d0 + c + i;
                    y[i] = ONE ? o[c + i] : o[c + i] * inv;
                    if (!ONE && cg != nullptr && d < a.dv) y[i] = sigmoid_times(cg[d], y[i]);
                }
                if (vec && d0 + c + 4 <= a.dv) {
                    if (a.out16 != nullptr) *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out16) + at + d0 + c) = make_uint2(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]));
                    else *reinterpret_cast<float4*>(a.out + at + d0 + c) = make_float4(y[0], y[1], y[2], y[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (d0 + c + i < a.dv) {
                            if (a.out16 != nullptr) reinterpret_cast<__nv_bfloat16*>(a.out16)[at + d0 + c + i] = __float2bfloat16_rn(y[i]);
                            else a.out[at + d0 + c + i] = y[i];
                        }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tm, 512); }
}

template <int DKS, int DVS, int KT>
int launch_split(const SplitParams& p, const SplitSrc& k, const SplitSrc& v, int nkeys, cudaStream_t st) {
    using Cfg = SplitCfg<DKS, DVS, KT>;
    CUtensorMap tk, tv;
    B2_TRY(make_tmap_parts(&tk, k.out, k.pitch, nkeys, 3 * k.heads, KT));
    B2_TRY(make_tmap_parts(&tv, v.out, v.pitch, nkeys, 3 * v.heads, KT));
    // Four threads a pair where a tile is a long chain (soft-cap, bias: 600 rows of a fp32 layer 850 -> 816 us a pass) and for few keys, where the
    // time goes into queries, first use and last write (a pass of 41 rows through four layers 339 -> 329, 200 rows through one 126.9 -> 123.9); from
    // there on two, whose exchanges are fewer (260 rows 241.0 / 240.2, 1000 rows 324.8 / 321.0, 2048 rows 336 / 332). 18 warps leave a thread 96 registers:
    // with value heads of 128 the four-thread form spills (208 / 148 bytes stored / loaded at <2, 2, 64, true, 16>, 132 / 140 without cap and bias).
    const bool extra = p.a.softcap > 0.f || p.a.rel != nullptr, wide = extra || nkeys <= FEW_KEYS;
    const bool one = p.a.chan_gate != nullptr && p.a.chan_step == 0;   // (a kernel of its own: in the others its divisions cost 1 % of a layer without them)
    auto kernel = extra ? (one ? attn_split_kernel<DKS, DVS, KT, true, 16, true> : attn_split_kernel<DKS, DVS, KT, true, 16>)
                  : wide ? (one ? attn_split_kernel<DKS, DVS, KT, false, 16, true> : attn_split_kernel<DKS, DVS, KT, false, 16>)
                         : (one ? attn_split_kernel<DKS, DVS, KT, false, 8, true> : attn_split_kernel<DKS, DVS, KT, false, 8>);
    B2_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM));
    launch_pdl(kernel, dim3(((p.a.rows + p.QT - 1) / p.QT) * p.a.G), dim3(64 + 32 * (wide ? 16 : 8)), Cfg::SMEM, st, tk, tv, p);
    B2_LAUNCH_CHECK();
    return 0;
}

int pad8(int n) { return (n + 7) / 8 * 8; }

// keys the call's rows see: nA kept first positions, then [first, key_end)
void key_range(const BiasAttnArgs& a, int& nA, int& first, int& nkeys) {
    const int pos0 = a.key_end - a.rows;
    first = a.mask_kind == MASK_WINDOW ? (pos0 - a.mask_size + 1 > 0 ? pos0 - a.mask_size + 1 : 0) : a.mask_kind == MASK_CHUNK ? pos0 / a.mask_size * a.mask_size : 0;
    nA = a.mask_kind == MASK_WINDOW ? (a.mask_keep < first ? a.mask_keep : first) : 0;
    nkeys = nA + a.key_end - first;
}

}  // namespace

size_t attn_split_bytes_per_key(int G, int Gv, int dk, int dv) { return (size_t)6 * ((size_t)G * pad8(dk) + (size_t)Gv * pad8(dv)); }

bool attn_split_fits(const BiasAttnArgs& a) {
    if (a.parts == nullptr || a.key_end < a.rows || a.nsplit != 1 || a.tile_rows != a.rows || a.vcache == a.kcache) return false;
    if (a.dk > 192 || a.dv > 128 || a.H / a.G > SP_M || a.rows < ATTN_SPLIT_MIN_ROWS) return false;
    int nA, first, nkeys;
    key_range(a, nA, first, nkeys);
    if (nkeys < ATTN_SPLIT_MIN_KEYS) return false;
    return (size_t)nkeys * attn_split_bytes_per_key(a.G, a.Gv > 0 ? a.Gv : a.G, a.dk, a.dv) <= a.parts_bytes;
}

int attn_split_f32(const BiasAttnArgs& a, cudaStream_t st) {
    const int Gv = a.Gv > 0 ? a.Gv : a.G;
    SplitParams p;
    int nkeys;
    p.a = a;
    key_range(a, p.nA0, p.first0, nkeys);
    p.HG = a.H / a.G;
    p.QT = SP_M / p.HG;
    const bool mat = a.kv_row_stride > 0;
    SplitSrc k, v;
    k.heads = a.G; k.n = a.dk; k.pitch = pad8(a.dk); k.out = reinterpret_cast<__nv_bfloat16*>(a.parts);
    k.base = mat ? a.kcache : a.kcache + (size_t)a.slot * a.G * a.Smax * a.dk;
    k.hs = mat ? a.dk : (int64_t)a.Smax * a.dk; k.ks = mat ? a.kv_row_stride : a.dk;
    v.heads = Gv; v.n = a.dv; v.pitch = pad8(a.dv); v.out = k.out + (size_t)3 * a.G * nkeys * k.pitch;
    v.base = mat ? a.vcache : a.vcache + (size_t)a.slot * Gv * a.Smax * a.dv;
    v.hs = mat ? a.dv : (int64_t)a.Smax * a.dv; v.ks = mat ? a.kv_row_stride_v : a.dv;
    for (SplitSrc* s : {&k, &v}) s->vec = s->hs % 4 == 0 && s->ks % 4 == 0 && (reinterpret_cast<uintptr_t>(s->base) & 15) == 0;
    const int64_t most = (int64_t)nkeys * (k.heads * (k.pitch / 8) > v.heads * (v.pitch / 8) ? k.heads * (k.pitch / 8) : v.heads * (v.pitch / 8));
    const int64_t blocks = (most + 255) / 256, cap = (int64_t)num_sms() * 8;
    launch_pdl(attn_split_kv_kernel, dim3((unsigned)(blocks < cap ? blocks : cap), 2), dim3(256), 0, st, k, v, nkeys, p.nA0, p.first0);
    B2_LAUNCH_CHECK();
    const bool v1 = a.dv <= 64;
    if (a.dk <= 64) return v1 ? launch_split<1, 1, 64>(p, k, v, nkeys, st) : launch_split<1, 2, 64>(p, k, v, nkeys, st);
    if (a.dk <= 128) return v1 ? launch_split<2, 1, 64>(p, k, v, nkeys, st) : launch_split<2, 2, 64>(p, k, v, nkeys, st);
    return v1 ? launch_split<3, 1, 32>(p, k, v, nkeys, st) : launch_split<3, 2, 32>(p, k, v, nkeys, st);
}

}  // namespace b2
