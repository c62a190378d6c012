// The linear recurrence of a long prompt (S <- D S + k v^T, y = S^T q per head, recurrent.cu) in blocks of 64 tokens, its contractions on the tensor cores.
// With G_t the product of the decays from the block's start through token t, per key, and S_0 the state in front of the block:
//   y_t = (q_t G_t)^T S_0 + sum_{s <= t} A[t][s] v_s,  A[t][s] = sum_keys q_t k_s d_(s+1) .. d_t,  S_64 = G_64 S_0 + sum_s (k_s d_(s+1) .. d_63) v_s^T
// (RWKV reads the state in front of a token: G_(t-1), A up to d_(t-1), A[t][t] = q_t u k_t). All decays are multiplied up, none divided by.
//   1. sb_prepare_kernel, a CTA per (block, head): the gates; A on the FMA pipe (a lane holds k_s of 8 or 16 keys and multiplies the decays on from token to
//      token: 1/8 of the arithmetic of walking a state of 256 columns); q G, k with the decays behind it and A as the bf16 parts of split.cuh, laid out as
//      the products read them;
//   2. sb_states_kernel, a CTA per (block, head, 128 columns): what the block adds to the state, V^T (128 x 64 tokens) times K;
//   3. sb_fold_kernel: the blocks in order, S = G S + what the block adds, a thread per 4 columns of a key; leaves the state in front of every block;
//   4. sb_output_kernel, a CTA per (block, head, 128 columns): S_0^T Q over the keys in blocks of 64, then V^T A; each in an accumulator of its own (the
//      tensor core cuts its fp32 sums off after every step of 16), added up in registers;
//   5. recurrent.cu's walk once more, for heads with an operand or a sum that the parts do not hold (infinities, NaN, magnitudes about 2^128): for the
//      others that launch only puts the new state in its place. Nothing before it touches the state or the inputs.
// What bounds it: the first kernel's instructions (the gates, A, the cutting into parts: 33 of 103 us at 1900 tokens, 8 heads of 128 x 256), then L2: the
// states pass through it four times (31 MB each; 21 + 10 + 32 us for the other three). The walk in chunks took 191 us there; one layer of gated linear attention
// of width 2048 444 -> 360 us. Smaller blocks would pass more states, larger ones square A; cutting the keys of a block over a cluster or the
// first kernel into parts of 16 tokens with plain products between them measured the same within 5 %.
#include <algorithm>
#include <type_traits>

#include "scan.cuh"
#include "split.cuh"

namespace b2 {
namespace {

constexpr float SB_HELD = 3.38e38f;   // magnitudes from 2^128 (1 - 2^-9) = 3.396e38 on round to a bf16 infinity (split.cuh)
constexpr int SB_THREADS = 256;

__device__ __forceinline__ bool held(float x) { return fabsf(x) < SB_HELD; }   // (a NaN is not)
__device__ __forceinline__ void put_parts(uint8_t* at, int part_bytes, const float (&x)[8]) {
    uint4 h, m, l;
    split8(x, h, m, l);
    *reinterpret_cast<uint4*>(at) = h;
    *reinterpret_cast<uint4*>(at + part_bytes) = m;
    *reinterpret_cast<uint4*>(at + 2 * part_bytes) = l;
}
__device__ __forceinline__ int sw128(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }   // 16-byte chunk of a row of 128 bytes

// KB: blocks of 64 keys
template <int MODE, int KB>
__global__ void __launch_bounds__(SB_THREADS, 2) sb_prepare_kernel(ScanArgs a, BlockScan p) {
    pdl_enter();
    constexpr int DKP = KB * 64, KQ = DKP / 4;
    extern __shared__ __align__(16) float sb_sm[];
    float *sq = sb_sm, *sd = sq + SB_TOK * DKP, *sk = sd + SB_TOK * DKP /* then A, in two halves */;
    const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const SeqSeg sg = a.segs[0];
    const int t0 = p.t0 + b * SB_TOK, nt = min(SB_TOK, p.t0 + p.n - t0), dk = a.dk;
    const size_t row0 = (size_t)sg.row0 + t0, bh = (size_t)b * a.heads + h;
    bool bad = false;
    for (int e = tid; e < SB_TOK * KQ; e += SB_THREADS) {
        const int t = e / KQ, key = (e % KQ) * 4;
        float q[4] = {0.f, 0.f, 0.f, 0.f}, k[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {1.f, 1.f, 1.f, 1.f};
        if (t < nt && key < dk) {
            const float4 q4 = *reinterpret_cast<const float4*>(a.q + (row0 + t) * a.ldq + (size_t)h * dk + key);
            q[0] = q4.x; q[1] = q4.y; q[2] = q4.z; q[3] = q4.w;
            if (MODE != SCAN_HGRN2) {
                const float4 k4 = *reinterpret_cast<const float4*>(a.k + (row0 + t) * a.ldk + (size_t)h * dk + key);
                k[0] = k4.x; k[1] = k4.y; k[2] = k4.z; k[3] = k4.w;
            }
            const float4 d4 = *reinterpret_cast<const float4*>(a.decay_in + (row0 + t) * a.ldd + (size_t)h * dk + key);
            d[0] = d4.x; d[1] = d4.y; d[2] = d4.z; d[3] = d4.w;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                d[i] = scan_decay<MODE>(a, h * dk + key + i, d[i]);
                if (MODE != SCAN_RWKV) q[i] = scan_query<MODE>(a, q[i]);
                if (MODE == SCAN_HGRN2) k[i] = 1.f - d[i];
                bad |= !held((fabsf(q[i]) + fabsf(k[i])) + fabsf(d[i]));
            }
        }
        *reinterpret_cast<float4*>(sq + t * DKP + key) = make_float4(q[0], q[1], q[2], q[3]);
        *reinterpret_cast<float4*>(sk + t * DKP + key) = make_float4(k[0], k[1], k[2], k[3]);
        *reinterpret_cast<float4*>(sd + t * DKP + key) = make_float4(d[0], d[1], d[2], d[3]);
    }
    __syncthreads();
    // A: a warp takes half of the keys (eight lanes share them out) and tokens s = 4 w + (0..3) + 16 j, four a lane, and walks t: a read of q_t and d_t
    // serves them all
    constexpr int KL = KB * 4;   // keys a lane: four consecutive ones of each 32 of its half
    const int grp = lane & 7, w4 = warp & 3, kh = warp >> 2, s0 = w4 * 4 + (lane >> 3);
    float w[4][KL];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < KB; ++i) {
            const float4 f = *reinterpret_cast<const float4*>(sk + (s0 + 16 * j) * DKP + kh * (DKP / 2) + i * 32 + grp * 4);
            w[j][4 * i] = f.x; w[j][4 * i + 1] = f.y; w[j][4 * i + 2] = f.z; w[j][4 * i + 3] = f.w;
        }
    float bon[MODE == SCAN_RWKV ? KL : 1];
    if (MODE == SCAN_RWKV)
#pragma unroll
        for (int i = 0; i < KL; ++i) {
            const int key = kh * (DKP / 2) + (i >> 2) * 32 + grp * 4 + (i & 3);
            bon[i] = key < dk ? a.bonus[(size_t)h * dk + key] : 0.f;
        }
    __syncthreads();
    if (tid < DKP) {   // k times the decays behind its token, in place
        float gd = 1.f;
#pragma unroll 8
        for (int t = SB_TOK - 1; t >= 0; --t) { sk[t * DKP + tid] *= gd; gd *= sd[t * DKP + tid]; }
        if (tid < dk) p.decay[bh * dk + tid] = gd;
    }
    __syncthreads();
    for (int u = tid; u < DKP * 8; u += SB_THREADS) {   // two chunks of 8 tokens (a sector of a row) and 16 keys a warp
        const int key = (u >> 7) * 16 + (u & 15), o = ((u >> 4) & 7);
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = sk[(o * 8 + j) * DKP + key];
        put_parts(p.k + bh * (3 * DKP * 128) + sw128(key, o), DKP * 128, x);
    }
    __syncthreads();
    for (int e = tid; e < 2 * SB_TOK * SB_TOK / 4; e += SB_THREADS) reinterpret_cast<float4*>(sk)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const auto walk = [&](int t, auto last, auto own) {   // tokens j <= last have begun; own: t is one of the warp's tokens of j == last
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        float q[KL], d[KL];
#pragma unroll
        for (int i = 0; i < KB; ++i) {
            const float4 q4 = *reinterpret_cast<const float4*>(sq + t * DKP + kh * (DKP / 2) + i * 32 + grp * 4);
            q[4 * i] = q4.x; q[4 * i + 1] = q4.y; q[4 * i + 2] = q4.z; q[4 * i + 3] = q4.w;
            const float4 d4 = *reinterpret_cast<const float4*>(sd + t * DKP + kh * (DKP / 2) + i * 32 + grp * 4);
            d[4 * i] = d4.x; d[4 * i + 1] = d4.y; d[4 * i + 2] = d4.z; d[4 * i + 3] = d4.w;
        }
#pragma unroll
        for (int j = 0; j <= last.value; ++j) {
            const int s = s0 + 16 * j;
            const bool mine = own.value != 0 && j == last.value, behind = !mine || t > s;
#pragma unroll
            for (int i = 0; i < KL; ++i) {
                if (MODE == SCAN_RWKV) {
                    acc[j] = fmaf(q[i], mine && t == s ? bon[i] * w[j][i] : w[j][i], acc[j]);
                    w[j][i] *= behind ? d[i] : 1.f;
                } else {
                    w[j][i] *= behind ? d[i] : 1.f;
                    acc[j] = fmaf(q[i], w[j][i], acc[j]);
                }
            }
            if (mine && t < s) acc[j] = 0.f;
        }
        // the eight lanes' sums: lane g ends up with j = 2 (g & 1) + (g >> 1 & 1)
        const bool b0 = grp & 1, b1 = grp & 2;
        float u0 = b0 ? acc[2] : acc[0], u1 = b0 ? acc[3] : acc[1];
        u0 += __shfl_xor_sync(0xffffffffu, b0 ? acc[0] : acc[2], 1);
        u1 += __shfl_xor_sync(0xffffffffu, b0 ? acc[1] : acc[3], 1);
        float r = b1 ? u1 : u0;
        r += __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
        r += __shfl_xor_sync(0xffffffffu, r, 4);
        if (grp < 4) sk[(kh * SB_TOK + t) * SB_TOK + s0 + 16 * (2 * (grp & 1) + (grp >> 1))] = r;
    };
    const auto quarter = [&](auto last) {
        const int t0q = 16 * last.value + 4 * w4;
        for (int t = t0q; t < t0q + 4; ++t) walk(t, last, std::integral_constant<int, 1>());
        const int end = last.value == 3 ? SB_TOK : t0q + 16;
#pragma unroll 2
        for (int t = t0q + 4; t < end; ++t) walk(t, last, std::integral_constant<int, 0>());
    };
    quarter(std::integral_constant<int, 0>());
    quarter(std::integral_constant<int, 1>());
    quarter(std::integral_constant<int, 2>());
    quarter(std::integral_constant<int, 3>());
    __syncthreads();
    if (tid < DKP) {   // q G, in place
        float gd = 1.f;
#pragma unroll 8
        for (int t = 0; t < SB_TOK; ++t) {
            if (MODE == SCAN_RWKV) { sq[t * DKP + tid] *= gd; gd *= sd[t * DKP + tid]; }
            else { gd *= sd[t * DKP + tid]; sq[t * DKP + tid] *= gd; }
        }
    }
    for (int u = tid; u < SB_TOK * 8; u += SB_THREADS) {
        const int t = u >> 3, o = u & 7;
        float x[8], z[8];
        load8(sk + t * SB_TOK, o * 8, SB_TOK, true, x);
        load8(sk + (SB_TOK + t) * SB_TOK, o * 8, SB_TOK, true, z);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] += z[j];
            bad |= !held(x[j]);
        }
        put_parts(p.a + bh * (3 * SB_TOK * 128) + sw128(t, o), SB_TOK * 128, x);
    }
    __syncthreads();
    for (int u = tid; u < SB_TOK * DKP / 8; u += SB_THREADS) {
        const int t = u / (DKP / 8), o = u % (DKP / 8);
        float x[8];
        load8(sq + t * DKP, o * 8, DKP, true, x);
        put_parts(p.q + (bh * KB + (o >> 3)) * (3 * SB_TOK * 128) + sw128(t, o & 7), SB_TOK * 128, x);
    }
    const int any = __syncthreads_or(bad);
    if (tid == 0) p.bad_in[bh] = any;
}

// 128 columns of V, transposed: a row of 64 tokens per column. Returns whether a value is one that the parts do not hold.
__device__ __forceinline__ bool put_values(const ScanArgs& a, uint8_t* sv, size_t row0, int nt, int h, int col0) {
    bool bad = false;
    float x[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int u = threadIdx.x + i * SB_THREADS, col = u & 127, o = u >> 7;
#pragma unroll
        for (int j = 0; j < 8; ++j) x[i][j] = o * 8 + j < nt && col0 + col < a.dv ? a.v[(row0 + o * 8 + j) * a.ldv + (size_t)h * a.dv + col0 + col] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int u = threadIdx.x + i * SB_THREADS;
#pragma unroll
        for (int j = 0; j < 8; ++j) bad |= !held(x[i][j]);
        put_parts(sv + sw128(u & 127, u >> 7), 128 * 128, x[i]);
    }
    return bad;
}
// D (+)= the six products of two operands of 64 columns in parts (A: 128 rows); issued by one warp
template <int N>
__device__ __forceinline__ void six_products(uint32_t tm, const uint8_t* sa, const uint8_t* sb, bool leader) {
    constexpr uint32_t idesc = make_idesc_bf16_f32(128, N);
    const uint64_t da = make_sw128_kmajor_desc(smem_u32(sa)), db = make_sw128_kmajor_desc(smem_u32(sb));
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
        const uint32_t pa = (SPLIT_A >> (2 * i)) & 3u, pb = (SPLIT_B >> (2 * i)) & 3u;
        if (leader)
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16(tm, da + (pa * (128 * 8) + 2 * k), db + (pb * (N * 8) + 2 * k), idesc, (i | k) != 0 ? 1u : 0u);
    }
}

template <int KB>
struct SbStates { static constexpr int V = 3 * 128 * 128, K = 3 * KB * 64 * 128, SMEM = V + K + 1024 + 64; };
template <int KB>
__global__ void __launch_bounds__(SB_THREADS, 2) sb_states_kernel(ScanArgs a, BlockScan p) {
    constexpr int DKP = KB * 64;
    using Cfg = SbStates<KB>;
    extern __shared__ uint8_t sb_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sb_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t *sv = smem, *sk = smem + Cfg::V;
    uint64_t *full = reinterpret_cast<uint64_t*>(smem + Cfg::V + Cfg::K), *done = full + 1;
    uint32_t* slot = reinterpret_cast<uint32_t*>(done + 1);
    const int ct = blockIdx.x, h = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t bh = (size_t)b * a.heads + h;
    if (threadIdx.x == 0) { mbar_init(full, 1); mbar_init(done, 1); fence_barrier_init(); }
    if (warp == 1) { tmem_alloc(slot, DKP); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *slot;
    pdl_trigger_small();
    pdl_wait();
    const SeqSeg sg = a.segs[0];
    const int t0 = p.t0 + b * SB_TOK, nt = min(SB_TOK, p.t0 + p.n - t0), col0 = ct * 128;
    if (threadIdx.x == 0) {
        mbar_arrive_expect_tx(full, Cfg::K);
        bulk_g2s(sk, p.k + bh * Cfg::K, Cfg::K, full);
    }
    const bool bad = put_values(a, sv, (size_t)sg.row0 + t0, nt, h, col0);
    fence_proxy_async();
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0) p.bad_v[bh * p.col_tiles + ct] = any;
    if (warp == 0) {
        const bool leader = elect_one();
        mbar_wait(full, 0);
        tc_fence_after();
        six_products<DKP>(tm, sv, sk, leader);
        if (leader) umma_commit(done);
        __syncwarp();
    }
    mbar_wait(done, 0);
    tc_fence_after();
    const int q = warp & 3, half = warp >> 2, col = col0 + q * 32 + lane;
    float* out = p.state + bh * a.dk * a.dv + col;
#pragma unroll
    for (int c = 0; c < DKP / 2; c += 32) {
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32(tm + (static_cast<uint32_t>(q * 32) << 16) + half * (DKP / 2) + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int key = half * (DKP / 2) + c + i;
            if (key < a.dk && col < a.dv) out[(size_t)key * a.dv] = __uint_as_float(v[i]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tm, DKP); }
}

// what a block adds to the state -> the state in front of it
__global__ void __launch_bounds__(256) sb_fold_kernel(ScanArgs a, BlockScan p) {
    pdl_enter();
    const SeqSeg sg = a.segs[0];
    const int h = blockIdx.y, per = a.dk * a.dv / 4, e = blockIdx.x * 256 + threadIdx.x;
    bool bad = false;
    if (e < per) {
        const int key = e * 4 / a.dv;
        const size_t head = (size_t)a.dk * a.dv, step = a.heads * head;
        float4* at = reinterpret_cast<float4*>(p.state + h * head) + e;
        const float* dec = p.decay + (size_t)h * a.dk + key;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (sg.pos0 > 0 || p.t0 > 0) s = reinterpret_cast<const float4*>(a.state + (size_t)sg.slot * step + h * head)[e];
        constexpr int U = 8;
        for (int b0 = 0; b0 < p.blocks; b0 += U) {
            float4 l[U];
            float d[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (b0 + u < p.blocks) {
                    l[u] = at[(size_t)(b0 + u) * (step / 4)];
                    d[u] = dec[(size_t)(b0 + u) * a.heads * a.dk];
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (b0 + u < p.blocks) {
                    at[(size_t)(b0 + u) * (step / 4)] = s;
                    bad |= !held(s.x) || !held(s.y) || !held(s.z) || !held(s.w);
                    s.x = fmaf(d[u], s.x, l[u].x); s.y = fmaf(d[u], s.y, l[u].y); s.z = fmaf(d[u], s.z, l[u].z); s.w = fmaf(d[u], s.w, l[u].w);
                }
        }
        bad |= !held(s.x) || !held(s.y) || !held(s.z) || !held(s.w);
        reinterpret_cast<float4*>(p.last + h * head)[e] = s;
    }
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0) p.bad_state[h * p.fold_ctas + blockIdx.x] = any;
}

constexpr int SB_OUT_A = 3 * 128 * 128, SB_OUT_B = 3 * SB_TOK * 128, SB_OUT_SMEM = SB_OUT_A + SB_OUT_B + 1024 + 64;
template <int KB>
__global__ void __launch_bounds__(SB_THREADS, 2) sb_output_kernel(ScanArgs a, BlockScan p) {
    extern __shared__ uint8_t sb_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sb_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t *sa = smem, *sb = smem + SB_OUT_A;
    uint64_t *full = reinterpret_cast<uint64_t*>(smem + SB_OUT_A + SB_OUT_B), *done = full + 1;
    uint32_t* slot = reinterpret_cast<uint32_t*>(done + 1);
    const int ct = blockIdx.x, h = blockIdx.y, b = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t bh = (size_t)b * a.heads + h;
    if (threadIdx.x == 0) { mbar_init(full, 1); mbar_init(done, 1); fence_barrier_init(); }
    if (warp == 1) { tmem_alloc(slot, SB_TOK); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = *slot;
    pdl_trigger_small();
    pdl_wait();
    const SeqSeg sg = a.segs[0];
    const int t0 = p.t0 + b * SB_TOK, nt = min(SB_TOK, p.t0 + p.n - t0), col0 = ct * 128;
    const int q = warp & 3, half = warp >> 2;
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    // what a stage holds of its first operand: 128 columns, transposed, of the state in front of the block (64 keys a stage) or of V (its tokens)
    float x[4][8];
    const auto load = [&](int blk) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int u = threadIdx.x + i * SB_THREADS, col = u & 127, at = (u >> 7) * 8;
            const float* src = blk < KB ? p.state + (bh * a.dk + blk * 64 + at) * a.dv + col0 + col : a.v + ((size_t)sg.row0 + t0 + at) * a.ldv + (size_t)h * a.dv + col0 + col;
            const int64_t ld = blk < KB ? a.dv : a.ldv;
            const int n = col0 + col >= a.dv ? 0 : blk < KB ? a.dk - blk * 64 - at : nt - at;
#pragma unroll
            for (int j = 0; j < 8; ++j) x[i][j] = j < n ? src[j * ld] : 0.f;
        }
    };
    load(0);
#pragma unroll 1
    for (int blk = 0; blk <= KB; ++blk) {
        if (threadIdx.x == 0) {   // (the products that read it last are done)
            mbar_arrive_expect_tx(full, SB_OUT_B);
            bulk_g2s(sb, blk < KB ? p.q + (bh * KB + blk) * SB_OUT_B : p.a + bh * SB_OUT_B, SB_OUT_B, full);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int u = threadIdx.x + i * SB_THREADS;
            put_parts(sa + sw128(u & 127, u >> 7), 128 * 128, x[i]);
        }
        fence_proxy_async();
        __syncthreads();   // (also: the accumulator of the block before has been read)
        if (warp == 0) {
            const bool leader = elect_one();
            mbar_wait(full, blk & 1);
            tc_fence_after();
            six_products<SB_TOK>(tm, sa, sb, leader);
            if (leader) umma_commit(done);
            __syncwarp();
        }
        if (blk < KB) load(blk + 1);   // on its way while the products run
        mbar_wait(done, blk & 1);
        tc_fence_after();
        uint32_t v[32];
        __syncwarp();
        tmem_ld_32x32(tm + (static_cast<uint32_t>(q * 32) << 16) + half * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[i] += __uint_as_float(v[i]);
        tc_fence_before();
    }
    const int col = col0 + q * 32 + lane;
    bool bad = false;
    if (col < a.dv) {
        const size_t row = (size_t)sg.row0 + t0 + half * 32;
        float* y = a.y + row * a.ldy + (size_t)h * a.dv + col;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (half * 32 + i < nt) {
                bad |= !held(acc[i]);
                y[(size_t)i * a.ldy] = acc[i];
            }
    }
    const int any = __syncthreads_or(bad);
    if (threadIdx.x == 0) p.bad_out[bh * p.col_tiles + ct] = any;
    tc_fence_before();
    __syncthreads();
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tm, SB_TOK); }
}

template <int MODE, int KB>
int launch_blocks(const ScanArgs& a, const BlockScan& p, cudaStream_t st) {
    constexpr size_t prep = (size_t)(2 * SB_TOK * KB * 64 + 2 * SB_TOK * SB_TOK) * sizeof(float);   // (64 tokens of up to 128 keys, then two halves of A)
    B2_CUDA_CHECK(cudaFuncSetAttribute(sb_prepare_kernel<MODE, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep));
    B2_CUDA_CHECK(cudaFuncSetAttribute(sb_states_kernel<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, SbStates<KB>::SMEM));
    B2_CUDA_CHECK(cudaFuncSetAttribute(sb_output_kernel<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, SB_OUT_SMEM));
    const dim3 tiles(p.col_tiles, a.heads, p.blocks);
    launch_pdl(sb_prepare_kernel<MODE, KB>, dim3(a.heads, p.blocks), dim3(SB_THREADS), prep, st, a, p);
    B2_LAUNCH_CHECK();
    launch_pdl(sb_states_kernel<KB>, tiles, dim3(SB_THREADS), SbStates<KB>::SMEM, st, a, p);
    B2_LAUNCH_CHECK();
    launch_pdl(sb_fold_kernel, dim3(p.fold_ctas, a.heads), dim3(256), 0, st, a, p);
    B2_LAUNCH_CHECK();
    launch_pdl(sb_output_kernel<KB>, tiles, dim3(SB_THREADS), SB_OUT_SMEM, st, a, p);
    B2_LAUNCH_CHECK();
    return 0;
}

size_t whole(size_t bytes) { return (bytes + 127) / 128 * 128; }
struct SbSizes {   // bytes
    int KB, ct, fold;
    size_t q, k, a, decay, state, flags, last;
    SbSizes(int heads, int dk, int dv, int blocks) {
        const size_t bh = (size_t)blocks * heads;
        KB = (dk + 63) / 64; ct = (dv + 127) / 128; fold = (dk * dv / 4 + 255) / 256;
        q = bh * KB * SB_OUT_B; k = q; a = bh * SB_OUT_B;
        decay = whole(bh * dk * 4); state = whole(bh * dk * dv * 4); last = whole((size_t)heads * dk * dv * 4);
        flags = whole((bh * (1 + 2 * ct) + (size_t)heads * fold) * 4);
    }
    size_t total() const { return q + k + a + decay + state + last + flags + 128; }
};
}  // namespace

size_t scan_blocks_bytes(int heads, int dk, int dv, int blocks) { return SbSizes(heads, dk, dv, blocks).total(); }

bool scan_blocks_fit(const ScanArgs& a) {
    // Five launches take some 45 us whatever the length, so short prompts stay with the walk. us, walk / blocks: 8 heads of 128 x 256 192 tokens 51 / 50, 384
    // 75 / 53, 1024 123 / 64, 2048 205 / 108; 8 of 128 x 128 (HGRN2) 256 tokens 55 / 58, 384 60 / 56, 1024 98 / 65; 16 of 64 x 64 256 tokens 41 / 42, 384 46 /
    // 48, 512 52 / 48, 2048 120 / 85; RWKV 16 of 64 384 tokens 48 / 45, 1024 78 / 49, 32 of 64 2048 tokens 173 / 142. One decay per token (SSD) walks
    // cheaper and gains nothing: 32 heads of 128 x 64 600 tokens 83 / 81, 2048 205 / 247.
    if (a.mode == SCAN_SSD || a.nseg != 1 || a.rows < (a.dk > 64 ? 320 : 448) || a.chunk_scratch == nullptr || a.dk > 128 || a.dk % 4 != 0 || a.dv % 4 != 0) return false;
    const auto off = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; };
    if (off(a.q) || a.ldq % 4 != 0 || (a.mode != SCAN_HGRN2 && (off(a.k) || a.ldk % 4 != 0)) || off(a.decay_in) || a.ldd % 4 != 0 || off(a.state)) return false;
    return scan_blocks_bytes(a.heads, a.dk, a.dv, std::min((a.rows + SB_TOK - 1) / SB_TOK, SB_MIN_PIECE)) <= a.chunk_floats * 4;
}

int scan_blocks_plan(const ScanArgs& a, int t0, BlockScan* out) {
    BlockScan p;
    int blocks = (a.rows - t0 + SB_TOK - 1) / SB_TOK;
    while (blocks > 1 && scan_blocks_bytes(a.heads, a.dk, a.dv, blocks) > a.chunk_floats * 4) --blocks;
    const SbSizes z(a.heads, a.dk, a.dv, blocks);
    B2_CHECK_ARG(z.total() <= a.chunk_floats * 4, "scan_blocks: no scratch for a block");
    p.t0 = t0; p.n = std::min(a.rows - t0, blocks * SB_TOK); p.blocks = blocks; p.key_blocks = z.KB; p.col_tiles = z.ct; p.fold_ctas = z.fold;
    uint8_t* at = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(a.chunk_scratch) + 127) & ~static_cast<uintptr_t>(127));
    p.q = at; at += z.q;
    p.k = at; at += z.k;
    p.a = at; at += z.a;
    p.decay = reinterpret_cast<float*>(at); at += z.decay;
    p.state = reinterpret_cast<float*>(at); at += z.state;
    p.last = reinterpret_cast<float*>(at); at += z.last;
    const size_t bh = (size_t)blocks * a.heads;
    p.bad_in = reinterpret_cast<int*>(at);
    p.bad_v = p.bad_in + bh;
    p.bad_out = p.bad_v + bh * z.ct;
    p.bad_state = p.bad_out + bh * z.ct;
    *out = p;
    return 0;
}

int scan_blocks_f32(const ScanArgs& a, const BlockScan& p, cudaStream_t st) {
    const bool two = p.key_blocks == 2;
    if (a.mode == SCAN_RWKV) return two ? launch_blocks<SCAN_RWKV, 2>(a, p, st) : launch_blocks<SCAN_RWKV, 1>(a, p, st);
    if (a.mode == SCAN_HGRN2) return two ? launch_blocks<SCAN_HGRN2, 2>(a, p, st) : launch_blocks<SCAN_HGRN2, 1>(a, p, st);
    return two ? launch_blocks<SCAN_GLA, 2>(a, p, st) : launch_blocks<SCAN_GLA, 1>(a, p, st);
}

}  // namespace b2
