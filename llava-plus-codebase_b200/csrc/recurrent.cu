// Recurrent mixers of the layer-list decoders: causal depthwise convolution with a carried tail, RWKV token shift, and the
// linear recurrence with a diagonal decay over a per-head [key, value] state (state-space, RWKV and HGRN2 forms). One code path
// serves a portion of a prompt (n rows of one slot) and a decode step (one row of each of B slots): the rows come as
// segments (kernels.h, SeqSeg). State, decays, step sizes and sums are fp32; a segment whose pos0 is 0 starts from zero
// state whatever its slot held before, so a slot that is handed to a new request needs no clearing.
#include <algorithm>

#include "scan.cuh"

namespace b2 {
namespace {

// ---- causal depthwise convolution + SiLU -----------------------------------------------------------------------------------
// One thread per (channel, tile of CONV_TILE tokens): it primes its window from the inputs in front of the tile (rows of this
// call, or the carried tail for positions before the call) and walks the tile. The compute kernel only READS the tail; a
// second small kernel replaces it afterwards, so tiles never race with the update.
constexpr int CONV_MAX_TAPS = 16, CONV_TILE = 32;
template <int FLAGS>   // CONV_SILU | CONV_ADD_INPUT; own_tail: every segment is ONE tile, whose thread replaces the carried inputs itself
__global__ void __launch_bounds__(128) causal_conv_kernel(const float* in, int64_t ld_in, const float* __restrict__ w,
                                                          const float* __restrict__ bias, float* __restrict__ tail,
                                                          float* __restrict__ out, int64_t ld_out, int C, int taps,
                                                          const SeqSeg* segs, int own_tail) {
    pdl_enter();
    const SeqSeg sg = segs[blockIdx.z];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int tt0 = blockIdx.y * CONV_TILE;
    if (c >= C || tt0 >= sg.n) return;
    // Window and taps are kept right-aligned in arrays of CONV_MAX_TAPS (all indices static): entry CONV_MAX_TAPS-1 is the
    // current token, the unused leading entries carry zero weights.
    float wt[CONV_MAX_TAPS], win[CONV_MAX_TAPS];
    const float* tl = tail + (size_t)sg.slot * (taps - 1) * C + c;
    const float* ip = in + (size_t)sg.row0 * ld_in + c;
#pragma unroll
    for (int jp = 0; jp < CONV_MAX_TAPS; ++jp) {
        const int tj = jp - (CONV_MAX_TAPS - taps);
        wt[jp] = tj >= 0 ? w[(size_t)c * taps + tj] : 0.f;
        // primed one step early (the loop shifts before it appends): entry jp holds the input of token tt0 - (CONV_MAX_TAPS - jp)
        const int t = tt0 - (CONV_MAX_TAPS - jp);
        float v = 0.f;
        if (jp >= CONV_MAX_TAPS - (taps - 1)) {  // the taps-1 tokens in front of the tile
            if (t >= 0) v = ip[(size_t)t * ld_in];
            else if (sg.pos0 > 0) v = tl[(size_t)(t + (taps - 1)) * C];
        }
        win[jp] = v;
    }
    const float b = bias != nullptr ? bias[c] : 0.f;
    float* op = out + (size_t)sg.row0 * ld_out + c;
    const int t_end = min(sg.n, tt0 + CONV_TILE);
    for (int t0 = tt0; t0 < t_end; t0 += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = t0 + u < t_end ? ip[(size_t)(t0 + u) * ld_in] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (t0 + u < t_end) {
#pragma unroll
                for (int jp = 0; jp < CONV_MAX_TAPS - 1; ++jp) win[jp] = win[jp + 1];
                win[CONV_MAX_TAPS - 1] = v[u];
                float acc = b;
#pragma unroll
                for (int jp = 0; jp < CONV_MAX_TAPS; ++jp) acc = fmaf(wt[jp], win[jp], acc);
                if (FLAGS & CONV_ADD_INPUT) acc += v[u];
                op[(size_t)(t0 + u) * ld_out] = (FLAGS & CONV_SILU) ? silu_f(acc) : acc;
            }
        }
    }
    if (own_tail && taps > 1) {   // the window now ends with the segment's last input: its last taps - 1 entries are the new carried inputs
        float* tw = tail + (size_t)sg.slot * (taps - 1) * C + c;
#pragma unroll
        for (int jp = 0; jp < CONV_MAX_TAPS; ++jp) {
            const int j = jp - (CONV_MAX_TAPS - (taps - 1));
            if (j >= 0) tw[(size_t)j * C] = win[jp];
        }
    }
}
// tail[j] := input of token n - (taps-1) + j of the segment; tokens before the call come from the old tail (or zero)
__global__ void __launch_bounds__(128) causal_conv_tail_kernel(const float* in, int64_t ld_in, float* __restrict__ tail, int C,
                                                               int taps, const SeqSeg* segs) {
    pdl_enter();
    const SeqSeg sg = segs[blockIdx.y];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C || sg.n <= 0) return;
    float* tl = tail + (size_t)sg.slot * (taps - 1) * C + c;
    float nv[CONV_MAX_TAPS];
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j) {
        nv[j] = 0.f;
        if (j < taps - 1) {
            const int t = sg.n - (taps - 1) + j;
            if (t >= 0) nv[j] = in[(size_t)(sg.row0 + t) * ld_in + c];
            else if (sg.pos0 > 0) nv[j] = tl[(size_t)(t + (taps - 1)) * C];
        }
    }
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j)
        if (j < taps - 1) tl[(size_t)j * C] = nv[j];
}

// ---- token shift: out[s][t] = x[t] + (x[t-1] - x[t]) * mu[s]; x[-1] of a call is the carried row (zero at a sequence start) ---
constexpr int SHIFT_MAX_MIX = 8, SHIFT_TILE = 8;
__global__ void __launch_bounds__(128) token_shift_mix_kernel(const float* x, const float* __restrict__ mu,
                                                              const float* prev, float* __restrict__ out, int64_t out_stride,
                                                              int cols, int n_mix, const SeqSeg* segs) {
    pdl_enter();
    const SeqSeg sg = segs[blockIdx.z];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int t0 = blockIdx.y * SHIFT_TILE;
    if (c >= cols || t0 >= sg.n) return;
    float m[SHIFT_MAX_MIX];
#pragma unroll
    for (int s = 0; s < SHIFT_MAX_MIX; ++s) m[s] = s < n_mix ? mu[(size_t)s * cols + c] : 0.f;
    float v[SHIFT_TILE + 1];
    v[0] = t0 > 0 ? x[(size_t)(sg.row0 + t0 - 1) * cols + c] : (sg.pos0 > 0 ? prev[(size_t)sg.slot * cols + c] : 0.f);
#pragma unroll
    for (int u = 0; u < SHIFT_TILE; ++u) v[u + 1] = t0 + u < sg.n ? x[(size_t)(sg.row0 + t0 + u) * cols + c] : 0.f;
#pragma unroll
    for (int u = 0; u < SHIFT_TILE; ++u) {
        if (t0 + u < sg.n) {
            const float d = v[u] - v[u + 1];
#pragma unroll
            for (int s = 0; s < SHIFT_MAX_MIX; ++s)
                if (s < n_mix) out[(size_t)s * out_stride + (size_t)(sg.row0 + t0 + u) * cols + c] = fmaf(d, m[s], v[u + 1]);
        }
    }
}
__global__ void __launch_bounds__(128) token_shift_carry_kernel(const float* x, float* __restrict__ prev, int cols,
                                                                const SeqSeg* segs) {
    pdl_enter();
    const SeqSeg sg = segs[blockIdx.y];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < cols && sg.n > 0) prev[(size_t)sg.slot * cols + c] = x[(size_t)(sg.row0 + sg.n - 1) * cols + c];
}

// ---- linear recurrence ------------------------------------------------------------------------------------------------
// S <- D S + k v^T, y = S^T q per head, D diagonal (one decay per key, or one per token), S and all sums fp32.
// A warp holds 64 keys x 16 columns of a head's state in registers, a lane 8 keys x 4 columns, so that a token costs a lane seven 16-byte reads
// of shared memory for its 96 multiply-adds; a CTA takes all keys (KW warps) of 64 columns (4 warps). Tokens come in tiles of SC_TT through
// two buffers (cp.async), the raw gates are turned into (q, k, decay) once per tile, the lanes' and warps' shares of y meet per token by
// shuffles and per tile in shared memory.
// A long prompt has few (head, column) CTAs and a long chain of tokens, so it is cut into chunks that run side by side, exactly (no decay is
// divided by): a first launch walks every chunk from an empty state (the first one from the slot's state, with its outputs) and leaves the
// chunk's final state and the product of its decays per key; a second launch starts each further chunk from what those fold to, S_c = P_c S_(c-1)
// + L_c, and writes its outputs. The chain is then 2 / C of the tokens for 5/3 of the arithmetic.
// Long prompts with a decay per key run in blocks on the tensor cores instead (scan_blocks.cu).
// 1900 tokens, 8 heads of 128 x 256 (gated linear attention): 625 -> 191 us (two walks of 90 us, 11 us for the gates beforehand; before, 8 keys x
// one column per thread and one chain). Issue slots bound a walk (74 % of them taken in the first, 58 % in the one that
// writes; with the gates' arithmetic in it 291 us for both, hence scan_prepare_kernel), then the multiply-add pipe. 600 tokens, 32 heads of 128 x 64 (state space): 152 -> 84 us, 16 heads of 64 x 64 (RWKV) 128 -> 58.
constexpr int SC_TT = 16, SC_COLS = 64, SC_MAX_CHUNKS = 10;

struct ScanPlan {
    int chunks = 1, len = 0;       // chunks of `len` tokens (1: the whole segment, whatever its length)
    int z0 = 0;                    // chunk of blockIdx.z == 0
    int second = 0;                // the launch that starts from folded states
    int prepared = 0;              // scan_prepare_kernel has made (q, decay) of the raw gates
    float *final_state = nullptr, *decays = nullptr;   // [chunk][head][dk][dv], [chunk][head][dk]
};

__device__ __forceinline__ void scan_cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void scan_cp4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// The gates' arithmetic in place over a long prompt's rows (workspaces of the call), where every column block of both launches would redo it
template <int MODE>
__global__ void __launch_bounds__(256) scan_prepare_kernel(ScanArgs a) {
    pdl_enter();
    const int c = blockIdx.x * 256 + threadIdx.x;
    const size_t r = (size_t)a.segs[0].row0 + blockIdx.y;
    if (c >= a.heads * a.dk) return;
    float* d = const_cast<float*>(a.decay_in) + r * a.ldd + c;
    *d = scan_decay<MODE>(a, c, *d);
    if (MODE != SCAN_RWKV) {
        float* q = const_cast<float*>(a.q) + r * a.ldq + c;
        *q = scan_query<MODE>(a, *q);
    }
}

// KW: warps over the keys (64 each); V16: every operand row is 16-byte aligned with sizes in whole fours. AFTER: behind scan_blocks_f32, whose tokens
// are walked only for heads that the products could not do; the other heads' state is put in its place.
template <int MODE, int KW, bool V16, bool AFTER>
__device__ __forceinline__ void linear_scan_body(const ScanArgs& a, const ScanPlan& p, const BlockScan& bs) {
    pdl_enter();
    constexpr int DKP = KW * 64, NTHR = KW * 128;
    constexpr bool PER_KEY = MODE != SCAN_SSD, HAS_K = MODE != SCAN_HGRN2;
    extern __shared__ __align__(16) float sm[];
    float* sQ = sm;                                  // [2][TT][DKP]
    float* sD = sQ + 2 * SC_TT * DKP;                // [2][TT][DKP] decays per key (SSD: [2][2][TT] step sizes, decays)
    float* sK = sD + 2 * SC_TT * DKP;                // [2][TT][DKP]
    float* sV = sK + 2 * SC_TT * DKP;                // [2][TT][COLS]
    float* sY = sV + 2 * SC_TT * SC_COLS;            // [KW][TT][COLS]
    const int chunk = p.chunks > 1 ? p.z0 + (int)blockIdx.z : 0;
    const SeqSeg sg = a.segs[p.chunks > 1 ? 0 : blockIdx.z];
    const int t_end = AFTER ? bs.t0 + bs.n : sg.n;
    const int t_lo = AFTER ? bs.t0 : chunk * p.len, t_hi = p.chunks > 1 && chunk + 1 < p.chunks ? min(sg.n, t_lo + p.len) : t_end;
    if (t_lo >= t_hi) return;
    const bool outputs = p.chunks == 1 || p.second != 0 || chunk == 0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, kw = warp % KW, cw = warp / KW, kg = lane & 7, cg = lane >> 3;
    const int h = blockIdx.y, col0 = blockIdx.x * SC_COLS, dk = a.dk, dv = a.dv;
    const int g = MODE == SCAN_SSD ? h / (a.heads / a.groups) : h;
    // a lane's keys: four consecutive ones out of each half of its warp's 64, so that eight key groups read 128 adjoining bytes
    const int key0 = kw * 64 + kg * 4, c0 = cw * 16 + cg * 4;   // keys key0 + (0..3) and key0 + 32 + (0..3); columns col0 + c0 + (0..3)
    auto key_of = [&](int i) { return key0 + (i >> 2) * 32 + (i & 3); };
    const float* qg = a.q + (size_t)sg.row0 * a.ldq + (size_t)g * dk;
    const float* kgm = HAS_K ? a.k + (size_t)sg.row0 * a.ldk + (size_t)g * dk : nullptr;
    const float* dg = a.decay_in + (size_t)sg.row0 * a.ldd + (PER_KEY ? (size_t)h * dk : (size_t)h);
    const float* vg = a.v + (size_t)sg.row0 * a.ldv + (size_t)h * dv + col0;
    const int ncol = min(SC_COLS, dv - col0);
    const size_t head_state = ((size_t)h * dk) * dv, all_state = (size_t)a.heads * dk * dv;
    if (AFTER) {
        int bad = 0;
        for (int b = tid; b < bs.blocks; b += NTHR) {
            const size_t bh = (size_t)b * a.heads + h;
            bad |= bs.bad_in[bh];
            for (int c = 0; c < bs.col_tiles; ++c) bad |= bs.bad_v[bh * bs.col_tiles + c] | bs.bad_out[bh * bs.col_tiles + c];
        }
        for (int i = tid; i < bs.fold_ctas; i += NTHR) bad |= bs.bad_state[h * bs.fold_ctas + i];
        if (!__syncthreads_or(bad)) {   // (whole fours: scan_blocks_fit)
            for (int e = tid; e < dk * (ncol >> 2); e += NTHR) {
                const size_t at = head_state + (size_t)(e / (ncol >> 2)) * dv + col0 + e % (ncol >> 2) * 4;
                *reinterpret_cast<float4*>(a.state + (size_t)sg.slot * all_state + at) = *reinterpret_cast<const float4*>(bs.last + at);
            }
            return;
        }
    }

    float S[8][4], pd[8];
    auto load_state = [&](const float* st, bool fold, const float* dec) {   // S = st, or S = dec S + st
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int key = key_of(i);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (key < dk) {
                const float* r = st + (size_t)key * dv + col0 + c0;
                if (V16 && c0 + 4 <= ncol) {
                    const float4 f = *reinterpret_cast<const float4*>(r);
                    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (c0 + j < ncol) v[j] = r[j];
                }
            }
            const float d = fold && key < dk ? dec[key] : 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) S[i][j] = fold ? fmaf(d, S[i][j], v[j]) : v[j];
        }
    };
    auto store_state = [&](float* st) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int key = key_of(i);
            if (key >= dk) continue;
            float* r = st + (size_t)key * dv + col0 + c0;
            if (V16 && c0 + 4 <= ncol) {
                *reinterpret_cast<float4*>(r) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) if (c0 + j < ncol) r[j] = S[i][j];
            }
        }
    };
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        pd[i] = 1.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) S[i][j] = 0.f;
    }
    auto fetch = [&](int t0, int buf) {   // raw rows of a tile; entries past dk / the last column are zeroed once, below
        const int nt = min(SC_TT, t_hi - t0);
        float *q = sQ + buf * SC_TT * DKP, *k = sK + buf * SC_TT * DKP, *d = sD + buf * SC_TT * DKP, *v = sV + buf * SC_TT * SC_COLS;
        if (V16) {
            const int n4 = dk >> 2, c4 = ncol >> 2;
            for (int e = tid; e < nt * n4; e += NTHR) {
                const int t = e / n4, o = (e - t * n4) * 4;
                if (outputs) scan_cp16(q + t * DKP + o, qg + (size_t)(t0 + t) * a.ldq + o);
                if (HAS_K) scan_cp16(k + t * DKP + o, kgm + (size_t)(t0 + t) * a.ldk + o);
                if (PER_KEY) scan_cp16(d + t * DKP + o, dg + (size_t)(t0 + t) * a.ldd + o);
            }
            for (int e = tid; e < nt * c4; e += NTHR) {
                const int t = e / c4, o = (e - t * c4) * 4;
                scan_cp16(v + t * SC_COLS + o, vg + (size_t)(t0 + t) * a.ldv + o);
            }
        } else {
            for (int e = tid; e < nt * dk; e += NTHR) {
                const int t = e / dk, o = e - t * dk;
                if (outputs) scan_cp4(q + t * DKP + o, qg + (size_t)(t0 + t) * a.ldq + o);
                if (HAS_K) scan_cp4(k + t * DKP + o, kgm + (size_t)(t0 + t) * a.ldk + o);
                if (PER_KEY) scan_cp4(d + t * DKP + o, dg + (size_t)(t0 + t) * a.ldd + o);
            }
            for (int e = tid; e < nt * ncol; e += NTHR) {
                const int t = e / ncol, o = e - t * ncol;
                scan_cp4(v + t * SC_COLS + o, vg + (size_t)(t0 + t) * a.ldv + o);
            }
        }
        if (!PER_KEY && tid < nt) scan_cp4(d + tid, dg + (size_t)(t0 + tid) * a.ldd);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(t_lo, 0);
    if (p.second != 0) {
        load_state(p.final_state + head_state, false, nullptr);
        for (int c = 1; c < chunk; ++c) load_state(p.final_state + (size_t)c * all_state + head_state, true, p.decays + ((size_t)c * a.heads + h) * dk);
    } else if (chunk == 0 && (sg.pos0 > 0 || (AFTER && t_lo > 0))) {
        load_state(a.state + (size_t)sg.slot * all_state + head_state, false, nullptr);
    }
    float bon[8];
    if (MODE == SCAN_RWKV) {
#pragma unroll
        for (int i = 0; i < 8; ++i) bon[i] = key_of(i) < dk ? a.bonus[(size_t)h * dk + key_of(i)] : 0.f;
    }
    float neg_a = 0.f, dtb = 0.f, skip = 0.f;
    if (MODE == SCAN_SSD) { neg_a = -expf(a.a_log[h]); dtb = a.dt_bias[h]; skip = a.skip[h]; }
    // entries that no copy writes: keys past dk (queries and keys 0), columns past the last one
    for (int e = tid; e < 2 * SC_TT * (DKP - dk); e += NTHR) {
        const int at = (e / (DKP - dk)) * DKP + dk + e % (DKP - dk);
        sQ[at] = 0.f; sK[at] = 0.f;
        if (PER_KEY) sD[at] = 0.f;
    }
    for (int e = tid; e < 2 * SC_TT * (SC_COLS - ncol); e += NTHR) sV[(e / (SC_COLS - ncol)) * SC_COLS + ncol + e % (SC_COLS - ncol)] = 0.f;

    int buf = 0;
    for (int t0 = t_lo; t0 < t_hi; t0 += SC_TT, buf ^= 1) {
        const int nt = min(SC_TT, t_hi - t0);
        float *q = sQ + buf * SC_TT * DKP, *k = sK + buf * SC_TT * DKP, *d = sD + buf * SC_TT * DKP, *v = sV + buf * SC_TT * SC_COLS;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (t0 + SC_TT < t_hi) fetch(t0 + SC_TT, buf ^ 1);   // (the other buffer was read before the barrier above)
        // the raw gates -> (q, k, decay)
        if (MODE == SCAN_SSD) {
            if (tid < nt) {   // the step size multiplies the value (dt B x^T = B (dt x)^T)
                const float dt = softplus_f(d[tid] + dtb);
                d[tid] = dt;
                d[SC_TT + tid] = expf(neg_a * dt);
            }
        } else if (p.prepared == 0 || MODE == SCAN_HGRN2) {
            for (int at = tid; at < nt * DKP; at += NTHR) {
                const int key = at % DKP;
                if (key >= dk) continue;
                float f = d[at];
                if (p.prepared == 0) {
                    d[at] = f = scan_decay<MODE>(a, h * dk + key, f);
                    if (outputs && MODE != SCAN_RWKV) q[at] = scan_query<MODE>(a, q[at]);
                }
                if (MODE == SCAN_HGRN2) k[at] = 1.f - f;
            }
        }
        if (MODE == SCAN_SSD || MODE == SCAN_HGRN2 || p.prepared == 0) __syncthreads();
        if (outputs) {
#pragma unroll 2
            for (int t = 0; t < nt; ++t) {
                float qv[8], kv[8], dvv[8], vv[4], y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float4 q4 = *reinterpret_cast<const float4*>(q + t * DKP + key0 + 32 * i), k4 = *reinterpret_cast<const float4*>(k + t * DKP + key0 + 32 * i);
                    qv[4 * i] = q4.x; qv[4 * i + 1] = q4.y; qv[4 * i + 2] = q4.z; qv[4 * i + 3] = q4.w;
                    kv[4 * i] = k4.x; kv[4 * i + 1] = k4.y; kv[4 * i + 2] = k4.z; kv[4 * i + 3] = k4.w;
                    if (PER_KEY) {
                        const float4 d4 = *reinterpret_cast<const float4*>(d + t * DKP + key0 + 32 * i);
                        dvv[4 * i] = d4.x; dvv[4 * i + 1] = d4.y; dvv[4 * i + 2] = d4.z; dvv[4 * i + 3] = d4.w;
                    }
                }
                const float4 v4 = *reinterpret_cast<const float4*>(v + t * SC_COLS + c0);
                const float dt = PER_KEY ? 1.f : d[t], dec = PER_KEY ? 0.f : d[SC_TT + t];
                vv[0] = v4.x * dt; vv[1] = v4.y * dt; vv[2] = v4.z * dt; vv[3] = v4.w * dt;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float de = PER_KEY ? dvv[i] : dec;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float x = kv[i] * vv[j];
                        if (MODE == SCAN_RWKV) {
                            y[j] = fmaf(qv[i], fmaf(bon[i], x, S[i][j]), y[j]);
                            S[i][j] = fmaf(de, S[i][j], x);
                        } else {
                            S[i][j] = fmaf(de, S[i][j], x);
                            y[j] = fmaf(qv[i], S[i][j], y[j]);
                        }
                    }
                }
                // sum over the eight key groups; lane kg ends up with column 2 (kg & 1) + (kg >> 1 & 1)
                const bool b0 = kg & 1, b1 = kg & 2;
                float u0 = b0 ? y[2] : y[0], u1 = b0 ? y[3] : y[1];
                u0 += __shfl_xor_sync(0xffffffffu, b0 ? y[0] : y[2], 1);
                u1 += __shfl_xor_sync(0xffffffffu, b0 ? y[1] : y[3], 1);
                float w0 = b1 ? u1 : u0;
                w0 += __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
                w0 += __shfl_xor_sync(0xffffffffu, w0, 4);
                if (kg < 4) sY[(kw * SC_TT + t) * SC_COLS + c0 + 2 * (kg & 1) + (kg >> 1)] = w0;
            }
        } else {
#pragma unroll 2
            for (int t = 0; t < nt; ++t) {
                float kv[8], dvv[8], vv[4];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float4 k4 = *reinterpret_cast<const float4*>(k + t * DKP + key0 + 32 * i);
                    kv[4 * i] = k4.x; kv[4 * i + 1] = k4.y; kv[4 * i + 2] = k4.z; kv[4 * i + 3] = k4.w;
                    if (PER_KEY) {
                        const float4 d4 = *reinterpret_cast<const float4*>(d + t * DKP + key0 + 32 * i);
                        dvv[4 * i] = d4.x; dvv[4 * i + 1] = d4.y; dvv[4 * i + 2] = d4.z; dvv[4 * i + 3] = d4.w;
                    }
                }
                const float4 v4 = *reinterpret_cast<const float4*>(v + t * SC_COLS + c0);
                const float dt = PER_KEY ? 1.f : d[t], dec = PER_KEY ? 0.f : d[SC_TT + t];
                vv[0] = v4.x * dt; vv[1] = v4.y * dt; vv[2] = v4.z * dt; vv[3] = v4.w * dt;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float de = PER_KEY ? dvv[i] : dec;
                    pd[i] *= de;
#pragma unroll
                    for (int j = 0; j < 4; ++j) S[i][j] = fmaf(de, S[i][j], kv[i] * vv[j]);
                }
            }
        }
        if (outputs) {
            __syncthreads();
            for (int e = tid; e < nt * SC_COLS; e += NTHR) {
                const int t = e / SC_COLS, c = e % SC_COLS;
                if (c >= ncol) continue;
                float y = sY[e];
#pragma unroll
                for (int w = 1; w < KW; ++w) y += sY[w * SC_TT * SC_COLS + e];
                if (MODE == SCAN_SSD) y = fmaf(skip, v[t * SC_COLS + c], y);
                a.y[(size_t)(sg.row0 + t0 + t) * a.ldy + (size_t)h * dv + col0 + c] = y;
            }
        }
    }
    if (p.chunks == 1 || chunk == p.chunks - 1) {
        store_state(a.state + (size_t)sg.slot * all_state + head_state);
    } else if (p.second == 0) {
        store_state(p.final_state + (size_t)chunk * all_state + head_state);
        if (blockIdx.x == 0 && cw == 0 && cg == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (key_of(i) < dk) p.decays[((size_t)chunk * a.heads + h) * dk + key_of(i)] = pd[i];
        }
    }
}
template <int MODE, int KW, bool V16>
__global__ void __launch_bounds__(KW * 128, KW == 4 ? 1 : 2) linear_scan_kernel(ScanArgs a, ScanPlan p) {
    linear_scan_body<MODE, KW, V16, false>(a, p, BlockScan());
}
template <int MODE, int KW>
__global__ void __launch_bounds__(KW * 128, 2) linear_scan_after_kernel(ScanArgs a, BlockScan blocks) {
    linear_scan_body<MODE, KW, true, true>(a, ScanPlan(), blocks);
}
}  // namespace

int causal_conv_silu_f32(const float* in, int64_t ld_in, const float* w, const float* bias, float* tail, float* out, int64_t ld_out, int C,
                         int taps, const SeqSeg* segs, int nseg, int max_n, cudaStream_t st) {
    B2_CHECK_ARG(bias != nullptr, "causal_conv_silu: null bias");
    return causal_conv_f32(in, ld_in, w, bias, tail, out, ld_out, C, taps, CONV_SILU, segs, nseg, max_n, st);
}

int causal_conv_f32(const float* in, int64_t ld_in, const float* w, const float* bias, float* tail, float* out, int64_t ld_out, int C, int taps,
                    int flags, const SeqSeg* segs, int nseg, int max_n, cudaStream_t st) {
    B2_CHECK_ARG(in && w && (tail || taps == 1) && out && in != out && segs && C > 0 && nseg > 0, "causal_conv: bad argument");
    B2_CHECK_ARG(taps >= 1 && taps <= CONV_MAX_TAPS, "causal_conv: 1..%d taps are supported (got %d)", CONV_MAX_TAPS, taps);
    // the grid covers the longest segment the call may hold; tiles past a segment's end return at once
    const dim3 grid((C + 127) / 128, (max_n + CONV_TILE - 1) / CONV_TILE, nseg);
    const int own = max_n <= CONV_TILE;   // one tile per segment (decode steps, short portions): no second kernel for the carried inputs
    switch (flags & (CONV_SILU | CONV_ADD_INPUT)) {
        case 0: launch_pdl(causal_conv_kernel<0>, dim3(grid), dim3(128), 0, st, in, ld_in, w, bias, tail, out, ld_out, C, taps, segs, own); break;
        case CONV_SILU: launch_pdl(causal_conv_kernel<CONV_SILU>, dim3(grid), dim3(128), 0, st, in, ld_in, w, bias, tail, out, ld_out, C, taps, segs,
                                   own); break;
        case CONV_ADD_INPUT: launch_pdl(causal_conv_kernel<CONV_ADD_INPUT>, dim3(grid), dim3(128), 0, st, in, ld_in, w, bias, tail, out, ld_out, C, taps,
                                        segs, own); break;
        default: launch_pdl(causal_conv_kernel<CONV_SILU | CONV_ADD_INPUT>, dim3(grid), dim3(128), 0, st, in, ld_in, w, bias, tail, out, ld_out, C, taps,
                            segs, own); break;
    }
    B2_LAUNCH_CHECK();
    if (taps > 1 && !own) {
        launch_pdl(causal_conv_tail_kernel, dim3((C + 127) / 128, nseg), dim3(128), 0, st, in, ld_in, tail, C, taps, segs);
        B2_LAUNCH_CHECK();
    }
    return 0;
}

int token_shift_mix_f32(const float* x, const float* mu, float* prev, float* out, int64_t out_stride, int cols, int n_mix, const SeqSeg* segs,
                        int nseg, int max_n, cudaStream_t st) {
    B2_CHECK_ARG(x && mu && prev && out && segs && cols > 0 && nseg > 0, "token_shift: bad argument");
    B2_CHECK_ARG(n_mix >= 1 && n_mix <= SHIFT_MAX_MIX, "token_shift: 1..%d mixes are supported (got %d)", SHIFT_MAX_MIX, n_mix);
    launch_pdl(token_shift_mix_kernel, dim3((cols + 127) / 128, (max_n + SHIFT_TILE - 1) / SHIFT_TILE, nseg), dim3(128), 0, st, x, mu, prev, out, out_stride,
               cols, n_mix, segs);
    B2_LAUNCH_CHECK();
    launch_pdl(token_shift_carry_kernel, dim3((cols + 127) / 128, nseg), dim3(128), 0, st, x, prev, cols, segs);
    B2_LAUNCH_CHECK();
    return 0;
}

template <int MODE, int KW, bool V16>
int launch_scan(const ScanArgs& a, cudaStream_t st) {
    constexpr size_t smem = (size_t)(6 * SC_TT * KW * 64 + 2 * SC_TT * SC_COLS + KW * SC_TT * SC_COLS) * sizeof(float);
    B2_CUDA_CHECK(cudaFuncSetAttribute(linear_scan_kernel<MODE, KW, V16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int cols = (a.dv + SC_COLS - 1) / SC_COLS, ctas = cols * a.heads;
    ScanPlan p;
    if constexpr (MODE != SCAN_SSD && V16 && KW <= 2) {
        if (scan_blocks_fit(a)) {
            B2_CUDA_CHECK(cudaFuncSetAttribute(linear_scan_after_kernel<MODE, KW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            BlockScan blocks;
            for (int t0 = 0; t0 < a.rows; t0 += blocks.n) {
                B2_TRY(scan_blocks_plan(a, t0, &blocks));
                B2_TRY(scan_blocks_f32(a, blocks, st));
                launch_pdl(linear_scan_after_kernel<MODE, KW>, dim3(cols, a.heads), dim3(KW * 128), smem, st, a, blocks);
                B2_LAUNCH_CHECK();
            }
            return 0;
        }
    }
    // Chunks: enough CTAs for two per SM, of 64 tokens and more; two chunks would walk the whole chain all the same
    // (the last chunk has no part in the first launch, the first one none in the second)
    int chunks = a.nseg == 1 && a.chunk_scratch != nullptr ? 1 + 2 * num_sms() / ctas : 1;
    chunks = std::min(std::min(chunks, SC_MAX_CHUNKS), a.rows / 64);
    if (chunks >= 3 && (size_t)(chunks - 1) * a.heads * a.dk * (a.dv + 1) <= a.chunk_floats) {
        p.len = ((a.rows + chunks - 1) / chunks + SC_TT - 1) / SC_TT * SC_TT;
        p.chunks = (a.rows + p.len - 1) / p.len;
    }
    if (p.chunks >= 3) {
        p.final_state = a.chunk_scratch;
        p.decays = a.chunk_scratch + (size_t)(p.chunks - 1) * a.heads * a.dk * a.dv;
        if (MODE != SCAN_SSD) {
            launch_pdl(scan_prepare_kernel<MODE>, dim3((a.heads * a.dk + 255) / 256, a.rows), dim3(256), 0, st, a);
            B2_LAUNCH_CHECK();
            p.prepared = 1;
        }
        launch_pdl(linear_scan_kernel<MODE, KW, V16>, dim3(cols, a.heads, p.chunks - 1), dim3(KW * 128), smem, st, a, p);
        B2_LAUNCH_CHECK();
        p.second = 1;
        p.z0 = 1;
        launch_pdl(linear_scan_kernel<MODE, KW, V16>, dim3(cols, a.heads, p.chunks - 1), dim3(KW * 128), smem, st, a, p);
    } else {
        p.chunks = 1;
        launch_pdl(linear_scan_kernel<MODE, KW, V16>, dim3(cols, a.heads, a.nseg), dim3(KW * 128), smem, st, a, p);
    }
    B2_LAUNCH_CHECK();
    return 0;
}
template <int MODE>
int scan_of_size(const ScanArgs& a, cudaStream_t st) {
    const uintptr_t ptrs = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v) | reinterpret_cast<uintptr_t>(a.state) |
                           (MODE == SCAN_SSD ? 0 : reinterpret_cast<uintptr_t>(a.decay_in));
    const int64_t sizes = a.dk | a.dv | a.ldq | (MODE == SCAN_HGRN2 ? 0 : a.ldk) | a.ldv | (MODE == SCAN_SSD ? 0 : a.ldd);
    const bool v16 = (ptrs & 15) == 0 && sizes % 4 == 0;
    if (a.dk <= 64) return v16 ? launch_scan<MODE, 1, true>(a, st) : launch_scan<MODE, 1, false>(a, st);
    if (a.dk <= 128) return v16 ? launch_scan<MODE, 2, true>(a, st) : launch_scan<MODE, 2, false>(a, st);
    return v16 ? launch_scan<MODE, 4, true>(a, st) : launch_scan<MODE, 4, false>(a, st);
}

// chunk states, or the blocks of a prompt of `rows` tokens, as many as fit into 96 MB but 8 at least (a longer prompt goes in pieces)
size_t linear_scan_scratch_floats(int mode, int heads, int dk, int dv, int rows) {
    const size_t chunks = (size_t)(SC_MAX_CHUNKS - 1) * heads * dk * (dv + 1);
    if (mode == SCAN_SSD || dk > 128) return chunks;
    int blocks = (rows + SB_TOK - 1) / SB_TOK;
    while (blocks > SB_MIN_PIECE && scan_blocks_bytes(heads, dk, dv, blocks) > (size_t)96 << 20) --blocks;
    return std::max(chunks, (scan_blocks_bytes(heads, dk, dv, blocks) + 3) / 4);
}

int linear_scan_f32(const ScanArgs& a, cudaStream_t st) {
    B2_CHECK_ARG(a.q && (a.k || a.mode == SCAN_HGRN2) && a.v && a.decay_in && a.state && a.y && a.segs && a.nseg > 0, "linear_scan: null argument");
    B2_CHECK_ARG(a.heads > 0 && a.dk > 0 && a.dv > 0, "linear_scan: bad sizes");
    B2_CHECK_ARG(a.dk <= 256, "linear_scan: key size %d exceeds 256", a.dk);
    if (a.mode == SCAN_SSD) {
        B2_CHECK_ARG(a.groups > 0 && a.heads % a.groups == 0 && a.dt_bias && a.a_log && a.skip, "linear_scan(ssd): heads %d / groups %d", a.heads, a.groups);
        return scan_of_size<SCAN_SSD>(a, st);
    }
    if (a.mode == SCAN_HGRN2) {
        B2_CHECK_ARG(a.gate_bias && a.gate_lower, "linear_scan(hgrn2): null gate bias / lower bound");
        return scan_of_size<SCAN_HGRN2>(a, st);
    }
    if (a.mode == SCAN_GLA) {
        B2_CHECK_ARG(a.gate_bias && a.tau > 0.f, "linear_scan(gla): null decay bias or a non-positive tau");
        return scan_of_size<SCAN_GLA>(a, st);
    }
    B2_CHECK_ARG(a.mode == SCAN_RWKV, "linear_scan: unknown mode %d", a.mode);
    B2_CHECK_ARG(a.bonus != nullptr, "linear_scan(rwkv): null bonus");
    return scan_of_size<SCAN_RWKV>(a, st);
}

}  // namespace b2
