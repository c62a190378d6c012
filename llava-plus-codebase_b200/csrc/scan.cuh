// What the two forms of the linear recurrence share (recurrent.cu walks it token by token, scan_blocks.cu in blocks of tokens on the tensor cores).
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace b2 {

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// The gates' arithmetic, on a query and a raw decay entry of key `key` of head h (SSD, one decay per token, has its own): the forget gate bounded
// below f = l + (1 - l) sigmoid(z + b) (HGRN2: what is forgotten, 1 - f, is what is written), sigmoid(z + b)^(1 / tau) = exp(log_sigmoid(z + b) /
// tau) with log_sigmoid(u) = min(u, 0) - log1p(exp(-|u|)) (GLA), exp(-exp(z)) (RWKV).
template <int MODE>
__device__ __forceinline__ float scan_decay(const ScanArgs& a, int at, float z) {   // at = h * dk + key
    if (MODE == SCAN_HGRN2) {
        const float low = a.gate_lower[at];
        return fmaf(1.f - low, 1.f / (1.f + expf(-(z + a.gate_bias[at]))), low);
    }
    if (MODE == SCAN_GLA) {
        const float u = z + a.gate_bias[at];
        return expf((fminf(u, 0.f) - log1pf(expf(-fabsf(u)))) / a.tau);
    }
    return expf(-expf(z));
}
template <int MODE>
__device__ __forceinline__ float scan_query(const ScanArgs& a, float q) { return MODE == SCAN_HGRN2 ? silu_f(q) : MODE == SCAN_GLA ? q * a.q_scale : q; }

// A piece of a prompt in blocks of tokens (scan_blocks.cu): rows [t0, t0 + n) of the segment. Scratch, for every block and head: operands of the
// products as bf16 parts, the state that the block starts from, its decay per key; flags that say whether the products could do it.
constexpr int SB_TOK = 64, SB_MIN_PIECE = 8;   // blocks of a piece, where the scratch does not hold the prompt
struct BlockScan {
    int t0 = 0, n = 0, blocks = 0, key_blocks = 0, col_tiles = 0, fold_ctas = 0;
    uint8_t *q = nullptr, *k = nullptr, *a = nullptr;        // [block][head][key block][part][64 tokens][128 B], [block][head][part][keys][128 B], [..][part][64][128 B]
    float *decay = nullptr, *state = nullptr, *last = nullptr;   // [block][head][dk], [block][head][dk][dv], [head][dk][dv]: the state behind the piece
    int *bad_in = nullptr, *bad_v = nullptr, *bad_state = nullptr, *bad_out = nullptr;   // [block][head], [block][head][col tile], [head][fold CTA], as bad_v
};
bool scan_blocks_fit(const ScanArgs& a);                     // sizes and alignment, a long enough prompt, scratch
size_t scan_blocks_bytes(int heads, int dk, int dv, int blocks);
int scan_blocks_plan(const ScanArgs& a, int t0, BlockScan* p);   // the piece from t0 on
int scan_blocks_f32(const ScanArgs& a, const BlockScan& p, cudaStream_t stream);

}  // namespace b2
