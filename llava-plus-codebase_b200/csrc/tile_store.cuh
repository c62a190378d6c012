// Way out of a GEMM tile: a warp's 32 accumulator rows pass through a shared-memory buffer of its own and leave in whole lines.
//
// tcgen05.ld gives a thread one row of the tile. Stored from there, every instruction writes 16 bytes of 32 rows: 32 tag look-ups, and half sectors
// that L2 takes one by one. With K = 1024 that took longer than the products (profiles/gemm_epilogue_stores.txt, M = 9232: N = 4096 with QuickGELU
// 76.9 us, 48.2 without stores and activation; N = 3072 54.6 / 36.6; N = 1024 with a residual 26.7 / 14.6). Here a thread puts its row's pieces
// into the swizzled box that TMA expects (16-byte stores, eight rows on eight bank groups) and one lane sends the box, while the warp goes on. The
// bounds of the tensor clip rows and columns that are not there. A residual is read in whole lines ahead of the accumulator and passes through the
// same buffer; fp32 outputs, which may accumulate, are read and written in whole lines by the warp itself.
//
// The loops over fp32 outputs and general gated units are short and rolled (16 and 8 columns): the prompt of a layer-list decoder runs each of its
// products once per layer, from cold instruction caches. With 32 columns unrolled, each with its switch over the activations (94 KB of code, 69 KB
// before), the fp32 products of a layer were slower than with row-wise stores (window attention, 2048 rows: 377 us a pass, 387), rolled 355. The bf16
// outputs of the vision tower and of LLaMA, the same kernel 23 or 32 times in a row, go 32 columns at a time (16 pictures: 6.76 ms, 7.05 with 16).
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace b2 {

__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* smem, int32_t c0, int32_t c1) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(tmap), "r"(smem_u32(smem)), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }  // the buffers may be written again
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }        // the stores are done

// 32 rows of CH bytes, as TMA's swizzle of that width lays them: 16-byte piece j of row r. (CH 128: buffer on 1024 bytes; CH 64: on 512.)
template <int CH>
__device__ __forceinline__ uint4* box_slot(uint8_t* buf, int r, int j) {
    static_assert(CH == 128 || CH == 64, "swizzle widths");
    return reinterpret_cast<uint4*>(CH == 128 ? buf + r * 128 + ((j ^ (r & 7)) << 4) : buf + r * 64 + ((j ^ ((r >> 1) & 3)) << 4));
}

// The box of one warp: CH bytes of its 32 rows on their way to columns col0.. of the output
template <int CH>
struct TileBox {
    const CUtensorMap* map;
    uint8_t* buf;
    int lane, row0, M, N;   // row0: the warp's first row (there is such a row when anything is sent); N: columns of the output

    __device__ __forceinline__ void begin() const {   // the last box has been read
        if (lane == 0) bulk_wait_read();
        __syncwarp();
    }
    __device__ __forceinline__ void send(int col0) const {
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && col0 < N) {
            tma_store_2d(map, buf, col0, row0);
            bulk_commit();
        }
    }
};

// A warp's box as it lies in global memory, in registers: CH bytes of 32 rows, 8 (CH 128) or 4 lanes side by side on a row. rows: of the warp that
// exist, bytes: of a row from the box's first column on that exist.
template <int CH>
struct RowBox {
    uint4 v[CH / 16];
    __device__ __forceinline__ void load(const void* first, size_t pitch, int lane, int rows, int bytes) {
        constexpr int PER = CH / 16;   // 16-byte pieces of a row
        const uint8_t* p = static_cast<const uint8_t*>(first) + (size_t)(lane / PER) * pitch + (lane % PER) * 16;
        const bool in = (lane % PER) * 16 < bytes;
#pragma unroll
        for (int i = 0; i < PER; ++i)
            v[i] = in && i * (32 / PER) + lane / PER < rows ? *reinterpret_cast<const uint4*>(p + (size_t)i * (32 / PER) * pitch) : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ void put(uint8_t* buf, int lane) const {
        constexpr int PER = CH / 16;
#pragma unroll
        for (int i = 0; i < PER; ++i) *box_slot<CH>(buf, i * (32 / PER) + lane / PER, lane % PER) = v[i];
    }
};

__device__ __forceinline__ void add_bf16x8(float* x, const uint4& b) {
    x[0] += bf16_lo(b.x); x[1] += bf16_hi(b.x); x[2] += bf16_lo(b.y); x[3] += bf16_hi(b.y);
    x[4] += bf16_lo(b.z); x[5] += bf16_hi(b.z); x[6] += bf16_lo(b.w); x[7] += bf16_hi(b.w);
}

// fp32 outputs of a few rows leave straight from the registers: there are few lines to open, and the way through the box is the longer chain behind a
// launch's products. us, straight / boxes: 8 rows N = 12288, K = 4096 23.7 / 25.0, N = 32000, K = 2048 25.2 / 27.3; 33 rows 24.5 / 25.6, 26.7 / 28.0; 64 rows
// 26.0 / 26.2, 29.7 / 29.1; 128 rows 29.3 / 27.1, 34.9 / 30.8.
constexpr int FEW_ROWS = 48;

// out = act(acc + bias) + residual, bf16, or (F32) fp32 with post activation, scale and accumulation, for a warp's COLS columns: accumulator columns
// from taddr on are output columns from col0 on. EP: bias, residual, ld_res, out, ld_out, post, alpha, accumulate. `ready` is called in front of the
// first read of the accumulator (behind the first requests to global memory), `drained` behind the last one.
// Rows that are not there are left out of the divisions: an IEEE division of a zero takes its slow path (1900 rows, N = 2 x 5120: 64 us, 74 with them).
template <int ACT, int CH, int COLS, bool F32, class EP, class Ready, class Drained>
__device__ __forceinline__ void store_tile(const TileBox<CH>& box, uint32_t taddr, int col0, const EP& ep, Ready ready, Drained drained) {
    constexpr int ELT = F32 ? 4 : 2, BOX_COLS = CH / ELT;
    constexpr int W = F32 ? 16 : 32, PER_BOX = BOX_COLS / W, CHUNKS = COLS / W;   // chunks of W columns
    static_assert(CHUNKS % PER_BOX == 0, "whole boxes");
    if (box.row0 >= box.M) {                        // rows behind the last one: nothing to write
        ready();
        drained();
        return;
    }
    const bool in = box.row0 + box.lane < box.M;
    const bool few = F32 && box.M <= FEW_ROWS && ep.post == 0 && ep.accumulate == 0;
    const bool has_old = F32 ? ep.accumulate != 0 : ep.residual != nullptr;
    RowBox<CH> old;                                 // what the next box is added to: the residual (bf16), or what the output holds (fp32)
    auto load_old = [&](int col) {
        const int ld = F32 ? ep.ld_out : ep.ld_res;
        const uint8_t* base = F32 ? static_cast<const uint8_t*>(ep.out) : reinterpret_cast<const uint8_t*>(ep.residual);
        old.load(base + ((size_t)box.row0 * ld + col) * ELT, (size_t)ld * ELT, box.lane, box.M - box.row0, (box.N - col) * ELT);
    };
    if (has_old) load_old(col0);
    uint32_t bias = 0;                              // of the next chunk: columns 2 l and 2 l + 1 in lane l < W / 2
    auto load_bias = [&](int col) { bias = box.lane < W / 2 && col + 2 * box.lane < box.N ? reinterpret_cast<const uint32_t*>(ep.bias + col)[box.lane] : 0u; };
    if (ep.bias != nullptr) load_bias(col0);
    ready();
#pragma unroll 1
    for (int c = 0; c < CHUNKS; ++c) {
        const int col = col0 + c * W, part = c % PER_BOX;
        if (!F32 && part == 0) {
            box.begin();
            if (has_old) {
                old.put(box.buf, box.lane);
                if (c + PER_BOX < CHUNKS) load_old(col + BOX_COLS);
            }
        }
        uint32_t v[W];
        __syncwarp();
        tmem_ld_cols(taddr + c * W, v);
        tmem_ld_wait();
        if (c == CHUNKS - 1) drained();
        float x[W];
#pragma unroll
        for (int e = 0; e < W; ++e) x[e] = __uint_as_float(v[e]);
        if (ep.bias != nullptr) {
#pragma unroll
            for (int i = 0; i < W / 2; ++i) {
                const uint32_t b = __shfl_sync(0xffffffffu, bias, i);
                x[2 * i] += bf16_lo(b);
                x[2 * i + 1] += bf16_hi(b);
            }
            if (c + 1 < CHUNKS) load_bias(col + W);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
            if constexpr (ACT == ACT_QUICK_GELU) x[e] = __fdividef(x[e], 1.0f + __expf(-1.702f * x[e]));
            if constexpr (ACT == ACT_GELU_ERF) x[e] = 0.5f * x[e] * (1.0f + erff(x[e] * 0.70710678118654752440f));
        }
        if constexpr (F32) {
            if (in && ep.residual != nullptr) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (col + i * 8 < box.N) add_bf16x8(x + i * 8, *reinterpret_cast<const uint4*>(ep.residual + (size_t)(box.row0 + box.lane) * ep.ld_res + col + i * 8));
            }
            if (few) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (in && col + 4 * i < box.N)
                        *reinterpret_cast<float4*>(static_cast<float*>(ep.out) + (size_t)(box.row0 + box.lane) * ep.ld_out + col + 4 * i) =
                            make_float4(ep.alpha * x[4 * i], ep.alpha * x[4 * i + 1], ep.alpha * x[4 * i + 2], ep.alpha * x[4 * i + 3]);
                continue;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *box_slot<CH>(box.buf, box.lane, part * 4 + i) =
                    make_uint4(__float_as_uint(x[4 * i]), __float_as_uint(x[4 * i + 1]), __float_as_uint(x[4 * i + 2]), __float_as_uint(x[4 * i + 3]));
            if (in && ep.post != 0) {
#pragma unroll 1
                for (int i = 0; i < 16; ++i) {
                    float* o = reinterpret_cast<float*>(box_slot<CH>(box.buf, box.lane, part * 4 + (i >> 2))) + (i & 3);
                    *o = epi_post_act(*o, ep.post);
                }
            }
            __syncwarp();
            if (part == PER_BOX - 1) {
                constexpr int PER = CH / 16;
                const int at = col - part * 16, pc = box.lane % PER, pr = box.lane / PER;
                float* op = static_cast<float*>(ep.out) + (size_t)(box.row0 + pr) * ep.ld_out + at + pc * 4;
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const uint4 u = *box_slot<CH>(box.buf, i * (32 / PER) + pr, pc);
                    float4 f = make_float4(ep.alpha * __uint_as_float(u.x), ep.alpha * __uint_as_float(u.y), ep.alpha * __uint_as_float(u.z), ep.alpha * __uint_as_float(u.w));
                    if (has_old) { f.x += __uint_as_float(old.v[i].x); f.y += __uint_as_float(old.v[i].y); f.z += __uint_as_float(old.v[i].z); f.w += __uint_as_float(old.v[i].w); }
                    if (box.row0 + i * (32 / PER) + pr < box.M && at + pc * 4 < box.N) *reinterpret_cast<float4*>(op + (size_t)i * (32 / PER) * ep.ld_out) = f;
                }
                if (has_old && c + 1 < CHUNKS) load_old(at + BOX_COLS);
                __syncwarp();
            }
        } else {
            if (has_old) {
#pragma unroll
                for (int i = 0; i < W / 8; ++i) add_bf16x8(x + i * 8, *box_slot<CH>(box.buf, box.lane, part * (W / 8) + i));
            }
#pragma unroll
            for (int i = 0; i < W / 8; ++i)
                *box_slot<CH>(box.buf, box.lane, part * (W / 8) + i) = make_uint4(pack_bf16(x[8 * i], x[8 * i + 1]), pack_bf16(x[8 * i + 2], x[8 * i + 3]),
                                                                           pack_bf16(x[8 * i + 4], x[8 * i + 5]), pack_bf16(x[8 * i + 6], x[8 * i + 7]));
            if (part == PER_BOX - 1) box.send(col - part * W);
        }
    }
}

// out = unit(gate, up), bf16, for a warp's COLS outputs, W at a time: gate columns from taddr on, the up columns of the same outputs 64 further
template <int CH, int COLS, int W, class Ready, class Drained, class Unit>
__device__ __forceinline__ void store_glu_tile(const TileBox<CH>& box, uint32_t taddr, int col0, Ready ready, Drained drained, Unit unit) {
    static_assert(COLS * 2 == CH, "one box");
    ready();
    if (box.row0 >= box.M) {
        drained();
        return;
    }
    const bool in = box.row0 + box.lane < box.M;
    box.begin();
#pragma unroll 1
    for (int c = 0; c < COLS / W; ++c) {
        uint32_t vg[W], vu[W];
        __syncwarp();
        tmem_ld_cols(taddr + c * W, vg);
        tmem_ld_cols(taddr + 64 + c * W, vu);
        tmem_ld_wait();
        if (c == COLS / W - 1) drained();
        if (in) {
#pragma unroll
            for (int i = 0; i < W / 8; ++i) {
                float y[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = unit(__uint_as_float(vg[i * 8 + e]), __uint_as_float(vu[i * 8 + e]));
                *box_slot<CH>(box.buf, box.lane, c * (W / 8) + i) = make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
            }
        }
    }
    box.send(col0);
}

// host: the bf16 output [rows, cols] (leading dimension ld) in boxes of 32 rows x box_bytes
int make_tmap_out(CUtensorMap* map, const void* ptr, int64_t rows, int64_t cols, int64_t ld, int box_bytes);

}  // namespace b2
