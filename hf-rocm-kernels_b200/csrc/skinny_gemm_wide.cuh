// FP8 GEMM for the larger decode batches (above 64 tokens, and 17 to 64 by a rule; up to 256 per launch) on
// B200 (sm_100a), plain and with swiglu in the epilogue.
//
// What bounds it: up to 256 tokens the product still needs only one pass over W, so the floor is the
// larger of N*K bytes of HBM and 2*M*N*K operations of the tensor cores (they meet near 250 tokens).
// The launches of 64 tokens that served these sizes before re-read W once per 64 tokens.
//
// Layout of the work: the TOKENS are the M = 128 side of tcgen05.mma (one or two accumulators of 128
// tokens in TMEM, each token one lane), the rows of W are the N side. Against the skinny kernel
// (W rows on the M side) this makes
//   * the height of a W tile free in steps of 16 rows, so that the number of tiles fits the number
//     of SMs (28672 rows: 138 tiles of 208 on 148 SMs instead of 224 of 128 in two waves);
//   * every output row contiguous in one thread's registers: no transposition, whole 32-byte
//     sectors per store, and gate and up columns of swiglu already in the same thread.
// Both accumulators use the W tile that a stage holds, so a K block costs one W tile and one
// activation tile per CTA whatever the token count.
//
// With few W tiles the K range is split over a thread-block cluster. CTA q of a cluster finishes a
// range of 16-column groups of the tile: every CTA sends those columns of its accumulators straight
// from registers into q's shared memory (asynchronous stores that count on q's mbarrier), q adds the
// partials in rank order (deterministic) and writes D. The receive buffer lies in the ring of stages,
// which is idle once the accumulators are complete; one cluster barrier between the two uses says so
// and also says that the peers' receive barriers are armed.
//
// Roles: warps 0-7 epilogue, warp 8 TMA producer, warp 9 MMA issuer. All mbarrier waits are bounded.
// A CTA that gave up still sends its blocks and waits (bounded) for its peers' before it leaves, so
// that no store arrives at shared memory of a CTA that is gone; it stores nothing, and the status
// word says why.
// The previous kernel on the stream may still run while the first W tiles are on their way (W does
// not depend on it); everything else is touched after griddepcontrol.wait.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "skinny_gemm_kernel.cuh"

namespace hfrk {

constexpr int kWideEpilogueWarps = 8;
constexpr int kWideThreads = 32 * (kWideEpilogueWarps + 2);
constexpr int kWideMaxTokens = 256;
constexpr int kWideMaxTile = 256;
constexpr int kWideMaxStages = 8;
constexpr int kWideMaxSplit = 8;
constexpr int kWideSlotBytes = 128 * kBlockK;   // activation slot of one accumulator in a stage

struct WideParams {
    void* d;
    const float* scale;
    float kind_factor;    // 0.5 per e4m3fnuz operand
    int m, n;
    int halves;           // accumulators of 128 tokens
    int rows_half;        // tokens per accumulator, a multiple of 8
    int tile_n;           // W rows per CTA (swiglu: half gate rows, half up rows)
    int acc_cols;         // TMEM columns between the two accumulators
    int tmem_cols;
    int num_kblocks;
    int split;            // CTAs per cluster along K
    int stages;
    int d_dtype;
    int accumulate;
    // swiglu only, as in GemmParams
    uint8_t* act_out;
    const float* act_scale;
    int act_cols;
    int act_fnuz;
    uint8_t* zero_ptr;
    unsigned long long zero_bytes;
};

struct WideCtrl {
    uint64_t full[kWideMaxStages];
    uint64_t empty[kWideMaxStages];
    uint64_t accum;
    uint64_t recv;
    uint32_t tmem_base;
    volatile uint32_t abort;
};
static_assert(sizeof(WideCtrl) <= kCtrlBytes, "control block grew");

// Sixteen swiglu outputs as fp8 bytes. gate and up are the two projections before the rounding to
// the 16-bit type that the unfused chain stores them in.
__device__ __forceinline__ uint4 wide_swiglu_16(const float (&gate)[16], const float (&up)[16], float scale, float inv_act,
                                                int mid_dtype, int fnuz) {
    float2 g[8], u[8];
    float top = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        g[i] = make_float2(round_trip_16(gate[2 * i] * scale, mid_dtype), round_trip_16(gate[2 * i + 1] * scale, mid_dtype));
        u[i] = make_float2(round_trip_16(up[2 * i] * scale, mid_dtype), round_trip_16(up[2 * i + 1] * scale, mid_dtype));
        top = fmaxf(top, fmaxf(fabsf(g[i].x), fabsf(g[i].y)));   // a NaN does not count, and is one on either path
    }
    uint32_t words[4];
    // the fast path encodes e4m3fnuz through twice the scale, which must not overflow
    if (top <= kSiluFastLimit && fabsf(inv_act) < 1e38f) {
        const float inv_fast = fnuz ? 2.0f * inv_act : inv_act;
        const float2 inv = make_float2(inv_fast, inv_fast);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float2 t = mul_f32x2(mul_f32x2(silu_f32x2(make_float2(-g[i].x, -g[i].y)), u[i]), inv);
            const uint32_t pair = pack_e4m3x2(t.x, t.y);
            words[i >> 1] = (i & 1) == 0 ? pair : words[i >> 1] | (pair << 16);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float2 t = make_float2(silu_f32(g[i].x) * u[i].x * inv_act, silu_f32(g[i].y) * u[i].y * inv_act);
            if (fnuz) t = make_float2(t.x * 2.0f, t.y * 2.0f);
            const uint32_t pair = pack_e4m3x2(t.x, t.y);
            words[i >> 1] = (i & 1) == 0 ? pair : words[i >> 1] | (pair << 16);
        }
    }
    if (fnuz) {
#pragma unroll
        for (int i = 0; i < 4; ++i) words[i] = clear_negative_zero_bytes(words[i]);
    }
    return make_uint4(words[0], words[1], words[2], words[3]);
}

// Where an epilogue thread stands: its token and what it may touch.
struct WideLane {
    int token;        // row of D
    int row_in_acc;   // token - first token of this accumulator
    bool valid;       // the token exists
    int row_id;       // index among the halves * rows_half rows of the receive buffer
    bool sends;       // the row exists in the receive buffer
    uint32_t taddr;   // TMEM address of this warp's lanes in its accumulator, column 0
};

// Eight consecutive outputs of one row of D as raw 16-byte words.
template <int DT>
struct Raw8 {
    uint4 q[DT == HFRK_F32 ? 2 : 1];
};

// An 8-column piece of a row of D that is inside the matrix and 16-byte aligned.
template <int DT>
__device__ __forceinline__ bool wide_vec_ok(const WideParams& p, int token, int col) {
    const size_t idx = static_cast<size_t>(token) * p.n + col;
    return token < p.m && col + 8 <= p.n && ((reinterpret_cast<uintptr_t>(p.d) + idx * out_bytes<DT>()) & 15u) == 0;
}

// D_in of a piece. Where rows of D are not 16-byte aligned its elements are read one by one, or in pairs, all
// of them before anything is stored: a load behind a store has to wait for it, and as eight such pairs per
// piece 14933 x 1024 at 29 tokens took 40 us (9.9 us with the loads ahead, 8.4 us storing).
template <int DT>
__device__ __forceinline__ Raw8<DT> wide_load_din(const WideParams& p, int token, int col, bool wanted) {
    constexpr int kWords = DT == HFRK_F32 ? 8 : 4;
    uint32_t w[kWords];
#pragma unroll
    for (int i = 0; i < kWords; ++i) w[i] = 0u;
    if (wanted && p.accumulate && token < p.m) {
        const uint8_t* const src = static_cast<const uint8_t*>(p.d) + (static_cast<size_t>(token) * p.n + col) * out_bytes<DT>();
        const int left = p.n - col;
        if (wide_vec_ok<DT>(p, token, col)) {
#pragma unroll
            for (int i = 0; i < kWords / 4; ++i) {
                const uint4 q = reinterpret_cast<const uint4*>(src)[i];
                w[4 * i] = q.x; w[4 * i + 1] = q.y; w[4 * i + 2] = q.z; w[4 * i + 3] = q.w;
            }
        } else if constexpr (DT == HFRK_F32) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i < left) w[i] = reinterpret_cast<const uint32_t*>(src)[i];
        } else if ((reinterpret_cast<uintptr_t>(src) & 3u) == 0 && left >= 8) {
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = reinterpret_cast<const uint32_t*>(src)[i];
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i < left) w[i >> 1] |= static_cast<uint32_t>(reinterpret_cast<const uint16_t*>(src)[i]) << (16 * (i & 1));
        }
    }
    Raw8<DT> r;
#pragma unroll
    for (int i = 0; i < kWords / 4; ++i) r.q[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
    return r;
}

// D <- D_in + scale * x for one piece of eight columns (D_in is zero in overwrite mode).
template <int DT>
__device__ __forceinline__ void wide_store_piece(const WideParams& p, int token, int col, float scale, const float (&x)[8],
                                                 const Raw8<DT>& din) {
    if (token >= p.m || col >= p.n) return;
    constexpr int kWords = DT == HFRK_F32 ? 8 : 4;
    uint32_t in[kWords], out[kWords];
#pragma unroll
    for (int i = 0; i < kWords / 4; ++i) {
        in[4 * i] = din.q[i].x; in[4 * i + 1] = din.q[i].y; in[4 * i + 2] = din.q[i].z; in[4 * i + 3] = din.q[i].w;
    }
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
        if constexpr (DT == HFRK_F32) {
            out[i] = __float_as_uint(fmaf(x[i], scale, __uint_as_float(in[i])));
        } else if constexpr (DT == HFRK_BF16) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&in[i]));
            const __nv_bfloat162 h = __floats2bfloat162_rn(fmaf(x[2 * i], scale, f.x), fmaf(x[2 * i + 1], scale, f.y));
            out[i] = *reinterpret_cast<const uint32_t*>(&h);
        } else {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&in[i]));
            const __half2 h = __floats2half2_rn(fmaf(x[2 * i], scale, f.x), fmaf(x[2 * i + 1], scale, f.y));
            out[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
    }
    uint8_t* const dst = static_cast<uint8_t*>(p.d) + (static_cast<size_t>(token) * p.n + col) * out_bytes<DT>();
    const int left = p.n - col;
    if (wide_vec_ok<DT>(p, token, col)) {
#pragma unroll
        for (int i = 0; i < kWords / 4; ++i)
            reinterpret_cast<uint4*>(dst)[i] = make_uint4(out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3]);
    } else if constexpr (DT == HFRK_F32) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < left) reinterpret_cast<uint32_t*>(dst)[i] = out[i];
    } else if ((reinterpret_cast<uintptr_t>(dst) & 3u) == 0 && left >= 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint32_t*>(dst)[i] = out[i];
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i < left) reinterpret_cast<uint16_t*>(dst)[i] = static_cast<uint16_t>(out[i >> 1] >> (16 * (i & 1)));
    }
}

// Column groups (16 columns; swiglu: 16 gate and 16 up columns) that CTA q of the cluster finishes.
__device__ __forceinline__ int wide_first_group(int q, int groups, int split) { return q * groups / split; }

// Float index in an owner's receive buffer: [sender][group][part][quad of columns][row][4]. `pitch` is the
// number of rows plus one: an odd pitch lets threads that read neighbouring pieces of one row hit
// different banks.
__device__ __forceinline__ uint32_t wide_recv_index(int sender, int own_groups, int group, int parts, int part, int quad,
                                                    int pitch, int row) {
    return static_cast<uint32_t>(((((sender * own_groups + group) * parts + part) * 4 + quad) * pitch + row) * 4);
}

template <int kParts>
__device__ __forceinline__ void wide_send(const WideParams& p, const WideLane& ln, float* recv, uint32_t recv_bar, int rank,
                                          int groups, int g_first, int g_step) {
    const uint32_t recv_addr = smem_u32(recv);
    const int pitch = p.halves * p.rows_half + 1;
    for (int i = 0; i < p.split; ++i) {
        // peers first, starting behind this CTA so that they are not all sent to at once; its own block last
        int q = rank + 1 + i;
        if (q >= p.split) q -= p.split;
        const int lo = wide_first_group(q, groups, p.split), hi = wide_first_group(q + 1, groups, p.split);
        const uint32_t bar = dsmem_map(recv_bar, static_cast<uint32_t>(q));
        const uint32_t base = dsmem_map(recv_addr, static_cast<uint32_t>(q));
        for (int g = lo + g_first; g < hi; g += g_step) {
#pragma unroll
            for (int part = 0; part < kParts; ++part) {
                uint32_t v[16];
                tmem_ld_32x32b_x16(ln.taddr + static_cast<uint32_t>(part * (p.tile_n / 2) + g * 16), v);
                tmem_ld_wait();
                if (ln.sends) {
#pragma unroll
                    for (int quad = 0; quad < 4; ++quad) {
                        const uint32_t at = wide_recv_index(rank, hi - lo, g - lo, kParts, part, quad, pitch, ln.row_id);
                        if (q == rank) {   // its own block stays out of the SM-to-SM network
                            *reinterpret_cast<uint4*>(recv + at) =
                                make_uint4(v[4 * quad], v[4 * quad + 1], v[4 * quad + 2], v[4 * quad + 3]);
                        } else {
                            st_async_v4_b32(base + 4u * at, v[4 * quad], v[4 * quad + 1], v[4 * quad + 2], v[4 * quad + 3], bar);
                        }
                    }
                }
            }
        }
    }
}

// Sum over the senders, in rank order, of one column group of this thread's row.
template <int kParts>
__device__ __forceinline__ void wide_gather(const WideParams& p, const WideLane& ln, const float* recv, int own_groups,
                                            int group, int part, float (&x)[16]) {
    const int pitch = p.halves * p.rows_half + 1;
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = 0.0f;
    for (int s = 0; s < p.split; ++s) {
#pragma unroll
        for (int quad = 0; quad < 4; ++quad) {
            const float4 f = *reinterpret_cast<const float4*>(
                recv + wide_recv_index(s, own_groups, group, kParts, part, quad, pitch, ln.row_id));
            x[4 * quad] += f.x; x[4 * quad + 1] += f.y; x[4 * quad + 2] += f.z; x[4 * quad + 3] += f.w;
        }
    }
}

__device__ __forceinline__ void wide_tmem_group(uint32_t taddr, float (&x)[16]) {
    uint32_t v[16];
    tmem_ld_32x32b_x16(taddr, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = __uint_as_float(v[j]);
}

// Plain epilogue without a K split. Every warp turns its 32 tokens x 32 columns at a time in its own
// piece of the idle ring, so that D is read and written in runs of 32 columns per token (64 bytes of a
// 16-bit D: whole sectors, 8 tokens per instruction). One token per lane instead (32 bytes at a stride
// of a row of D) made the read of D_in the longest part of the call: 28672 x 4096 at 256 tokens took
// 74 us with D_in and 32 us without.
constexpr int kWideChunk = 32;
constexpr int kWidePitch = kWideChunk + 4;   // floats per token of the turned piece
constexpr int kWideTurnBytes = kWideEpilogueWarps * 32 * kWidePitch * 4;

template <int DT, typename Wait>
__device__ __forceinline__ void wide_epilogue_direct(const WideParams& p, const WideLane& ln, uint8_t* ring, int warp,
                                                     int lane, int g_first, int g_step, float scale, Wait wait_accum) {
    float* const turn = reinterpret_cast<float*>(ring) + warp * 32 * kWidePitch;
    const int n0 = blockIdx.x * p.tile_n;
    const int token0 = __shfl_sync(0xffffffffu, ln.token, 0);
    const int row_end = p.rows_half - __shfl_sync(0xffffffffu, ln.row_in_acc, 0);   // this warp's rows that hold tokens
    const int my_row = lane >> 2, my_col = (lane & 3) * 8;
    Raw8<DT> next_din[4];   // D_in of the chunk after the current one is on its way while that one is finished
    auto load_chunk = [&](int c0) {
        const int col_in_tile = c0 + my_col;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = my_row + 8 * i;
            next_din[i] = wide_load_din<DT>(p, token0 + r, n0 + col_in_tile, col_in_tile < p.tile_n && r < row_end);
        }
    };
    load_chunk(g_first * kWideChunk);
    const bool ok = wait_accum();
    for (int c0 = g_first * kWideChunk; c0 < p.tile_n; c0 += g_step * kWideChunk) {
        const int col_in_tile = c0 + my_col;
        const bool col_ok = col_in_tile < p.tile_n;
        Raw8<DT> din[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) din[i] = next_din[i];
        load_chunk(c0 + g_step * kWideChunk);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            if (c0 + 16 * part >= p.tile_n) break;
            uint32_t v[16];
            tmem_ld_32x32b_x16(ln.taddr + static_cast<uint32_t>(c0 + 16 * part), v);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                *reinterpret_cast<uint4*>(turn + lane * kWidePitch + 16 * part + 4 * q) =
                    make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = my_row + 8 * i;
            if (ok && col_ok && r < row_end) {
                const float4 f = *reinterpret_cast<const float4*>(turn + r * kWidePitch + my_col);
                const float4 h = *reinterpret_cast<const float4*>(turn + r * kWidePitch + my_col + 4);
                const float x[8] = {f.x, f.y, f.z, f.w, h.x, h.y, h.z, h.w};
                wide_store_piece<DT>(p, token0 + r, n0 + col_in_tile, scale, x, din[i]);
            }
        }
        __syncwarp();
    }
}

// Plain epilogue of an owner in the K split: work item = (token, 8 columns), neighbouring threads take
// neighbouring pieces of a token. D_in of the first items is requested before the partials are waited for.
template <int DT, typename Wait, typename Send>
__device__ __forceinline__ void wide_epilogue_owner(const WideParams& p, const float* recv, uint32_t recv_bar, int rank,
                                                    int groups, float scale, Wait wait_accum, Send send) {
    constexpr int kAhead = 4;
    constexpr int kStep = 32 * kWideEpilogueWarps;
    const int lo = wide_first_group(rank, groups, p.split), own = wide_first_group(rank + 1, groups, p.split) - lo;
    const int rows = p.halves * p.rows_half, pieces = 2 * own > 0 ? 2 * own : 1, items = own > 0 ? rows * pieces : 0;
    const int n0 = blockIdx.x * p.tile_n + lo * 16;
    Raw8<DT> din[kAhead] = {};
    auto load_ahead = [&](int base) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int item = base + i * kStep;
            const int row = item / pieces;
            din[i] = wide_load_din<DT>(p, row, n0 + (item - row * pieces) * 8, item < items);
        }
    };
    if (p.accumulate) load_ahead(threadIdx.x);
    const bool ok = wait_accum();
    send();
    if (own == 0) return;
    uint32_t own_abort = 0u;   // not the CTA's flag: the peers' stores are waited for in any case
    const bool landed = mbar_wait_bounded(recv_bar, 0u, &own_abort, kRoleEpilogue);
    if (!landed || !ok) return;
    for (int base = threadIdx.x; base < items; base += kAhead * kStep) {
        if (p.accumulate && base != static_cast<int>(threadIdx.x)) load_ahead(base);
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int item = base + i * kStep;
            if (item >= items) break;
            const int row = item / pieces, piece = item - row * pieces;
            float x[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            for (int s = 0; s < p.split; ++s) {
                const uint32_t at = wide_recv_index(s, own, piece >> 1, 1, 0, (piece & 1) * 2, rows + 1, row);
                const float4 f = *reinterpret_cast<const float4*>(recv + at);
                const float4 h = *reinterpret_cast<const float4*>(recv + at + 4 * (rows + 1));
                x[0] += f.x; x[1] += f.y; x[2] += f.z; x[3] += f.w;
                x[4] += h.x; x[5] += h.y; x[6] += h.z; x[7] += h.w;
            }
            wide_store_piece<DT>(p, row, n0 + piece * 8, scale, x, din[i]);
        }
    }
}

template <int DT, typename Wait, typename Send>
__device__ __forceinline__ void wide_epilogue_plain(const WideParams& p, const WideLane& ln, uint8_t* ring,
                                                    uint32_t recv_bar, int rank, int groups, int warp, int lane, int g_first,
                                                    int g_step, float scale, Wait wait_accum, Send send) {
    if (p.split == 1) {
        wide_epilogue_direct<DT>(p, ln, ring, warp, lane, g_first, g_step, scale, wait_accum);
    } else {
        wide_epilogue_owner<DT>(p, reinterpret_cast<const float*>(ring), recv_bar, rank, groups, scale, wait_accum, send);
    }
}

__device__ __forceinline__ void wide_epilogue_swiglu(const WideParams& p, const WideLane& ln, const float* recv, int rank,
                                                     int groups, int g_first, int g_step, float scale, bool store) {
    const int half = p.tile_n / 2;
    const bool direct = p.split == 1;
    const int lo = direct ? 0 : wide_first_group(rank, groups, p.split);
    const int hi = direct ? groups : wide_first_group(rank + 1, groups, p.split);
    const float inv_act = 1.0f / __ldg(p.act_scale);
    for (int g = lo + g_first; g < hi; g += g_step) {
        float gate[16], up[16];
        if (direct) {
            wide_tmem_group(ln.taddr + static_cast<uint32_t>(g * 16), gate);
            wide_tmem_group(ln.taddr + static_cast<uint32_t>(half + g * 16), up);
        } else if (ln.sends) {
            wide_gather<2>(p, ln, recv, hi - lo, g - lo, 0, gate);
            wide_gather<2>(p, ln, recv, hi - lo, g - lo, 1, up);
        }
        const int col = static_cast<int>(blockIdx.x) * half + g * 16;
        if (store && ln.valid && col < p.act_cols) {   // act_cols % 16 == 0: a group is inside or outside
            *reinterpret_cast<uint4*>(p.act_out + static_cast<size_t>(ln.token) * p.act_cols + col) =
                wide_swiglu_16(gate, up, scale, inv_act, p.d_dtype, p.act_fnuz);
        }
    }
}

template <bool kSwiglu>
__global__ void __launch_bounds__(kWideThreads, 2)
skinny_gemm_fp8_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                            const WideParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t ring_addr = (raw_addr + 1023u) & ~1023u;
    uint8_t* const ring_ptr = smem_raw + (ring_addr - raw_addr);
    // a stage: one activation slot per accumulator, then the W tile (all multiples of 1024 bytes)
    const uint32_t a_slots = static_cast<uint32_t>(p.halves) * kWideSlotBytes;
    const uint32_t stage_bytes = a_slots + static_cast<uint32_t>(p.tile_n) * kBlockK;
    // bytes that land: rows of an activation slot past rows_half keep stale shared memory; their
    // accumulator lanes are never read
    const uint32_t stage_tx = static_cast<uint32_t>(p.halves * p.rows_half + p.tile_n) * kBlockK;
    WideCtrl* const ctrl = reinterpret_cast<WideCtrl*>(ring_ptr + static_cast<size_t>(p.stages) * stage_bytes);
    const uint32_t full_bar = smem_u32(&ctrl->full[0]);
    const uint32_t empty_bar = smem_u32(&ctrl->empty[0]);
    const uint32_t accum_bar = smem_u32(&ctrl->accum);
    const uint32_t recv_bar = smem_u32(&ctrl->recv);
    constexpr int kParts = kSwiglu ? 2 : 1;
    const int groups = p.tile_n / (16 * kParts);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const bool producer_warp = warp == kWideEpilogueWarps;
    const bool mma_warp = warp == kWideEpilogueWarps + 1;

    const int rank = p.split > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
    const int kb_base = p.num_kblocks / p.split, kb_rem = p.num_kblocks % p.split;
    const int kb_count = kb_base + (rank < kb_rem ? 1 : 0);
    const int kb_start = rank * kb_base + (rank < kb_rem ? rank : kb_rem);
    const int prologue = kb_count < p.stages ? kb_count : p.stages;

    auto load_w = [&](uint32_t stage, uint32_t bar, int k_coord, uint64_t policy) {
        if (kSwiglu) {
            const int half = p.tile_n / 2;
            const int g0 = static_cast<int>(blockIdx.x) * half;
            tma_load_2d(stage + a_slots, &tmap_w, bar, k_coord, g0, policy);
            tma_load_2d(stage + a_slots + static_cast<uint32_t>(half) * kBlockK, &tmap_w, bar, k_coord, p.act_cols + g0,
                        policy);
        } else {
            tma_load_2d(stage + a_slots, &tmap_w, bar, k_coord, static_cast<int>(blockIdx.x) * p.tile_n, policy);
        }
    };
    auto load_a = [&](uint32_t stage, uint32_t bar, int k_coord, uint64_t policy) {
        tma_load_2d(stage, &tmap_a, bar, k_coord, 0, policy);
        if (p.halves > 1) tma_load_2d(stage + kWideSlotBytes, &tmap_a, bar, k_coord, p.rows_half, policy);
    };

    uint64_t pol_w = 0, pol_a = 0;
    if (producer_warp) {
        if (lane == 0) {
            ctrl->abort = 0u;
            for (int s = 0; s < p.stages; ++s) {
                mbar_init(full_bar + 8u * s, 1);
                mbar_init(empty_bar + 8u * s, 1);
            }
            mbar_init(accum_bar, 1);
            mbar_init(recv_bar, 1);
            mbar_init_fence();
            if (p.split > 1) {
                const int own = wide_first_group(rank + 1, groups, p.split) - wide_first_group(rank, groups, p.split);
                mbar_arrive_expect_tx(recv_bar, static_cast<uint32_t>((p.split - 1) * own * kParts * 64 * p.halves * p.rows_half));
            }
        }
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"r"(kWideThreads) : "memory");
        if (lane == 0) {
            prefetch_tensormap(&tmap_w);
            prefetch_tensormap(&tmap_a);
            pol_w = l2_policy_evict_first();
            pol_a = l2_policy_evict_last();
            for (int i = 0; i < prologue; ++i) {
                mbar_arrive_expect_tx(full_bar + 8u * i, stage_tx);
                load_w(ring_addr + i * stage_bytes, full_bar + 8u * i, (kb_start + i) * kBlockK, pol_w);
            }
            pdl_wait_prior_grids();
            for (int i = 0; i < prologue; ++i)
                load_a(ring_addr + i * stage_bytes, full_bar + 8u * i, (kb_start + i) * kBlockK, pol_a);
        }
        __syncwarp();
    } else {
        if (mma_warp) {
            tmem_alloc(smem_u32(&ctrl->tmem_base), static_cast<uint32_t>(p.tmem_cols));
            tmem_relinquish_alloc_permit();
            tcgen05_fence_before_sync();
        }
        asm volatile("bar.sync 2, %0;" ::"r"(kWideThreads) : "memory");
        tcgen05_fence_after_sync();
        // after this CTA's TMEM is allocated: CTAs of the next grid must not take columns that a CTA of
        // this one (whose cluster may be waiting for it) has yet to get
        if (mma_warp) pdl_launch_dependents();
    }

    if (producer_warp) {
        if (lane == 0) {
            uint32_t s = 0, parity = 0, stage_addr = ring_addr;
            int k_coord = (kb_start + prologue) * kBlockK;
            int issued = prologue;
            for (int i = prologue; i < kb_count; ++i) {
                if (!mbar_wait_bounded(empty_bar + 8u * s, parity, &ctrl->abort, kRoleProducer)) break;
                mbar_arrive_expect_tx(full_bar + 8u * s, stage_tx);
                load_w(stage_addr, full_bar + 8u * s, k_coord, pol_w);
                load_a(stage_addr, full_bar + 8u * s, k_coord, pol_a);
                issued = i + 1;
                k_coord += kBlockK;
                stage_addr += stage_bytes;
                if (++s == static_cast<uint32_t>(p.stages)) {
                    s = 0;
                    stage_addr = ring_addr;
                    parity ^= 1u;
                }
            }
            if (ctrl->abort) {
                // give the copies already in flight a bounded chance to land before the CTA goes on
                for (int st = 0; st < p.stages && st < issued; ++st) {
                    const int last = ((issued - 1 - st) / p.stages) * p.stages + st;
                    const uint32_t par = static_cast<uint32_t>(last / p.stages) & 1u;
                    const long long start = clock64();
                    while (!mbar_try_wait(full_bar + 8u * st, par)) {
                        if (clock64() - start > kWaitLimitCycles / 8) break;
                    }
                }
            }
        }
        __syncwarp();
        // releases the receive barrier's initialisation to the peers
        if (p.split > 1) cluster_arrive_release();
    } else if (mma_warp) {
        const uint32_t tmem_acc = ctrl->tmem_base;
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_e4m3_f32(128, p.tile_n);
            const uint64_t desc_fixed = umma_desc_kmajor_sw128(0u);
            uint32_t s = 0, parity = 0, stage_addr = ring_addr;
            for (int i = 0; i < kb_count; ++i) {
                if (!mbar_wait_bounded(full_bar + 8u * s, parity, &ctrl->abort, kRoleMma)) break;
                tcgen05_fence_after_sync();
                const uint64_t w_desc = desc_fixed + ((stage_addr + a_slots) >> 4);
                for (int h = 0; h < p.halves; ++h) {
                    const uint64_t a_desc = desc_fixed + ((stage_addr + static_cast<uint32_t>(h) * kWideSlotBytes) >> 4);
                    const uint32_t acc = tmem_acc + static_cast<uint32_t>(h * p.acc_cols);
#pragma unroll
                    for (int kk = 0; kk < kBlockK / kUmmaK; ++kk)
                        umma_f8f6f4(acc, a_desc + 2u * kk, w_desc + 2u * kk, idesc, (i | kk) != 0 ? 1u : 0u);
                }
                if (i + p.stages < kb_count) umma_commit(empty_bar + 8u * s);
                stage_addr += stage_bytes;
                if (++s == static_cast<uint32_t>(p.stages)) {
                    s = 0;
                    stage_addr = ring_addr;
                    parity ^= 1u;
                }
            }
            umma_commit(accum_bar);
            // the ring may be handed to the peers' partials once the tensor core has read it
            if (p.split > 1) (void)mbar_wait_bounded(accum_bar, 0u, &ctrl->abort, kRoleMma);
        }
        __syncwarp();
        if (p.split > 1) cluster_arrive_release();
    } else {
        pdl_wait_prior_grids();
        const int quarter = warp & 3, group_of_warps = warp >> 2;
        const int row = quarter * 32 + lane;
        const int acc = p.halves > 1 ? group_of_warps : 0;
        WideLane ln;
        ln.token = acc * p.rows_half + row;
        ln.row_in_acc = row;
        ln.sends = row < p.rows_half;
        ln.valid = ln.sends && ln.token < p.m;
        ln.row_id = ln.token;
        ln.taddr = ctrl->tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc * p.acc_cols);
        // two accumulators: four warps each; one accumulator: the two sets of warps take turns on its columns
        const int g_first = p.halves > 1 ? 0 : group_of_warps, g_step = p.halves > 1 ? 1 : 2;
        const float scale = __ldg(p.scale) * p.kind_factor;

        auto wait_accum = [&]() {
            bool ok = mbar_wait_bounded(accum_bar, 0u, &ctrl->abort, kRoleEpilogue);
            ok = __all_sync(0xffffffffu, ok) && ctrl->abort == 0u;
            ok = __all_sync(0xffffffffu, ok);
            tcgen05_fence_after_sync();
            return ok;
        };
        auto send = [&]() {
            cluster_arrive_relaxed();
            cluster_wait_acquire();
            wide_send<kParts>(p, ln, reinterpret_cast<float*>(ring_ptr), recv_bar, rank, groups, g_first, g_step);
            // the CTA's own block was written with ordinary stores by its other epilogue warps
            asm volatile("bar.sync 1, %0;" ::"r"(32 * kWideEpilogueWarps) : "memory");
        };
        if constexpr (kSwiglu) {
            bool ok = wait_accum();
            if (p.split > 1) send();
            if (p.split > 1 && wide_first_group(rank, groups, p.split) < wide_first_group(rank + 1, groups, p.split)) {
                uint32_t own_abort = 0u;   // not the CTA's flag: the peers' stores are waited for in any case
                const bool landed = mbar_wait_bounded(recv_bar, 0u, &own_abort, kRoleEpilogue);
                ok = __all_sync(0xffffffffu, landed) && ok;
            }
            wide_epilogue_swiglu(p, ln, reinterpret_cast<const float*>(ring_ptr), rank, groups, g_first, g_step, scale, ok);
            const size_t cta = static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x;
            const size_t ctas = static_cast<size_t>(gridDim.x) * gridDim.y;
            const size_t vecs = static_cast<size_t>(p.zero_bytes / 16);
            constexpr size_t kPer = 32 * kWideEpilogueWarps;
            for (size_t i = cta * kPer + threadIdx.x; i < vecs; i += ctas * kPer)
                reinterpret_cast<uint4*>(p.zero_ptr)[i] = make_uint4(0, 0, 0, 0);
        } else if (p.d_dtype == HFRK_BF16) {
            wide_epilogue_plain<HFRK_BF16>(p, ln, ring_ptr, recv_bar, rank, groups, warp, lane, g_first, g_step, scale, wait_accum,
                                             send);
        } else if (p.d_dtype == HFRK_F16) {
            wide_epilogue_plain<HFRK_F16>(p, ln, ring_ptr, recv_bar, rank, groups, warp, lane, g_first, g_step, scale, wait_accum,
                                             send);
        } else {
            wide_epilogue_plain<HFRK_F32>(p, ln, ring_ptr, recv_bar, rank, groups, warp, lane, g_first, g_step, scale, wait_accum, send);
        }
    }
    if (p.split > 1 && warp >= kWideEpilogueWarps) cluster_wait_acquire();

    tcgen05_fence_before_sync();
    __syncthreads();
    if (mma_warp) tmem_dealloc(ctrl->tmem_base, static_cast<uint32_t>(p.tmem_cols));
}

}  // namespace hfrk
