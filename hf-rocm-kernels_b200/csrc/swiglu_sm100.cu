// SwiGLU fused with the fp8 quantisation of the down projection's input and with the zeroing of
// the buffer that projection accumulates into.
//
//   out[r, c] = e4m3( silu(gate_up[r, c]) * gate_up[r, hidden + c] * (1 / scale) ),   next_buffer <- 0
//
// Replaces the reference's launcher and kernels csrc/op_src/swiglu/swiglu_dispatch.cu:8-42,
// swiglu_vectorized.cu and swiglu_scalar.cu:24-66 (fp16 in, e4m3fnuz out, one 16-byte load of gate
// and one of up per thread and 8 outputs). The arithmetic keeps the reference's order: silu in
// fp32, times up, times the reciprocal of the scale, then one rounding to fp8.
//
// HBM should bound it (4 bytes read and 1 written per output element), but at 31 instructions per
// element the issue slots did: 41.2 us at 2048 x 14336 (3.56 TB/s, 75 % of the issue slots busy, DRAM 39 %).
// Now 23 per element: two fp32 operations per instruction and a cheaper quotient with the same bits for every
// 16-bit gate (silu_f32x2), row and column carried along instead of two 64-bit divisions per vector, and the scale
// of e4m3fnuz folded into the factor: 29 to 31 us (4.7 to 5.1 TB/s, issue slots 70 % busy; what is left is mostly
// expf and the conversions).
// Every thread owns 8 consecutive outputs of one row (two 16-byte loads, one 8-byte store), two such
// vectors in flight. CTAs of 128 threads, at most 16 per SM, stride over the matrix: ten of them are
// resident, the others even out the end (300 x 14336: 6.2 us, 7.2 us as CTAs of 256 that each do their
// two vectors and leave, 6.3 us with just the CTAs that are resident), so
// rows of any length keep all SMs loading. It is launched as a
// programmatic dependent of the GEMM before it and releases the GEMM after it at once: that
// GEMM's weight prefetch overlaps this kernel entirely.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "../../include/hfrk_b200.h"
#include "host_common.h"
#include "elementwise_common.cuh"
#include "ptx_sm100.cuh"

namespace hfrk {
namespace {

constexpr int kSwigluThreads = 128;
constexpr int kSwigluCtasPerSm = 16;
// The element-by-element kernel, one element in flight per thread, wants larger CTAs (115 x 5135: 4.2 us, 4.8 as
// CTAs of 128).
constexpr int kScalarThreads = 256;
constexpr int kScalarCtasPerSm = 8;

__device__ __forceinline__ float2 pair_f32(uint32_t w, __half) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
__device__ __forceinline__ float2 pair_f32(uint32_t w, __nv_bfloat16) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}
__device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b, __half) {
    const __half2 m = __hmax2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&m);
}
__device__ __forceinline__ uint32_t max_abs(uint32_t a, uint32_t b, __nv_bfloat16) {
    const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&m);
}

template <typename T, bool kFnuz>
__device__ __forceinline__ uint2 swiglu_8(const uint4& gate_raw, const uint4& up_raw, float inv_scale) {
    const uint32_t g[4] = {gate_raw.x, gate_raw.y, gate_raw.z, gate_raw.w};
    const uint32_t u[4] = {up_raw.x, up_raw.y, up_raw.z, up_raw.w};
    // largest |gate| of the eight (a NaN does not count, and is one on either path)
    const uint32_t abs_mask = 0x7fff7fffu;
    const float2 top = pair_f32(max_abs(max_abs(g[0] & abs_mask, g[1] & abs_mask, T()),
                                        max_abs(g[2] & abs_mask, g[3] & abs_mask, T()), T()), T());
    // the fast path encodes e4m3fnuz through twice the scale, which must not overflow
    const bool fast = fmaxf(top.x, top.y) <= kSiluFastLimit && fabsf(inv_scale) < 1e38f;
    const float inv_fast = kFnuz ? 2.0f * inv_scale : inv_scale;
    const float2 inv = make_float2(inv_fast, inv_fast);
    uint32_t half_words[4];
    if (fast) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 t = mul_f32x2(mul_f32x2(silu_f32x2(pair_f32(g[j] ^ 0x80008000u, T())), pair_f32(u[j], T())), inv);
            half_words[j] = pack_e4m3x2(t.x, t.y);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 x = pair_f32(g[j], T()), y = pair_f32(u[j], T());
            float2 t = make_float2(silu_f32(x.x) * y.x * inv_scale, silu_f32(x.y) * y.y * inv_scale);
            // An e4m3fnuz byte is worth half of the same byte read as e4m3fn: encode twice the value.
            if (kFnuz) t = make_float2(t.x * 2.0f, t.y * 2.0f);
            half_words[j] = pack_e4m3x2(t.x, t.y);
        }
    }
    uint2 packed = make_uint2(half_words[0] | (half_words[1] << 16), half_words[2] | (half_words[3] << 16));
    if (kFnuz) {
        packed.x = clear_negative_zero_bytes(packed.x);
        packed.y = clear_negative_zero_bytes(packed.y);
    }
    return packed;
}

// Vector path: hidden % 8 == 0, gate_up 16-byte aligned, out 8-byte aligned.
template <typename T, bool kFnuz>
__global__ void __launch_bounds__(kSwigluThreads)
swiglu_fp8_vec8_kernel(const T* __restrict__ gate_up, const float* __restrict__ scale_dev, uint8_t* __restrict__ out,
                       uint8_t* __restrict__ next_buffer, size_t buffer_bytes, int rows, int hidden) {
    pdl_launch_dependents();
    pdl_wait_prior_grids();
    const float inv_scale = 1.0f / __ldg(scale_dev);
    const unsigned vecs_per_row = hidden >= 8 ? static_cast<unsigned>(hidden) >> 3 : 1u;
    const unsigned end_row = hidden >= 8 ? static_cast<unsigned>(rows) : 0u;
    const unsigned stride = gridDim.x * blockDim.x;
    // (row, vector) of this thread's item and the step to its next one: divisions once per thread, 32 bits
    const unsigned step_rows = stride / vecs_per_row, step_vecs = stride - step_rows * vecs_per_row;
    const unsigned first = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned row = first / vecs_per_row, vec = first - row * vecs_per_row;
    const size_t row_in = static_cast<size_t>(vecs_per_row) * 2;
    const uint4* const in = reinterpret_cast<const uint4*>(gate_up);
    uint2* const dst = reinterpret_cast<uint2*>(out);
    auto advance = [&]() {
        row += step_rows;
        vec += step_vecs;
        if (vec >= vecs_per_row) {
            vec -= vecs_per_row;
            ++row;
        }
    };
    // Two independent vectors per iteration: four 16-byte loads in flight per thread.
    while (row < end_row) {
        const size_t at1 = row * row_in + vec, to1 = static_cast<size_t>(row) * vecs_per_row + vec;
        const uint4 g1 = __ldcs(in + at1), u1 = __ldcs(in + at1 + vecs_per_row);
        advance();
        const bool second = row < end_row;
        const size_t at2 = row * row_in + vec, to2 = static_cast<size_t>(row) * vecs_per_row + vec;
        uint4 g2 = make_uint4(0, 0, 0, 0), u2 = g2;
        if (second) {
            g2 = __ldcs(in + at2);
            u2 = __ldcs(in + at2 + vecs_per_row);
        }
        dst[to1] = swiglu_8<T, kFnuz>(g1, u1, inv_scale);
        if (!second) break;
        dst[to2] = swiglu_8<T, kFnuz>(g2, u2, inv_scale);
        advance();
    }
    zero_range_shared(next_buffer, buffer_bytes);
}

// Scalar path: any hidden, any alignment.
template <typename T, bool kFnuz>
__global__ void __launch_bounds__(kScalarThreads)
swiglu_fp8_scalar_kernel(const T* __restrict__ gate_up, const float* __restrict__ scale_dev,
                         uint8_t* __restrict__ out, uint8_t* __restrict__ next_buffer, size_t buffer_bytes, int rows,
                         int hidden) {
    pdl_launch_dependents();
    pdl_wait_prior_grids();
    const float inv_scale = 1.0f / __ldg(scale_dev);
    const size_t total = static_cast<size_t>(rows) * hidden;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const size_t r = i / hidden, c = i - r * hidden;
        const T* row = gate_up + r * 2 * hidden;
        float t = silu_f32(to_f32<T>(row[c]));
        t *= to_f32<T>(row[hidden + c]);
        t *= inv_scale;
        if (kFnuz) t *= 2.0f;
        uint8_t byte = static_cast<uint8_t>(pack_e4m3x2(t, 0.0f) & 0xffu);
        if (kFnuz && byte == 0x80u) byte = 0;
        out[i] = byte;
    }
    zero_range(next_buffer, buffer_bytes);
}

template <typename T>
int launch_swiglu(const void* gate_up, const float* scale_dev, void* out, void* next_buffer, int rows, int hidden,
                  size_t buffer_bytes, bool fnuz, bool vec, cudaStream_t stream) {
    const size_t items = static_cast<size_t>(rows) * (vec ? hidden / 8 : hidden);
    // Enough threads for one item each, capped at a full machine: the kernels stride over what is left.
    const size_t threads = vec ? kSwigluThreads : kScalarThreads;
    size_t want = (items + threads - 1) / threads;
    const size_t zero_want = (buffer_bytes / 16 + threads - 1) / threads;
    if (zero_want > want) want = zero_want;
    const size_t cap = static_cast<size_t>(kSmCount) * (vec ? kSwigluCtasPerSm : kScalarCtasPerSm);
    const unsigned grid = static_cast<unsigned>(want < 1 ? 1 : (want > cap ? cap : want));
    const T* in = static_cast<const T*>(gate_up);
    uint8_t* o = static_cast<uint8_t*>(out);
    uint8_t* nb = static_cast<uint8_t*>(next_buffer);
    if (vec) {
        return fnuz ? launch_elementwise(swiglu_fp8_vec8_kernel<T, true>, grid, kSwigluThreads, stream, in,
                                         scale_dev, o, nb, buffer_bytes, rows, hidden)
                    : launch_elementwise(swiglu_fp8_vec8_kernel<T, false>, grid, kSwigluThreads, stream, in,
                                         scale_dev, o, nb, buffer_bytes, rows, hidden);
    }
    return fnuz ? launch_elementwise(swiglu_fp8_scalar_kernel<T, true>, grid, kScalarThreads, stream, in, scale_dev,
                                     o, nb, buffer_bytes, rows, hidden)
                : launch_elementwise(swiglu_fp8_scalar_kernel<T, false>, grid, kScalarThreads, stream, in, scale_dev,
                                     o, nb, buffer_bytes, rows, hidden);
}

}  // namespace
}  // namespace hfrk

extern "C" int hfrk_swiglu_fp8(const void* gate_up, const float* scale_dev, void* out, void* next_buffer, int rows,
                               int hidden, int64_t buffer_cols, int in_dtype, int out_kind, int force_scalar,
                               void* stream) {
    using namespace hfrk;
    if (rows < 0 || hidden < 0 || buffer_cols < 0) {
        set_last_error("swiglu: negative extent");
        return HFRK_INVALID_CONFIG;
    }
    if (in_dtype != HFRK_F16 && in_dtype != HFRK_BF16) {
        set_last_error("swiglu: gate_up must be fp16 or bf16");
        return HFRK_BAD_DTYPE;
    }
    if (out_kind != HFRK_E4M3FN && out_kind != HFRK_E4M3FNUZ) {
        set_last_error("swiglu: output must be e4m3fn or e4m3fnuz");
        return HFRK_BAD_DTYPE;
    }
    const size_t buffer_bytes = static_cast<size_t>(rows) * static_cast<size_t>(buffer_cols) * 2;
    if (static_cast<size_t>(rows) * hidden == 0 && buffer_bytes == 0) return HFRK_SUCCESS;
    if (scale_dev == nullptr || (static_cast<size_t>(rows) * hidden != 0 && (gate_up == nullptr || out == nullptr)) ||
        (buffer_bytes != 0 && next_buffer == nullptr)) {
        set_last_error("swiglu: null pointer");
        return HFRK_INVALID_CONFIG;
    }
    if ((reinterpret_cast<uintptr_t>(gate_up) & 1u) || (reinterpret_cast<uintptr_t>(next_buffer) & 1u)) {
        set_last_error("swiglu: 16-bit tensors must be 2-byte aligned");
        return HFRK_BAD_ALIGNMENT;
    }
    const bool vec = !force_scalar && hidden % 8 == 0 && (reinterpret_cast<uintptr_t>(gate_up) & 15u) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & 7u) == 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool fnuz = out_kind == HFRK_E4M3FNUZ;
    if (in_dtype == HFRK_F16)
        return launch_swiglu<__half>(gate_up, scale_dev, out, next_buffer, rows, hidden, buffer_bytes, fnuz, vec, s);
    return launch_swiglu<__nv_bfloat16>(gate_up, scale_dev, out, next_buffer, rows, hidden, buffer_bytes, fnuz, vec,
                                        s);
}
