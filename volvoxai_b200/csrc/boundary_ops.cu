// The F32 <-> byte boundary of a static W8A8 island and the byte-to-byte bridge between two
// quantized domains: QuantizeLinear, DequantizeLinear, RequantizeLinear. HBM-bound elementwise
// work: 16 elements per thread, 128-bit accesses where the pointers allow.  Between fp32 and bytes a thread's
// elements are four groups of four, 1024 elements apart, so that a warp's load or store of either side is one run
// of consecutive bytes (sixteen consecutive elements per thread were 64-byte strides on the fp32 side).  Unaligned, and
// in the last block, they are single elements 256 apart, read ahead of their arithmetic (6 M elements one
// off, us, one after the other / this way: quantize 10.4 / 8.9, dequantize 11.8 / 6.4, requantize 18.2 / 7.7; 64 K
// elements 3.9 / 3.0, 3.9 / 1.6, 2.5 / 2.2).  All three are launched with programmatic dependent launch, each in the
// shadow of the launch before it.
//
// Arithmetic (CPU authority of the reference, restated in oracle/w8a8_oracle.c):
//   quantize    NaN -> zero point; t = f32(x / scale) + f32(zero); saturate; ties to even
//               (native/src/kernels/quantize_linear_ops.inc:155-170, 230-254)
//   dequantize  f32((x - zero) * scale), one rounding (:9-16, 95-122)
//   requantize  t = f32(f32(x - in_zero) * f32(in_scale / out_scale)) + f32(out_zero); NaN -> out
//               zero point; saturate; ties to even (portable_inference_kernels.inc:2437-2463)
// CUDA twins in the reference: vx_cuda_quantize_i8u8, vx_cuda_dequantize_i8u8,
// vx_cuda_requantize_i8u8 (native/src/backends/cuda/kernels/
// cuda_forward_quantized_basic_kernels.inc:163-193), one element per thread.
#include "common.cuh"
#include <string.h>

namespace vxb {

namespace {

constexpr int kThreads = 256;
constexpr int kPerThread = 16;

__device__ __forceinline__ int32_t quantize1(float v, float scale, float zero_f, int32_t zero, float lo_f,
                                             float hi_f, int32_t lo, int32_t hi) {
    if (v != v) return zero;
    const float t = __fadd_rn(__fdiv_rn(v, scale), zero_f);
    if (t <= lo_f) return lo;
    if (t >= hi_f) return hi;
    return __float2int_rn(t);   // finite and inside the range here: round to nearest even
}
// f32(byte - zero) without a conversion instruction: the byte in the low mantissa bits of 2^23, less 2^23 + zero (and
// 128 more for signed bytes, whose sign bit is flipped first).  Every step is exact.
__device__ __forceinline__ float centred(uint32_t word, int i, float base) {
    return __fadd_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7440 | i)), -base);
}
__device__ __forceinline__ float centre_base(int32_t zero, bool is_unsigned) {
    return 8388608.0f + __int2float_rn(zero + (is_unsigned ? 0 : 128));
}
// one rounding per step; the product can be infinite (it then saturates), never NaN
__device__ __forceinline__ float requantized(float x, float multiplier, float zero_f) { return __fadd_rn(__fmul_rn(x, multiplier), zero_f); }

// FAST (the host found the scale within 2^+-30 and its significand not all ones): the IEEE quotient through
// div_const.  Elements whose quotient is far outside every byte range are first brought to +-4096 scales, which
// saturates all the same and keeps div_const's operands in its range; a quotient too small for it rounds, with the
// zero point added, to the zero point either way.
template <bool FAST, bool UNSIGNED>
__device__ __forceinline__ int32_t quantize_any(float v, float scale, float rcp, float bound, float zero_f, int32_t zero) {
    if constexpr (FAST) {
        const float t = __fadd_rn(div_const(fminf(fmaxf(v, -bound), bound), scale, rcp), zero_f);
        return v != v ? zero : byte_code<UNSIGNED>(t);
    } else {
        constexpr int32_t lo = UNSIGNED ? 0 : -128, hi = UNSIGNED ? 255 : 127;
        return quantize1(v, scale, zero_f, zero, (float)lo, (float)hi, lo, hi);
    }
}

template <bool FAST, bool UNSIGNED>
__global__ void __launch_bounds__(kThreads)
quantize_linear_kernel(const float* __restrict__ x, unsigned long long n, float scale, float rcp, int32_t zero,
                       uint8_t* __restrict__ out, int vec) {
    pdl_release();
    pdl_wait();
    const float zero_f = __int2float_rn(zero), bound = __fmul_rn(scale, 4096.0f);
    const unsigned long long block = (unsigned long long)blockIdx.x * (kThreads * kPerThread);
    if (vec && block + kThreads * kPerThread <= n) {
        const float4* in = reinterpret_cast<const float4*>(x + block) + threadIdx.x;
        uint32_t* dst = reinterpret_cast<uint32_t*>(out + block) + threadIdx.x;
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = __ldg(in + j * kThreads);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int32_t a = quantize_any<FAST, UNSIGNED>(v[j].x, scale, rcp, bound, zero_f, zero);
            const int32_t b = quantize_any<FAST, UNSIGNED>(v[j].y, scale, rcp, bound, zero_f, zero);
            const int32_t c = quantize_any<FAST, UNSIGNED>(v[j].z, scale, rcp, bound, zero_f, zero);
            const int32_t d = quantize_any<FAST, UNSIGNED>(v[j].w, scale, rcp, bound, zero_f, zero);
            dst[j * kThreads] = __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
        }
    } else {
        const unsigned long long first = block + threadIdx.x;
        constexpr int kBatch = FAST ? 8 : 4;   // elements loaded ahead of their arithmetic (the IEEE division's code is long)
#pragma unroll(FAST ? 2 : 1)
        for (int j = 0; j < kPerThread; j += kBatch) {
            float v[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; i++) { const unsigned long long at = first + (j + i) * kThreads; v[i] = at < n ? __ldg(x + at) : 0.0f; }
#pragma unroll
            for (int i = 0; i < kBatch; i++) {
                const unsigned long long at = first + (j + i) * kThreads;
                if (at < n) out[at] = (uint8_t)quantize_any<FAST, UNSIGNED>(v[i], scale, rcp, bound, zero_f, zero);
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads)
dequantize_linear_kernel(const uint8_t* __restrict__ x, unsigned long long n, float scale, int32_t zero,
                         int is_unsigned, float* __restrict__ out, int vec) {
    pdl_release();
    pdl_wait();
    const float base = centre_base(zero, is_unsigned);
    const uint32_t flip = is_unsigned ? 0u : 0x80808080u;
    const unsigned long long block = (unsigned long long)blockIdx.x * (kThreads * kPerThread);
    if (vec && block + kThreads * kPerThread <= n) {
        const uint32_t* in = reinterpret_cast<const uint32_t*>(x + block) + threadIdx.x;
        float4* dst = reinterpret_cast<float4*>(out + block) + threadIdx.x;
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) w[j] = __ldg(in + j * kThreads) ^ flip;
#pragma unroll
        for (int j = 0; j < 4; j++)
            dst[j * kThreads] = make_float4(__fmul_rn(centred(w[j], 0, base), scale), __fmul_rn(centred(w[j], 1, base), scale),
                                            __fmul_rn(centred(w[j], 2, base), scale), __fmul_rn(centred(w[j], 3, base), scale));
    } else {
        const unsigned long long first = block + threadIdx.x;
        uint32_t v[kPerThread];
#pragma unroll
        for (int i = 0; i < kPerThread; i++) { const unsigned long long at = first + i * kThreads; v[i] = at < n ? __ldg(x + at) : 0u; }
#pragma unroll
        for (int i = 0; i < kPerThread; i++) {
            const unsigned long long at = first + i * kThreads;
            if (at < n) out[at] = __fmul_rn(centred(v[i] ^ (flip & 0xffu), 0, base), scale);
        }
    }
}

template <bool OUT_UNSIGNED>
__global__ void __launch_bounds__(kThreads)
requantize_linear_kernel(const uint8_t* __restrict__ x, unsigned long long n, float multiplier, int32_t in_zero,
                         int in_unsigned, int32_t zero, uint8_t* __restrict__ out, int vec) {
    pdl_release();
    pdl_wait();
    const float base = centre_base(in_zero, in_unsigned), zero_f = __int2float_rn(zero);
    const uint32_t flip = in_unsigned ? 0u : 0x80808080u;
    const unsigned long long block = (unsigned long long)blockIdx.x * (kThreads * kPerThread), at = block + threadIdx.x * kPerThread;
    if (vec && at + kPerThread <= n) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(x + at));
        const uint32_t w[4] = {v.x ^ flip, v.y ^ flip, v.z ^ flip, v.w ^ flip};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int32_t a = byte_code<OUT_UNSIGNED>(requantized(centred(w[j], 0, base), multiplier, zero_f));
            const int32_t b = byte_code<OUT_UNSIGNED>(requantized(centred(w[j], 1, base), multiplier, zero_f));
            const int32_t c = byte_code<OUT_UNSIGNED>(requantized(centred(w[j], 2, base), multiplier, zero_f));
            const int32_t d = byte_code<OUT_UNSIGNED>(requantized(centred(w[j], 3, base), multiplier, zero_f));
            o[j] = __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
        }
        *reinterpret_cast<uint4*>(out + at) = make_uint4(o[0], o[1], o[2], o[3]);
    } else if (vec) {
        for (unsigned long long i = at; i < n; i++)   // the last, fewer than sixteen, elements
            out[i] = (uint8_t)byte_code<OUT_UNSIGNED>(requantized(centred(x[i] ^ (flip & 0xffu), 0, base), multiplier, zero_f));
    } else {
        const unsigned long long first = block + threadIdx.x;
        uint32_t v[kPerThread];
#pragma unroll
        for (int i = 0; i < kPerThread; i++) { const unsigned long long e = first + i * kThreads; v[i] = e < n ? __ldg(x + e) : 0u; }
#pragma unroll
        for (int i = 0; i < kPerThread; i++) {
            const unsigned long long e = first + i * kThreads;
            if (e < n) out[e] = (uint8_t)byte_code<OUT_UNSIGNED>(requantized(centred(v[i] ^ (flip & 0xffu), 0, base), multiplier, zero_f));
        }
    }
}

inline unsigned int grid_for(unsigned long long n) {
    return (unsigned int)((n + (unsigned long long)kThreads * kPerThread - 1) / ((unsigned long long)kThreads * kPerThread));
}
inline int aligned16(const void* a, const void* b) { return (((uintptr_t)a | (uintptr_t)b) & 15u) == 0 ? 1 : 0; }

}  // namespace

cudaError_t launch_quantize_linear(const float* x, unsigned long long n, float scale, int32_t zero, bool out_unsigned,
                                   void* out, cudaStream_t stream) {
    if (!n) return cudaSuccess;
    uint32_t bits;
    memcpy(&bits, &scale, 4);
    const bool fast = scale >= 9.31322574615478515625e-10f && scale <= 1073741824.0f && (bits & 0x007fffffu) != 0x007fffffu;
    auto kernel = fast ? (out_unsigned ? quantize_linear_kernel<true, true> : quantize_linear_kernel<true, false>)
                       : (out_unsigned ? quantize_linear_kernel<false, true> : quantize_linear_kernel<false, false>);
    return launch_pdl(kernel, dim3(grid_for(n)), dim3(kThreads), 0, stream, x, n, scale, (float)(1.0 / (double)scale), zero,
                      (uint8_t*)out, aligned16(x, out));
}

cudaError_t launch_dequantize_linear(const void* x, unsigned long long n, float scale, int32_t zero, bool in_unsigned,
                                     float* out, cudaStream_t stream) {
    if (!n) return cudaSuccess;
    return launch_pdl(dequantize_linear_kernel, dim3(grid_for(n)), dim3(kThreads), 0, stream, (const uint8_t*)x, n, scale, zero,
                      in_unsigned ? 1 : 0, out, aligned16(x, out));
}

cudaError_t launch_requantize_linear(const void* x, unsigned long long n, float multiplier, int32_t in_zero,
                                     bool in_unsigned, int32_t out_zero, bool out_unsigned, void* out,
                                     cudaStream_t stream) {
    if (!n) return cudaSuccess;
    return launch_pdl(out_unsigned ? requantize_linear_kernel<true> : requantize_linear_kernel<false>, dim3(grid_for(n)), dim3(kThreads), 0,
                      stream, (const uint8_t*)x, n, multiplier, in_zero, in_unsigned ? 1 : 0, out_zero, (uint8_t*)out, aligned16(x, out));
}

}  // namespace vxb
