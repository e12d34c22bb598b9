// K1: per-token symmetric int8 quantizer, plus the small layout helpers
// (weight repack, zero-point folding, byte copies).  HBM-bound byte work:
// 128-bit loads, 128-bit stores, one pass over the fp32 activations.
//
// Arithmetic contract (reference: native/src/kernels/packed_linear_ops.inc
// :97-153 AVX2, :1574-1597 scalar; CUDA twin cuda_forward_llm_kernels.inc
// :195-247):
//   row invalid if any element has an all-ones exponent (NaN/Inf)
//   amax  = max |x|;  scale = amax == 0 ? 1 : amax / 127  (IEEE divide)
//   scale = max(scale, 2^-126)
//   q     = cvt.rni(clamp(x / scale, -127, 127))            (IEEE divide, ties to even)
// A reciprocal-multiply would move half-way values across a rounding
// boundary, so the divide is __fdiv_rn on every element.
#include "quantize.cuh"
#include <cooperative_groups.h>

namespace vxb {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxVecPerThread = 8;   // float4 per thread kept in registers (K <= 8192)
constexpr uint32_t kClusterMaxRows = 32;   // up to this many rows a cluster of CTAs shares each row

// Reduce (max, or-flag) over THREADS_PER_ROW consecutive threads (power of two).
template <int THREADS_PER_ROW>
__device__ __forceinline__ void row_reduce(float& amax, int& bad, float* smem_max, int* smem_bad) {
    constexpr int kWarpSpan = THREADS_PER_ROW < 32 ? THREADS_PER_ROW : 32;
#pragma unroll
    for (int off = kWarpSpan / 2; off > 0; off >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        bad |= __shfl_xor_sync(0xffffffffu, bad, off);
    }
    if constexpr (THREADS_PER_ROW > 32) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (lane == 0) { smem_max[warp] = amax; smem_bad[warp] = bad; }
        __syncthreads();
        constexpr int kWarps = THREADS_PER_ROW / 32;
        const int first = (threadIdx.x / THREADS_PER_ROW) * kWarps;  // this row's first warp
        float m = 0.0f; int b = 0;
#pragma unroll
        for (int i = 0; i < kWarps; i++) { m = fmaxf(m, smem_max[first + i]); b |= smem_bad[first + i]; }
        amax = m; bad = b;
    }
}

// Every quantizer waits until the kernel before it has finished with the activations and the q scratch, and lets the
// consumer kernel start its prologue and its first weight loads: after that wait as a rule, before it (`early`) where the
// caller says so (api.cu's release_early).  Released before the wait, the consumer sets up and loads beside the
// predecessor's last tiles and holds them up; released after it, its set-up is on the call's path.  us a pass, early /
// late: 8 x 4096 -> 14336 in a stream of calls 16.7 / 15.8, replayed from a graph 15.9 / 15.4; 64 x 1024 -> 3072 8.3 / 7.2
// and 7.6 / 6.8; decode layers replayed from a graph, 64 rows of hidden 1024 36.7 / 36.0, 8 rows of 576 28.4 / 25.8, 16 of
// 2048 44.5 / 42.9 (41.4 / 38.3, 31.7 / 28.5, 47.4 / 45.2 in a stream).
__device__ __forceinline__ void wait_and_release(bool early) {
    if (early) pdl_release();
    pdl_wait();
    if (!early) pdl_release();
}

// THREADS_PER_ROW threads cooperate on one row; kThreads/THREADS_PER_ROW rows per CTA.
// VEC: row addressed as float4 (k % 4 == 0, 16-byte aligned base and ldq % 16 == 0).
// CACHE: the row's float4s stay in registers between the two passes.
template <int THREADS_PER_ROW, bool CACHE>
__global__ void __launch_bounds__(kThreads)
quantize_rows_vec(const float* __restrict__ x, uint32_t rows, uint32_t k, int8_t* __restrict__ q,
                  uint32_t ldq, float* __restrict__ row_scales, int32_t* __restrict__ valid, bool early) {
    __shared__ float smem_max[kThreads / 32];
    __shared__ int smem_bad[kThreads / 32];
    wait_and_release(early);
    constexpr int kRowsPerCta = kThreads / THREADS_PER_ROW;
    const uint32_t row = blockIdx.x * kRowsPerCta + threadIdx.x / THREADS_PER_ROW;
    const int t = threadIdx.x % THREADS_PER_ROW;
    const bool active = row < rows;
    const uint32_t nvec = k / 4;
    const float4* in = reinterpret_cast<const float4*>(x + (size_t)(active ? row : 0) * k);

    float4 cache[CACHE ? kMaxVecPerThread : 1];
    float amax = 0.0f; int bad = 0;
    if (active) {
        if constexpr (CACHE) {
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const uint32_t v = t + i * THREADS_PER_ROW;
                cache[i] = v < nvec ? __ldg(in + v) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const float4 c = cache[i];
                bad |= nonfinite_bits(c.x) | nonfinite_bits(c.y) | nonfinite_bits(c.z) | nonfinite_bits(c.w);
                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(c.z), fabsf(c.w))));
            }
        } else {
            for (uint32_t v = t; v < nvec; v += THREADS_PER_ROW) {
                const float4 c = __ldg(in + v);
                bad |= nonfinite_bits(c.x) | nonfinite_bits(c.y) | nonfinite_bits(c.z) | nonfinite_bits(c.w);
                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(c.z), fabsf(c.w))));
            }
        }
    }
    row_reduce<THREADS_PER_ROW>(amax, bad, smem_max, smem_bad);
    if (!active) return;

    float scale = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 127.0f);
    scale = fmaxf(scale, 1.1754943508222875e-38f);
    if (t == 0) {
        row_scales[row] = bad ? __int_as_float(0x7fc00000) : scale;
        if (valid) valid[row] = bad ? 0 : 1;
    }
    uint32_t* out = reinterpret_cast<uint32_t*>(q + (size_t)row * ldq);
    const uint32_t nwords = ldq / 4;
    const RowDivisor div(scale);
    if constexpr (CACHE) {
        if (div.fast && !bad) {
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const uint32_t v = t + i * THREADS_PER_ROW;
                if (v < nwords) out[v] = v < nvec ? pack4t<true>(cache[i], div) : 0u;
            }
        } else {
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const uint32_t v = t + i * THREADS_PER_ROW;
                if (v < nwords) out[v] = (v < nvec && !bad) ? pack4t<false>(cache[i], div) : 0u;
            }
        }
        for (uint32_t v = t + kMaxVecPerThread * THREADS_PER_ROW; v < nwords; v += THREADS_PER_ROW) out[v] = 0u;
    } else {
        for (uint32_t v = t; v < nwords; v += THREADS_PER_ROW)
            out[v] = (v < nvec && !bad) ? pack4(__ldg(in + v), div) : 0u;
    }
}

// Few rows (decode): one row per CTA leaves most of the GPU idle and makes the kernel a chain of
// dependent loads. Here a thread-block cluster of S CTAs shares a row: each CTA keeps its K/S
// slice in registers (at most 8 float4 per thread), the S partial (absmax, non-finite) pairs
// are exchanged through distributed shared memory, and every CTA quantizes its own slice.
// grid = (S, rows), cluster = (S, 1, 1). max and OR are exact in any order, so the result is
// bit-identical to the one-CTA kernel.
template <int S>
__global__ void __launch_bounds__(kThreads)
quantize_rows_cluster(const float* __restrict__ x, uint32_t rows, uint32_t k, int8_t* __restrict__ q,
                      uint32_t ldq, float* __restrict__ row_scales, int32_t* __restrict__ valid, bool early) {
    namespace cg = cooperative_groups;
    __shared__ float smem_max[kThreads / 32];
    __shared__ int smem_bad[kThreads / 32];
    __shared__ float peer_max[S];
    __shared__ int peer_bad[S];
    wait_and_release(early);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const uint32_t row = blockIdx.y;
    const uint32_t nvec = k / 4, nwords = ldq / 4;
    const uint32_t seg = (nwords + S - 1) / S;                 // words (= float4s) of this CTA's slice
    const uint32_t w0 = rank * seg;
    const float4* in = reinterpret_cast<const float4*>(x + (size_t)row * k);

    float4 cache[kMaxVecPerThread];
    float amax = 0.0f; int bad = 0;
#pragma unroll
    for (int i = 0; i < kMaxVecPerThread; i++) {
        const uint32_t o = threadIdx.x + i * kThreads, v = w0 + o;
        cache[i] = (o < seg && v < nvec) ? __ldg(in + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < kMaxVecPerThread; i++) {
        const float4 c = cache[i];
        bad |= nonfinite_bits(c.x) | nonfinite_bits(c.y) | nonfinite_bits(c.z) | nonfinite_bits(c.w);
        amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(c.z), fabsf(c.w))));
    }
    row_reduce<kThreads>(amax, bad, smem_max, smem_bad);
    if (threadIdx.x < S) {
        // thread p publishes this CTA's pair in CTA p's table
        *cluster.map_shared_rank(&peer_max[rank], threadIdx.x) = amax;
        *cluster.map_shared_rank(&peer_bad[rank], threadIdx.x) = bad;
    }
    cluster.sync();
    amax = 0.0f; bad = 0;
#pragma unroll
    for (int p = 0; p < S; p++) { amax = fmaxf(amax, peer_max[p]); bad |= peer_bad[p]; }

    float scale = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 127.0f);
    scale = fmaxf(scale, 1.1754943508222875e-38f);
    if (rank == 0 && threadIdx.x == 0) {
        row_scales[row] = bad ? __int_as_float(0x7fc00000) : scale;
        if (valid) valid[row] = bad ? 0 : 1;
    }
    uint32_t* out = reinterpret_cast<uint32_t*>(q + (size_t)row * ldq);
    const RowDivisor div(scale);
    const bool fast = div.fast && !bad;
#pragma unroll
    for (int i = 0; i < kMaxVecPerThread; i++) {
        const uint32_t o = threadIdx.x + i * kThreads, v = w0 + o;
        if (o < seg && v < nwords)
            out[v] = (v < nvec && !bad) ? (fast ? pack4t<true>(cache[i], div) : pack4t<false>(cache[i], div)) : 0u;
    }
}

template <int S>
cudaError_t launch_cluster(const float* x, uint32_t rows, uint32_t k, int8_t* q, uint32_t ldq,
                           float* row_scales, int32_t* valid, cudaStream_t stream, bool early) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S, rows); cfg.blockDim = dim3(kThreads); cfg.dynamicSmemBytes = 0; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, quantize_rows_cluster<S>, x, rows, k, q, ldq, row_scales, valid, early);
}

// Any k, any alignment: thread t of a row's THREADS_PER_ROW takes the elements t, t + THREADS_PER_ROW, ..., so
// that every load instruction covers 128 consecutive bytes per warp and every (byte) store a whole sector of the
// padded code row, whatever the row's first byte is.  PER: at most so many elements per thread, which stay in registers
// between the absmax and the quantizing pass; 0: rows of more than 8192 elements, read twice.  Alone, one warp per row that
// reads it twice / 32 elements per thread for every width, which a narrow row paid for / the width's own number: 4096 x
// 4099 64.8 / 24.7 / 24.7 us, 777 x 1283 6.3 / 5.7 / 3.4, 2048 x 576 6.1 / 7.1 / 3.5, 4096 x 128 3.3 / 5.2 / 1.9.
constexpr int kMaxPerThread = 4 * kMaxVecPerThread;
template <int THREADS_PER_ROW, int PER>
__global__ void __launch_bounds__(kThreads)
quantize_rows_any(const float* __restrict__ x, uint32_t rows, uint32_t k, int8_t* __restrict__ q,
                  uint32_t ldq, float* __restrict__ row_scales, int32_t* __restrict__ valid, bool early) {
    __shared__ float smem_max[kThreads / 32];
    __shared__ int smem_bad[kThreads / 32];
    wait_and_release(early);
    constexpr uint32_t kRowsPerCta = kThreads / THREADS_PER_ROW;
    const uint32_t row = blockIdx.x * kRowsPerCta + threadIdx.x / THREADS_PER_ROW;
    const uint32_t t = threadIdx.x % THREADS_PER_ROW;
    const bool active = row < rows;
    const float* in = x + (size_t)(active ? row : 0) * k;

    float cache[PER ? PER : 1];
    float amax = 0.0f; int bad = 0;
    if (active) {
        if constexpr (PER != 0) {
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const uint32_t j = t + i * THREADS_PER_ROW;
                cache[i] = j < k ? __ldg(in + j) : 0.0f;
            }
#pragma unroll
            for (int i = 0; i < PER; i++) {
                bad |= nonfinite_bits(cache[i]);
                amax = fmaxf(amax, fabsf(cache[i]));
            }
        } else {
#pragma unroll 8
            for (uint32_t j = t; j < k; j += THREADS_PER_ROW) {
                const float v = __ldg(in + j);
                bad |= nonfinite_bits(v);
                amax = fmaxf(amax, fabsf(v));
            }
        }
    }
    row_reduce<THREADS_PER_ROW>(amax, bad, smem_max, smem_bad);
    if (!active) return;

    const float scale = row_scale_from_amax(amax);
    if (t == 0) {
        row_scales[row] = bad ? __int_as_float(0x7fc00000) : scale;
        if (valid) valid[row] = bad ? 0 : 1;
    }
    int8_t* out = q + (size_t)row * ldq;
    const RowDivisor div(scale);
    uint32_t done = 0;
    if constexpr (PER != 0) {
        if (div.fast && !bad) {
            const uint64_t rcp2 = f32x2(div.rcp, div.rcp), neg_d2 = f32x2(-div.scale, -div.scale);
#pragma unroll
            for (int i = 0; i < PER; i += 2) {
                const uint32_t j = t + i * THREADS_PER_ROW;
                int32_t a, b;
                quant2_fast(cache[i], cache[i + 1], rcp2, neg_d2, a, b);   // zero past the row's end: code 0
                if (j < ldq) out[j] = (int8_t)a;
                if (j + THREADS_PER_ROW < ldq) out[j + THREADS_PER_ROW] = (int8_t)b;
            }
        } else {
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const uint32_t j = t + i * THREADS_PER_ROW;
                if (j < ldq) out[j] = (j < k && !bad) ? (int8_t)quant1<false>(cache[i], div) : (int8_t)0;
            }
        }
        done = PER * THREADS_PER_ROW;
    }
#pragma unroll 8
    for (uint32_t j = done + t; j < ldq; j += THREADS_PER_ROW)
        out[j] = (j < k && !bad) ? (int8_t)(div.fast ? quant1<true>(__ldg(in + j), div) : quant1<false>(__ldg(in + j), div)) : (int8_t)0;
}

// Sixteen output bytes per thread; VEC: rows of whole 16-byte pieces, read as such.
template <bool VEC>
__global__ void __launch_bounds__(kThreads)
copy_bytes_padded_kernel(const uint8_t* __restrict__ src, uint32_t rows, uint32_t k, uint8_t* __restrict__ dst,
                         uint32_t ld, uint32_t xor_mask) {
    pdl_wait();
    pdl_release();
    const uint32_t per_row = ld / 16u;
    const uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    const uint32_t row = (uint32_t)(i / per_row), at = (uint32_t)(i - (uint64_t)row * per_row) * 16u;
    if (row >= rows) return;
    const uint8_t* in = src + (size_t)row * k + at;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if constexpr (VEC) {
        if (at < k) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(in));
            const uint32_t m = xor_mask * 0x01010101u;
            w[0] = v.x ^ m; w[1] = v.y ^ m; w[2] = v.z ^ m; w[3] = v.w ^ m;
        }
    } else {
#pragma unroll
        for (uint32_t j = 0; j < 16; j++)
            if (at + j < k) w[j >> 2] |= (uint32_t)(uint8_t)(__ldg(in + j) ^ xor_mask) << (8u * (j & 3u));
    }
    *reinterpret_cast<uint4*>(dst + (size_t)row * ld + at) = make_uint4(w[0], w[1], w[2], w[3]);
}

// One warp per weight row: copy (with optional ^0x80), zero the padding, sum the codes.
__global__ void __launch_bounds__(kThreads)
repack_weight_kernel(const uint8_t* __restrict__ src, uint32_t src_ld, uint32_t n, uint32_t k,
                     uint32_t xor_mask, int8_t* __restrict__ dst, uint32_t kpad,
                     int32_t* __restrict__ wsum) {
    const uint32_t row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= n) return;
    const uint8_t* in = src + (size_t)row * src_ld;
    int8_t* out = dst + (size_t)row * kpad;
    int32_t sum = 0;
    for (uint32_t j = lane; j < kpad; j += 32) {
        const int8_t v = j < k ? (int8_t)(in[j] ^ xor_mask) : (int8_t)0;
        out[j] = v;
        sum += v;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (lane == 0) wsum[row] = sum;
}

template <int TPR>
cudaError_t launch_vec(const float* x, uint32_t rows, uint32_t k, int8_t* q, uint32_t ldq,
                       float* row_scales, int32_t* valid, cudaStream_t stream, bool early) {
    constexpr int kRowsPerCta = kThreads / TPR;
    const uint32_t grid = (rows + kRowsPerCta - 1) / kRowsPerCta;
    if (k / 4 <= (uint32_t)TPR * kMaxVecPerThread)
        return launch_pdl(quantize_rows_vec<TPR, true>, dim3(grid), dim3(kThreads), 0, stream,
                          x, rows, k, q, ldq, row_scales, valid, early);
    return launch_pdl(quantize_rows_vec<TPR, false>, dim3(grid), dim3(kThreads), 0, stream,
                      x, rows, k, q, ldq, row_scales, valid, early);
}

template <int TPR, int PER>
cudaError_t launch_any_per(const float* x, uint32_t rows, uint32_t k, int8_t* q, uint32_t ldq,
                           float* row_scales, int32_t* valid, cudaStream_t stream, bool early) {
    constexpr uint32_t kRowsPerCta = kThreads / TPR;
    return launch_pdl(quantize_rows_any<TPR, PER>, dim3((rows + kRowsPerCta - 1) / kRowsPerCta), dim3(kThreads), 0, stream,
                      x, rows, k, q, ldq, row_scales, valid, early);
}
template <int TPR>
cudaError_t launch_any(const float* x, uint32_t rows, uint32_t k, int8_t* q, uint32_t ldq,
                       float* row_scales, int32_t* valid, cudaStream_t stream, bool early) {
    if (k <= (uint32_t)TPR * 4) return launch_any_per<TPR, 4>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    if (k <= (uint32_t)TPR * 8) return launch_any_per<TPR, 8>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    if (k <= (uint32_t)TPR * 16) return launch_any_per<TPR, 16>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    if (k <= (uint32_t)TPR * kMaxPerThread) return launch_any_per<TPR, kMaxPerThread>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    return launch_any_per<kThreads, 0>(x, rows, k, q, ldq, row_scales, valid, stream, early);   // (TPR is kThreads then)
}


// ---- RMSNorm folded into the quantizer --------------------------------------------------------
// The decode and prefill patterns RMSNorm -> {q,k,v} and RMSNorm -> {gate,up} read the residual
// stream once: normalize, (optionally) persist the normalized row for other consumers, quantize.
// Arithmetic of the normalization follows the reference's CPU operator
// (native/src/kernels/softmax_rmsnorm.inc:3-16): squares and their mean in double,
// inv = 1 / sqrt(mean + eps) in double, y = float((double(x) * inv) * double(gamma)).  The squares
// are exact in double; only the order of the double additions differs from the sequential loop
// (tree instead of left to right), which moves the mean by at most a few units of 2^-53.

template <int THREADS_PER_ROW>
__device__ __forceinline__ double row_sum(double v, double* smem_sum) {
    constexpr int kWarpSpan = THREADS_PER_ROW < 32 ? THREADS_PER_ROW : 32;
#pragma unroll
    for (int off = kWarpSpan / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if constexpr (THREADS_PER_ROW > 32) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (lane == 0) smem_sum[warp] = v;
        __syncthreads();
        constexpr int kWarps = THREADS_PER_ROW / 32;
        const int first = (threadIdx.x / THREADS_PER_ROW) * kWarps;
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < kWarps; i++) s += smem_sum[first + i];
        v = s;
    }
    return v;
}

template <int THREADS_PER_ROW, bool CACHE>
__global__ void __launch_bounds__(kThreads)
rmsnorm_quantize_rows_vec(const float* __restrict__ x, const float* __restrict__ gamma, double eps,
                          uint32_t rows, uint32_t k, float* __restrict__ norm_out, int8_t* __restrict__ q,
                          uint32_t ldq, float* __restrict__ row_scales, int32_t* __restrict__ valid) {
    __shared__ float smem_max[kThreads / 32];
    __shared__ int smem_bad[kThreads / 32];
    __shared__ double smem_sum[kThreads / 32];
    pdl_wait();
    pdl_release();
    constexpr int kRowsPerCta = kThreads / THREADS_PER_ROW;
    const uint32_t row = blockIdx.x * kRowsPerCta + threadIdx.x / THREADS_PER_ROW;
    const int t = threadIdx.x % THREADS_PER_ROW;
    const bool active = row < rows;
    const uint32_t nvec = k / 4;
    const float4* in = reinterpret_cast<const float4*>(x + (size_t)(active ? row : 0) * k);
    const float4* g4 = reinterpret_cast<const float4*>(gamma);
    float4* nout = norm_out ? reinterpret_cast<float4*>(norm_out + (size_t)(active ? row : 0) * k) : nullptr;

    float4 cache[CACHE ? kMaxVecPerThread : 1];
    double ss = 0.0, ss2 = 0.0;
    if (active) {
        if constexpr (CACHE) {
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const uint32_t v = t + i * THREADS_PER_ROW;
                cache[i] = v < nvec ? __ldg(in + v) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i += 2) {   // two chains of double additions
                ss = square_sum4(cache[i], ss);
                ss2 = square_sum4(cache[i + 1], ss2);
            }
            ss += ss2;
        } else {
            for (uint32_t v = t; v < nvec; v += THREADS_PER_ROW) ss = square_sum4(__ldg(in + v), ss);
        }
    }
    ss = row_sum<THREADS_PER_ROW>(ss, smem_sum);
    // one thread per row does the double-precision division and square root (slow, shared units); the others
    // take the result from shared memory
    __shared__ double smem_inv[kThreads / 8];
    if (t == 0) smem_inv[threadIdx.x / THREADS_PER_ROW] = row_inverse(ss, k, eps);
    if constexpr (THREADS_PER_ROW > 32) __syncthreads(); else __syncwarp();
    const double inv = smem_inv[threadIdx.x / THREADS_PER_ROW];

    float amax = 0.0f; int bad = 0;
    if (active) {
        if constexpr (CACHE) {
#pragma unroll
            for (int i = 0; i < kMaxVecPerThread; i++) {
                const uint32_t v = t + i * THREADS_PER_ROW;
                if (v < nvec) {
                    const float4 c = norm4(cache[i], inv, __ldg(g4 + v));
                    cache[i] = c;
                    if (nout) nout[v] = c;
                    bad |= nonfinite_bits(c.x) | nonfinite_bits(c.y) | nonfinite_bits(c.z) | nonfinite_bits(c.w);
                    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(c.z), fabsf(c.w))));
                }
            }
        } else {
            for (uint32_t v = t; v < nvec; v += THREADS_PER_ROW) {
                const float4 c = norm4(__ldg(in + v), inv, __ldg(g4 + v));
                if (nout) nout[v] = c;
                bad |= nonfinite_bits(c.x) | nonfinite_bits(c.y) | nonfinite_bits(c.z) | nonfinite_bits(c.w);
                amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(c.z), fabsf(c.w))));
            }
        }
    }
    row_reduce<THREADS_PER_ROW>(amax, bad, smem_max, smem_bad);
    if (!active) return;

    float scale = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 127.0f);
    scale = fmaxf(scale, 1.1754943508222875e-38f);
    if (t == 0) {
        row_scales[row] = bad ? __int_as_float(0x7fc00000) : scale;
        if (valid) valid[row] = bad ? 0 : 1;
    }
    uint32_t* out = reinterpret_cast<uint32_t*>(q + (size_t)row * ldq);
    const uint32_t nwords = ldq / 4;
    const RowDivisor div(scale);
    if constexpr (CACHE) {
        const bool fast = div.fast && !bad;
#pragma unroll
        for (int i = 0; i < kMaxVecPerThread; i++) {
            const uint32_t v = t + i * THREADS_PER_ROW;
            if (v < nwords)
                out[v] = (v < nvec && !bad) ? (fast ? pack4t<true>(cache[i], div) : pack4t<false>(cache[i], div)) : 0u;
        }
        for (uint32_t v = t + kMaxVecPerThread * THREADS_PER_ROW; v < nwords; v += THREADS_PER_ROW) out[v] = 0u;
    } else {
        for (uint32_t v = t; v < nwords; v += THREADS_PER_ROW)
            out[v] = (v < nvec && !bad) ? pack4(norm4(__ldg(in + v), inv, __ldg(g4 + v)), div) : 0u;
    }
}

// Any k / alignment: one warp per row, scalar accesses, the row is read three times.
__global__ void __launch_bounds__(kThreads)
rmsnorm_quantize_rows_scalar(const float* __restrict__ x, const float* __restrict__ gamma, double eps,
                             uint32_t rows, uint32_t k, float* __restrict__ norm_out, int8_t* __restrict__ q,
                             uint32_t ldq, float* __restrict__ row_scales, int32_t* __restrict__ valid) {
    pdl_wait();
    pdl_release();
    const uint32_t row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* in = x + (size_t)row * k;
    double ss = 0.0;
    for (uint32_t j = lane; j < k; j += 32) ss = __fma_rn((double)in[j], (double)in[j], ss);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const double inv = row_inverse(ss, k, eps);
    float amax = 0.0f; int bad = 0;
    for (uint32_t j = lane; j < k; j += 32) {
        const float v = norm1(in[j], inv, gamma[j]);
        if (norm_out) norm_out[(size_t)row * k + j] = v;
        bad |= nonfinite_bits(v);
        amax = fmaxf(amax, fabsf(v));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        bad |= __shfl_xor_sync(0xffffffffu, bad, off);
    }
    float scale = amax == 0.0f ? 1.0f : __fdiv_rn(amax, 127.0f);
    scale = fmaxf(scale, 1.1754943508222875e-38f);
    if (lane == 0) {
        row_scales[row] = bad ? __int_as_float(0x7fc00000) : scale;
        if (valid) valid[row] = bad ? 0 : 1;
    }
    int8_t* out = q + (size_t)row * ldq;
    const RowDivisor div(scale);
    for (uint32_t j = lane; j < ldq; j += 32)
        out[j] = (j < k && !bad) ? (int8_t)quant1<false>(norm1(in[j], inv, gamma[j]), div) : (int8_t)0;
}

template <int TPR>
cudaError_t launch_norm_vec(const float* x, const float* gamma, double eps, uint32_t rows, uint32_t k,
                            float* norm_out, int8_t* q, uint32_t ldq, float* row_scales, int32_t* valid,
                            cudaStream_t stream) {
    constexpr int kRowsPerCta = kThreads / TPR;
    const uint32_t grid = (rows + kRowsPerCta - 1) / kRowsPerCta;
    if (k / 4 <= (uint32_t)TPR * kMaxVecPerThread)
        return launch_pdl(rmsnorm_quantize_rows_vec<TPR, true>, dim3(grid), dim3(kThreads), 0, stream,
                          x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid);
    return launch_pdl(rmsnorm_quantize_rows_vec<TPR, false>, dim3(grid), dim3(kThreads), 0, stream,
                      x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid);
}

}  // namespace

// Threads per row: enough that a thread holds at most 32 elements, then doubled while the whole launch has fewer
// threads than half the chip's resident ones and every thread keeps at least 4 elements.
uint32_t quantize_any_threads(uint32_t rows, uint32_t k) {
    uint32_t tpr = 32;
    while (tpr < (uint32_t)kThreads && k > tpr * kMaxPerThread) tpr *= 2;
    while (tpr < (uint32_t)kThreads && (uint64_t)rows * tpr < 148u * 1024u && k >= 8u * tpr) tpr *= 2;
    return tpr;
}

// ... with 128-bit loads: at most 8 float4 per thread, then doubled (from 8 to 32) while the whole launch stays within 256
// threads per SM and every thread keeps a float4, or within 1024 per SM and it keeps four (two at K up to 256); with the
// RMSNorm's longer row within 512 per SM.  Chosen by the whole call (us, rows from memory, N = 2048): shorter shares cost row
// reductions and blocks (300 x 1024 with 256 threads per row 10.4, with 64 10.2; 777 x 576 with 128 9.9, with 32 9.5; 1024 x
// 256 with 64 8.7, with 32 8.1), fewer threads leave the GEMM's first loads beside rows still to come (2048 x 1024 with 64
// 12.4, with 32 13.5; 4096 x 256 with 32 12.5, with 8 14.5; 1024 x 2048 with 128 13.8, with 64 14.7), although the quantizer
// alone is then faster.  With the norm, alone: 64 x 1024 with 32 and 256 threads 4.9 and 2.7, 512 x 1024 with 256 4.2, with 128
// 3.3.
uint32_t quantize_vec_threads(uint32_t rows, uint32_t k, bool norm) {
    const uint64_t few = 148u * (norm ? 512u : 256u), most = norm ? few : 148u * 1024u;
    uint32_t tpr = k <= 256 ? 8 : k <= 1024 ? 32 : k <= 2048 ? 64 : k <= 4096 ? 128 : 256;
    for (;;) {
        const uint32_t next = tpr == 8 ? 32u : 2u * tpr;
        const uint64_t threads = (uint64_t)rows * next;
        const uint32_t keep = threads <= few ? 1u : k <= 256 ? 2u : 4u;
        if (next > (uint32_t)kThreads || threads > most || k / 4u < keep * next) return tpr;
        tpr = next;
    }
}

cudaError_t launch_quantize_rows(const float* x, uint32_t rows, uint32_t k, int8_t* q, uint32_t ldq,
                                 float* row_scales, int32_t* valid, cudaStream_t stream, bool early) {
    if (rows == 0) return cudaSuccess;
    const bool vec = (k % 4 == 0) && (ldq % 4 == 0) && ((uintptr_t)x % 16 == 0) && ((uintptr_t)q % 4 == 0);
    if (!vec) {
        // one warp per row where that alone fills the chip, more threads per row (and loads in flight) otherwise
        const uint32_t tpr = quantize_any_threads(rows, k);
        if (tpr == 32) return launch_any<32>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        if (tpr == 64) return launch_any<64>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        if (tpr == 128) return launch_any<128>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        return launch_any<256>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    }
    // Few long rows: a cluster of 2..8 CTAs per row (each thread then holds one or two float4)
    if (rows <= kClusterMaxRows && ldq / 4 >= 2u * kThreads && ldq / 4 <= 8u * kThreads * kMaxVecPerThread) {
        const uint32_t per = (ldq / 4 + kThreads - 1) / kThreads;   // float4 per thread with one CTA
        if (per >= 8) return launch_cluster<8>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        if (per >= 4) return launch_cluster<4>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        return launch_cluster<2>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    }
    switch (quantize_vec_threads(rows, k)) {
        case 8: return launch_vec<8>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        case 32: return launch_vec<32>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        case 64: return launch_vec<64>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        case 128: return launch_vec<128>(x, rows, k, q, ldq, row_scales, valid, stream, early);
        default: return launch_vec<256>(x, rows, k, q, ldq, row_scales, valid, stream, early);
    }
}

cudaError_t launch_rmsnorm_quantize_rows(const float* x, const float* gamma, float epsilon, uint32_t rows,
                                         uint32_t k, float* norm_out, int8_t* q, uint32_t ldq,
                                         float* row_scales, int32_t* valid, cudaStream_t stream) {
    if (rows == 0) return cudaSuccess;
    const double eps = (double)epsilon;
    const bool vec = (k % 4 == 0) && (ldq % 4 == 0) && ((uintptr_t)x % 16 == 0) && ((uintptr_t)gamma % 16 == 0) &&
                     ((uintptr_t)norm_out % 16 == 0) && ((uintptr_t)q % 4 == 0);
    if (!vec) {
        const uint32_t grid = (rows + kThreads / 32 - 1) / (kThreads / 32);
        return launch_pdl(rmsnorm_quantize_rows_scalar, dim3(grid), dim3(kThreads), 0, stream,
                          x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid);
    }
    switch (quantize_vec_threads(rows, k, true)) {
        case 8: return launch_norm_vec<8>(x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid, stream);
        case 32: return launch_norm_vec<32>(x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid, stream);
        case 64: return launch_norm_vec<64>(x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid, stream);
        case 128: return launch_norm_vec<128>(x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid, stream);
        default: return launch_norm_vec<256>(x, gamma, eps, rows, k, norm_out, q, ldq, row_scales, valid, stream);
    }
}

cudaError_t launch_copy_bytes_padded(const uint8_t* src, uint32_t rows, uint32_t k, uint8_t* dst,
                                     uint32_t ld, uint32_t xor_mask, cudaStream_t stream) {
    if (!rows) return cudaSuccess;
    if (ld % 16u || ((uintptr_t)dst & 15u)) return cudaErrorInvalidValue;
    const uint32_t grid = (uint32_t)(((uint64_t)rows * (ld / 16u) + kThreads - 1) / kThreads);
    if (k % 16u == 0 && ((uintptr_t)src & 15u) == 0)
        return launch_pdl(copy_bytes_padded_kernel<true>, dim3(grid), dim3(kThreads), 0, stream, src, rows, k, dst, ld, xor_mask);
    return launch_pdl(copy_bytes_padded_kernel<false>, dim3(grid), dim3(kThreads), 0, stream, src, rows, k, dst, ld, xor_mask);
}

cudaError_t launch_repack_weight(const uint8_t* src, uint32_t src_ld, uint32_t n, uint32_t k,
                                 uint32_t xor_mask, int8_t* dst, uint32_t kpad, int32_t* wsum,
                                 cudaStream_t stream) {
    if (!n) return cudaSuccess;
    const uint32_t grid = (n + kThreads / 32 - 1) / (kThreads / 32);
    repack_weight_kernel<<<grid, kThreads, 0, stream>>>(src, src_ld, n, k, xor_mask, dst, kpad, wsum);
    return cudaGetLastError();
}

}  // namespace vxb
