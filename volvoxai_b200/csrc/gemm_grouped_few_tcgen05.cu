// K2f: weights with grouped scales and FEW token rows (batched decode, up to 64 rows), on the tensor cores.
//
//   y[m,n] = (sum over groups g, ascending, of f32(dot_g[m,n]) * f32(as[m] * ws[n,g])) + bias[n]
//
// The arithmetic is the grouped GEMM's (gemm_grouped_tcgen05.cu), every product and sum rounded on its own; what
// differs is who is who.  The weights are the UMMA M operand (128 or 64 channels, one per TMEM lane) and the tokens
// the N operand (16 .. 64 columns; up to 8 tokens only the first 8 are drained), so that every lane of every drain warp owns a channel and a group costs a warp
// five instructions per token.  With the tokens as M (the large kernel), 8 tokens left two of eight warps to drain
// 128 columns for 32 lanes, 24 of them dead, group after group.  Whole call, quantizer included, G = 128: 8 x 4096 ->
// 14336 15.5 us (30.8 before, both without what Python adds; the weights alone take 9.0 at the measured copy rate),
// 8 x 4096 -> 4096 9.7 (27.3), 64 x 4096 -> 14336 18.9 (28.2).
//
// A stage is 256 bytes of K: one TMA box of weights ([2 K blocks][channels x 128 B]), one of activations, one commit,
// and the 1 .. 8 groups that lie in it, each in accumulator columns of its own, drained together.  The ring of a CTA holds
// about 200 KB, which is what keeps the HBM stream going, half of that in the form below that leaves room for a second CTA.
//
//   warp 0        TMA producer, activations (waits for the launch before this one)
//   warp 1        allocates TMEM; one lane issues the MMAs (of the short tiles every other stage's; another warp the rest)
//   warps 2..     drain: one per TMEM lane quarter (two for 64 tokens, 32 tokens each)
//   next warp     TMA producer, weights (waits for nothing)
//
// Channels per tile: 128; 64 where the tiles of 128 would leave half of the SMs without one (an MMA takes its 128 or 64
// clocks whatever the token count, so a tile of 128 channels and K = 4096 is 8.6 us of tensor pipe, of 64 half that).
// Every wait on an mbarrier is bounded; on expiry the kernel raises the status word, drains, frees its TMEM and
// returns.
#include "tcgen05.cuh"

namespace vxb {

namespace {

using namespace tc;

constexpr uint32_t kSpan = 128, kSpans = 2;   // K bytes of a swizzle span, spans per stage
constexpr uint32_t kMaxStages = 12, kMaxBufs = 4;

// BM channels per tile, LT live token slots, MPG MMAs (32 bytes of K) per group
template <uint32_t BM, uint32_t LT, uint32_t MPG> struct Few {
    static constexpr uint32_t NT = LT < 16 ? 16 : LT;               // token columns of the MMA
    // Up to 16 tokens of 128-channel tiles two CTAs fit an SM (half of its shared memory and TMEM each).  Between launches
    // of prepared activations the next one's CTAs so start their weights while this launch drains.  Behind a row quantizer
    // the GEMM before it has ended when this one starts, and half the ring is still the faster form; us from a graph / in a
    // stream, this and the whole SM's ring per CTA: 8 x 4096 -> 14336 16.1/16.3 and 16.3/17.2, 16 x 4096 -> 14336 17.8/18.0
    // and 18.6/18.9, 8 x 4096 -> 14336 at G = 32 19.5/19.9 and 20.7/21.2, 5 x 2048 -> 11008 9.1/9.8 and 9.2/9.9,
    // 8 x 8192 -> 28672 51.4/52.2 and 51.4/52.0.  The short tiles want the deep ring (8 x 4096 -> 4096 13.7 us, 14.6 with
    // half of it).
    static constexpr bool kTwo = BM == 128 && LT <= 16;
    static constexpr uint32_t kCtas = kTwo ? 2 : 1, kTmemCols = kTwo ? 256 : 512, kSmemBudget = (kTwo ? 110 : 216) * 1024;
    static constexpr uint32_t kDrainWarps = NT == 64 ? 8 : 4;
    static constexpr uint32_t kTokens = LT * 4 / kDrainWarps;       // tokens per drain thread
    static constexpr uint32_t kWBytes = kSpans * BM * kSpan, kXBytes = kSpans * NT * kSpan, kStageBytes = kWBytes + kXBytes;
    static constexpr uint32_t kGroups = 8 / MPG;                    // groups per stage
    // Stages whose scales are requested ahead: a stage of 64 channels lasts 0.3 us, of 128 twice that, a scale from memory
    // up to one (8 x 14336 -> 4096: 40.1 us one stage ahead, 23.6 four ahead; 8 x 4096 -> 14336 16.4, 15.5).  Where a
    // stage is long and its drain is too (64 tokens 18.9 us, 20.3 four ahead; eight groups 18.8, 19.7) one is enough.
    static constexpr uint32_t kAhead = BM == 64 ? (kGroups >= 8 ? 2 : 4) : LT <= 8 && kGroups <= 4 ? 4 : 1;
    static constexpr uint32_t kAccCols = NT * kGroups;
    static constexpr uint32_t kBufs = kTmemCols / kAccCols < kMaxBufs ? kTmemCols / kAccCols : kMaxBufs;
    // Short tiles: two threads issue, stage by stage in turn (a thread starts an MMA every hundred clocks or so, and
    // one of 64 rows is done in 64).  Stages and accumulators then come in even numbers, so that each belongs to one
    // of them: a parity wait means something only to a waiter that saw the phase before.
    static constexpr uint32_t kIssuers = BM == 64 && kBufs % 2 == 0 ? 2 : 1;
    static constexpr uint32_t kWWarp = 2 + kDrainWarps;
    static constexpr uint32_t kThreads = 32 * (kWWarp + kIssuers);  // the second issuer is the last warp
    static constexpr uint32_t kFit = kSmemBudget / kStageBytes;
    static constexpr uint32_t kStages = (kFit < kMaxStages ? kFit : kMaxStages) / kIssuers * kIssuers;
    static constexpr uint32_t kOffBars = kStages * kStageBytes;
    static constexpr uint32_t kNumBars = 2 * kStages + 2 * kBufs;
    static constexpr uint32_t kOffTmemPtr = kOffBars + kNumBars * 8;
    static constexpr uint32_t kOffAbort = kOffTmemPtr + 4;
    static constexpr uint32_t kSmemBytes = kOffAbort + 8 + 1024;
    static_assert(kSmemBytes <= 227 * 1024 && kStages >= 2 && kBufs >= 1 && kStages % kIssuers == 0, "launch shape");
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_tokens(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
__device__ __forceinline__ void tmem_ld_tokens(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld_tokens(uint32_t taddr, uint32_t (&r)[32]) { tmem_ld32(taddr, r); }

template <uint32_t BM, uint32_t LT, uint32_t MPG>
__global__ void __launch_bounds__(Few<BM, LT, MPG>::kThreads, Few<BM, LT, MPG>::kCtas)
gemm_i8_grouped_few_kernel(const __grid_constant__ GemmGroupedArgs args) {
    using C = Few<BM, LT, MPG>;
    constexpr uint32_t NT = C::NT;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto w_addr = [&](uint32_t s) { return smem_u32(base + s * C::kStageBytes); };
    auto full = [&](uint32_t s) { return smem_u32(base + C::kOffBars + s * 8); };
    auto empty = [&](uint32_t s) { return smem_u32(base + C::kOffBars + (C::kStages + s) * 8); };
    auto tmem_full = [&](uint32_t b) { return smem_u32(base + C::kOffBars + (2 * C::kStages + b) * 8); };
    auto tmem_empty = [&](uint32_t b) { return smem_u32(base + C::kOffBars + (2 * C::kStages + C::kBufs + b) * 8); };
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(base + C::kOffTmemPtr);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base + C::kOffAbort);

    const uint32_t tiles = (args.n + BM - 1) / BM;
    const uint32_t all_ks = args.kpad / 32u;
    const uint32_t total_ks = all_ks < args.groups * MPG ? all_ks : args.groups * MPG;
    const uint32_t num_kb = (total_ks + 7u) / 8u;                   // stages per tile

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < C::kStages; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (uint32_t b = 0; b < C::kBufs; b++) { mbar_init(tmem_full(b), 1); mbar_init(tmem_empty(b), C::kDrainWarps); }
        arm_abort(abort_flag, args.status);
        fence_barrier_init();
        prefetch_tmap(&args.tmap_a);
        prefetch_tmap(&args.tmap_b);
        pdl_release();   // the next launch in the stream may begin its own prologue
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_ptr), C::kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_ptr;

    if (warp == 0 || warp == C::kWWarp) {
        // ---------------- TMA producers ----------------
        if (lane == 0) {
            const bool weights = warp != 0;
            uint32_t stage = 0, phase = 0, armed = 0, armed_parity = 0;
            bool ok = true;
            if (!weights) pdl_wait();   // the activations come from the launch before this one
            for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
                for (uint32_t kb = 0; kb < num_kb; kb++) {
                    if (!mbar_wait(empty(stage), phase ^ 1u, abort_flag)) { ok = false; break; }
                    if (weights) {
                        tma_load_3d(w_addr(stage), &args.tmap_b, full(stage), 0, (int32_t)(t * BM), (int32_t)(kb * kSpans));
                    } else {
                        mbar_expect_tx(full(stage), C::kStageBytes);
                        tma_load_3d(w_addr(stage) + C::kWBytes, &args.tmap_a, full(stage), 0, 0, (int32_t)(kb * kSpans));
                        armed |= 1u << stage;
                        armed_parity = (armed_parity & ~(1u << stage)) | (phase << stage);
                    }
                    if (++stage == C::kStages) { stage = 0; phase ^= 1u; }
                }
            }
            if (!ok && !weights) {
                // drain: give this CTA's own copies in flight a bounded time to land
                for (uint32_t s = 0; s < C::kStages; s++) {
                    if (!(armed & (1u << s))) continue;
                    for (uint32_t i = 0; i < 2000; i++) {
                        if (mbar_try_wait(full(s), (armed_parity >> s) & 1u)) break;
                        __nanosleep(500);
                    }
                }
            }
        }
    } else if (warp == 1 || warp > C::kWWarp) {
        // ---------------- MMA issuers: stages `me`, me + kIssuers, ... of this CTA's ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = make_idesc(BM, NT);
            const uint32_t me = warp == 1 ? 0u : 1u;
            uint32_t stage = me, phase = 0, buf = me, buf_phase = 0, kb = me;
            for (uint32_t t = blockIdx.x;;) {
                while (kb >= num_kb) { kb -= num_kb; t += gridDim.x; }
                if (t >= tiles) break;
                if (!mbar_wait(tmem_empty(buf), buf_phase ^ 1u, abort_flag)) break;
                if (!mbar_try_wait(full(stage), phase) && !mbar_wait(full(stage), phase, abort_flag)) break;
                tc_fence_after();
                const uint32_t w_lo = smem_desc_lo(w_addr(stage)), x_lo = smem_desc_lo(w_addr(stage) + C::kWBytes);
                const uint32_t left = total_ks - kb * 8u;
#pragma unroll
                for (uint32_t j = 0; j < 8; j++) {
                    if (j >= left) break;
                    const uint32_t span = j >> 2, in = 2u * (j & 3u);    // +32 bytes of K = +2
                    umma_i8_lo_first(tmem_base + buf * C::kAccCols + (j / MPG) * NT, w_lo + span * (BM * kSpan >> 4) + in,
                                     x_lo + span * (NT * kSpan >> 4) + in, idesc, j % MPG);
                }
                umma_commit(empty(stage));
                umma_commit(tmem_full(buf));
                kb += C::kIssuers;
                if ((stage += C::kIssuers) >= C::kStages) { stage = me; phase ^= 1u; }
                if ((buf += C::kIssuers) >= C::kBufs) { buf = me; buf_phase ^= 1u; }
            }
        }
    } else {
        // ---------------- drain (warps 2 ..): thread = one channel ----------------
        const uint32_t quarter = warp & 3u;                          // TMEM lanes [32*quarter, +32)
        const uint32_t m0 = ((warp - 2u) >> 2) * C::kTokens;         // first of this warp's tokens
        // accumulator row r sits in TMEM lane r (128 rows) or in lane 32*(r/16) + r%16 (64 rows)
        const uint32_t row = BM == 128 ? quarter * 32u + lane : quarter * 16u + (lane & 15u);
        const uint32_t taddr0 = tmem_base + ((quarter * 32u) << 16) + m0;
        uint32_t buf = 0, buf_phase = 0;
        bool ok = true;
        pdl_wait();   // row scales come from the launch before this one, and one may still read the output
        float as[C::kTokens];
#pragma unroll
        for (uint32_t i = 0; i < C::kTokens; i++) as[i] = m0 + i < args.rows ? __ldg(args.row_scales + m0 + i) : 0.0f;
        for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            const uint32_t n = t * BM + row;                         // n < n_pad: the scale table has a (zero) entry
            const float* gs = args.gscales_t + n;
            float sum[C::kTokens];
#pragma unroll
            for (uint32_t i = 0; i < C::kTokens; i++) sum[i] = 0.0f;
            // the scales of the next kAhead stages' groups are on their way while this stage's are used
            float ahead[C::kAhead][C::kGroups];
#pragma unroll
            for (uint32_t u = 0; u < C::kAhead; u++)
#pragma unroll
                for (uint32_t g = 0; g < C::kGroups; g++)
                    ahead[u][g] = u * C::kGroups + g < args.groups ? __ldg(gs + (size_t)(u * C::kGroups + g) * args.n_pad) : 0.0f;
#pragma unroll 1
            for (uint32_t kb0 = 0; ok && kb0 < num_kb; kb0 += C::kAhead)
#pragma unroll
            for (uint32_t u = 0; u < C::kAhead; u++) {
                const uint32_t kb = kb0 + u;
                if (kb >= num_kb) break;
                const uint32_t g0 = kb * C::kGroups;
                float cur[C::kGroups];
#pragma unroll
                for (uint32_t g = 0; g < C::kGroups; g++) {
                    cur[g] = ahead[u][g];
                    const uint32_t ng = g0 + C::kAhead * C::kGroups + g;
                    ahead[u][g] = ng < args.groups ? __ldg(gs + (size_t)ng * args.n_pad) : 0.0f;
                }
                ok = __all_sync(0xffffffffu, mbar_wait(tmem_full(buf), buf_phase, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr = taddr0 + buf * C::kAccCols;
#pragma unroll
                for (uint32_t g = 0; g < C::kGroups; g++) {
                    if (g0 + g >= args.groups) break;                // uniform
                    uint32_t r[C::kTokens];
                    tmem_ld_tokens(taddr + g * NT, r);
                    tmem_ld_wait(r);
#pragma unroll
                    for (uint32_t i = 0; i < C::kTokens; i++) {
                        // |dot| < 2^22: the exact fp32 value without a conversion instruction
                        const float f = __fadd_rn(__uint_as_float(r[i] + 0x4B400000u), -12582912.0f);
                        sum[i] = __fadd_rn(sum[i], __fmul_rn(f, __fmul_rn(as[i], cur[g])));
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tmem_empty(buf));
                if (++buf == C::kBufs) { buf = 0; buf_phase ^= 1u; }
            }
            if (!ok) break;
            if (n < args.n && (BM == 128 || lane < 16)) {
                const float bias = args.bias ? __ldg(args.bias + n) : 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < C::kTokens; i++)
                    if (m0 + i < args.rows) args.out[(size_t)(m0 + i) * args.ld + n] = __fadd_rn(sum[i], bias);
            }
        }
    }

    // ---------------- teardown ----------------
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        nap(200);
        if (threadIdx.x == 0 && args.status) atomicExch(args.status, 1);
        __syncthreads();
    }
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, C::kTmemCols);
}

template <uint32_t BM, uint32_t LT, uint32_t MPG>
cudaError_t launch_few(const GemmGroupedArgs& args, uint32_t grid, cudaStream_t stream) {
    using C = Few<BM, LT, MPG>;
    cudaError_t e = ensure_dynamic_smem<gemm_i8_grouped_few_kernel<BM, LT, MPG>>(C::kSmemBytes);
    if (e != cudaSuccess) return e;
    return launch_pdl(gemm_i8_grouped_few_kernel<BM, LT, MPG>, dim3(grid), dim3(C::kThreads), C::kSmemBytes, stream, args);
}
template <uint32_t BM, uint32_t LT>
cudaError_t launch_few_group(const GemmGroupedArgs& args, uint32_t grid, cudaStream_t stream) {
    switch (args.group) {
        case 32: return launch_few<BM, LT, 1>(args, grid, stream);
        case 64: return launch_few<BM, LT, 2>(args, grid, stream);
        case 128: return launch_few<BM, LT, 4>(args, grid, stream);
        case 256: return launch_few<BM, LT, 8>(args, grid, stream);
        default: return cudaErrorInvalidValue;
    }
}
template <uint32_t BM>
cudaError_t launch_few_tokens(const GemmGroupedArgs& args, uint32_t tokens, uint32_t grid, cudaStream_t stream) {
    switch (tokens) {
        case 8: return launch_few_group<BM, 8>(args, grid, stream);
        case 16: return launch_few_group<BM, 16>(args, grid, stream);
        case 32: return launch_few_group<BM, 32>(args, grid, stream);
        default: return launch_few_group<BM, 64>(args, grid, stream);
    }
}

}  // namespace

GroupedFewShape grouped_few_shape(uint32_t rows, uint32_t n, int sm_count) {
    GroupedFewShape s{};
    if (rows == 0 || rows > kGroupedFewMaxRows) return s;
    s.tokens = rows <= 8 ? 8u : rows <= 16 ? 16u : rows <= 32 ? 32u : 64u;
    s.slots = s.tokens < 16u ? 16u : s.tokens;
    s.channels = 2u * ((n + 127u) / 128u) <= (uint32_t)sm_count ? 64u : 128u;
    const uint32_t tiles = (n + s.channels - 1) / s.channels;
    s.grid = tiles < (uint32_t)sm_count ? tiles : (uint32_t)sm_count;
    s.threads = (s.slots == 64 ? 352u : 224u) + (s.channels == 64 ? 32u : 0u);   // (a second issuer)
    return s;
}

cudaError_t launch_gemm_grouped_few(const GemmGroupedArgs& args, int sm_count, cudaStream_t stream) {
    if (args.rows == 0 || args.n == 0) return cudaSuccess;
    const GroupedFewShape s = grouped_few_shape(args.rows, args.n, sm_count);
    if (!s.slots || !args.groups || args.n_pad % 128u != 0 || args.n_pad < args.n || args.kpad % kSpan != 0) return cudaErrorInvalidValue;
    return s.channels == 64 ? launch_few_tokens<64>(args, s.tokens, s.grid, stream) : launch_few_tokens<128>(args, s.tokens, s.grid, stream);
}

}  // namespace vxb
