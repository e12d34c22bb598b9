// Variant table, launch planning and registry rows (declarations: include/vxb200_plan.h).
// Host code only; nothing here touches a device, so tests drive it on a CPU-only box.
// Counterpart of vx_cuda_packed_plan / vx_cuda_packed_select
// (native/src/backends/cuda/packed_launch_plan.h:33-125).
#include "../../include/vxb200_plan.h"
#include "../../include/vxb200_w8a8.h"
#include "common.cuh"

#include <cstdarg>
#include <cstdio>
#include <cstring>

using namespace vxb;

namespace {

const VxbVariant kVariants[] = {
#define VXB_VARIANT_ROW(id, route, label, symbol, bm, bn, bk, threads, cluster, smem, min_rows, max_rows, epi, weights, group, flags, prio) \
    {#id, route, label, symbol, bm, bn, bk, threads, cluster, smem, min_rows, max_rows, epi, weights, group, flags, prio},
    VXB_VARIANTS(VXB_VARIANT_ROW)
#undef VXB_VARIANT_ROW
};

int refuse(char* why, uint32_t bytes, const char* fmt, ...) {
    if (why && bytes) {
        va_list ap; va_start(ap, fmt);
        vsnprintf(why, bytes, fmt, ap);
        va_end(ap);
    }
    return 0;
}

uint32_t ceil_div(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// Admission of one variant for one query (the fields of the table, nothing else).
bool admitted(const VxbVariant& v, const VxbPlanQuery& q, char* why, uint32_t bytes) {
    if (!(v.weight_mask & q.weight_kind)) { refuse(why, bytes, "%s does not serve this weight kind", v.id); return false; }
    if (!(v.epilogue_mask & q.epilogue)) { refuse(why, bytes, "%s does not produce this output", v.id); return false; }
    if (q.rows < v.min_rows || (v.max_rows && q.rows > v.max_rows)) {
        refuse(why, bytes, "%s serves %u..%u rows (got %u)", v.id, v.min_rows, v.max_rows, q.rows);
        return false;
    }
    if (v.group_size && v.group_size != q.group_size) { refuse(why, bytes, "%s needs group size %u", v.id, v.group_size); return false; }
    if (q.n_peers && !(v.flags & VXB_VF_PEERS)) { refuse(why, bytes, "%s has no peer stores", v.id); return false; }
    if (q.n_peers && v.cluster > 1 && (!q.out_store_aligned || q.epilogue != VXB_EPI_I8)) {
        refuse(why, bytes, "%s stores to peers as TMA tiles only: int8 output, 16-byte aligned buffers", v.id);
        return false;
    }
    if (q.fused_tail && !(v.flags & VXB_VF_FUSED_TAIL)) { refuse(why, bytes, "%s has no fused epilogue tail", v.id); return false; }
    if (v.flags & VXB_VF_TILE_STORE) {
        if (!q.out_store_aligned) { refuse(why, bytes, "%s needs a 16-byte aligned output base and row pitch", v.id); return false; }
        if (q.fused_tail & 2u) { refuse(why, bytes, "%s has no SiLU*Mul tail", v.id); return false; }
    }
    if ((v.flags & VXB_VF_SILU_STORE) && (!q.out_store_aligned || q.fused_tail != 2u)) {
        refuse(why, bytes, "%s is the SiLU*Mul tail into a 16-byte aligned output", v.id);
        return false;
    }
    if (v.cluster > 1 && q.pair_clusters == 0) { refuse(why, bytes, "no co-resident CTA pairs on this device"); return false; }
    if (v.flags & VXB_VF_FUSED_K1) {
        if (!q.fp32_input) { refuse(why, bytes, "%s starts from fp32 rows", v.id); return false; }
        if ((q.k & 3u) || round_up(q.k, kKAlign) > 8192u || q.n > 256u * (q.sm_count ? q.sm_count : 148u)) {
            refuse(why, bytes, "%s needs d_in %% 4 == 0, a padded K of at most 8192 and one channel tile per CTA", v.id);
            return false;
        }
    }
    return true;
}

// Grid, threads and cluster of the chosen variant; false when the kernel has no launch shape.
bool geometry(VxbVariantId id, const VxbPlanQuery& q, VxbLaunchPlan* p) {
    const VxbVariant& v = kVariants[id];
    const uint32_t kpad = round_up(q.k, kKAlign), sms = q.sm_count ? q.sm_count : 148u;
    p->variant = id; p->route = v.route;
    p->tile_rows = v.tile_rows; p->tile_columns = v.tile_columns; p->tile_k = v.tile_k;
    p->threads = v.threads; p->cluster = v.cluster;
    switch (id) {
        case VXB_VARIANT_DECODE_ROWS: case VXB_VARIANT_DECODE_FUSED: {
            DecodeRowsArgs a{};
            a.rows = q.rows; a.n = q.n; a.kpad = kpad;
            if (id == VXB_VARIANT_DECODE_FUSED) { a.x_f32 = reinterpret_cast<const float*>(uintptr_t(16)); a.k = q.k; }
            decode_rows_plan(q.n, (int)sms, &a.tile_rows, &a.tiles_per_cta);
            a.w_stage_bytes = round_up(a.tile_rows * kKAlign, 1024u);
            if (!decode_rows_configure(a)) return false;
            p->tile_rows = decode_rows_token_slots(q.rows);
            p->tile_columns = a.tile_rows;
            p->grid = ceil_div(q.n, a.tiles_per_cta * a.tile_rows);
            p->threads = decode_rows_threads(a.pair != 0);
            return true;
        }
        case VXB_VARIANT_DECODE_STREAMK: {
            const uint64_t units = (uint64_t)ceil_div(q.n, 128) * (kpad / 128);
            p->tile_rows = decode_token_slots(q.rows);
            p->grid = units < sms ? (uint32_t)units : sms;
            p->workspace_bytes += (uint64_t)128 * q.n * 4 + (uint64_t)ceil_div(q.n, 128) * 4;
            return true;
        }
        case VXB_VARIANT_GEMV_DP4A: case VXB_VARIANT_GEMV_GROUPED: case VXB_VARIANT_GEMV_W4_GROUPED: {
            const GemvShape s = gemv_shape(id == VXB_VARIANT_GEMV_DP4A ? 0 : id == VXB_VARIANT_GEMV_GROUPED ? 1 : 2,
                                           q.rows, q.n, kpad, (int)sms);
            p->tile_rows = s.mr; p->tile_columns = 8 * s.ch; p->tile_k = s.kchunk; p->grid = s.grid;
            return true;
        }
        case VXB_VARIANT_SIMT_DP4A:
            p->grid = ceil_div(q.n, 128) * q.rows; p->tile_rows = 1;
            return true;
        case VXB_VARIANT_DP4A_GROUPED:
            p->grid = ceil_div(q.n, 128) * (q.rows == 1 ? 1 : ceil_div(q.rows, 4));
            return true;
        case VXB_VARIANT_TCGEN05: case VXB_VARIANT_TCGEN05_WIDE: case VXB_VARIANT_TCGEN05_WIDE_SILU: case VXB_VARIANT_GROUPED_TCGEN05: {
            if (id == VXB_VARIANT_GROUPED_TCGEN05) {
                const GroupedFewShape few = grouped_few_shape(q.rows, q.n, (int)sms);   // few rows: weights as the M operand
                if (few.slots) {
                    p->tile_rows = few.slots; p->tile_columns = few.channels; p->tile_k = 256;
                    p->threads = few.threads; p->grid = few.grid;
                    return true;
                }
            }
            const uint32_t tiles = ceil_div(q.rows, v.tile_rows) * ceil_div(q.n, v.tile_columns);
            p->grid = tiles < sms ? tiles : sms;
            return true;
        }
        case VXB_VARIANT_TCGEN05_PAIR: case VXB_VARIANT_TCGEN05_PAIR_NARROW: {
            const uint32_t tiles = ceil_div(q.rows, v.tile_rows) * ceil_div(q.n, v.tile_columns);
            p->grid = 2 * (tiles < q.pair_clusters ? tiles : q.pair_clusters);
            return true;
        }
        default: return false;
    }
}

// The per-row quantizer in front of the GEMM when the call starts from fp32 activations
// (the selection rule of launch_quantize_rows, for aligned buffers).
void plan_quantizer(const VxbPlanQuery& q, VxbLaunchPlan* p) {
    const uint32_t kpad = round_up(q.k, kKAlign);
    p->workspace_bytes += (uint64_t)q.rows * kpad + (uint64_t)q.rows * 4;
    p->launches += 1;
    if (q.k % 4 != 0) {
        p->quantizer = VXB_QUANTIZER_SCALAR; p->quantizer_grid = ceil_div(q.rows, 256 / quantize_any_threads(q.rows, q.k)); p->quantizer_cluster = 1;
        return;
    }
    const uint32_t words = kpad / 4;
    if (q.rows <= 32 && words >= 512 && words <= 8u * 256u * 8u) {
        const uint32_t per = ceil_div(words, 256);
        p->quantizer = VXB_QUANTIZER_CLUSTER;
        p->quantizer_cluster = per >= 8 ? 8 : per >= 4 ? 4 : 2;
        p->quantizer_grid = p->quantizer_cluster * q.rows;
        return;
    }
    const uint32_t tpr = quantize_vec_threads(q.rows, q.k);
    p->quantizer = VXB_QUANTIZER_VEC; p->quantizer_cluster = 1;
    p->quantizer_grid = ceil_div(q.rows, 256 / tpr);
}

// 65 to 128 rows in the decode kernel (128 token slots, 128 clocks an MMA: its time grows with the rows, the 32-channel
// pieces of a CTA's share and K) instead of tiles, whose time is one wave and how the output leaves them: TMA stores for
// aligned 32-bit words, 16 bytes a lane for aligned int8, the warps' store tiles for unaligned rows, eight warps for the
// SiLU * Mul tail.  us replayed from a graph, decode / tiles, at K -> N and 65, 96 and 128 rows (N 3072, 6144 and 11008:
// one, two and three pieces):
//   unaligned fp32 512 -> 3072 8.2/11.3 8.9/11.4 9.8/11.7;  1024 -> 6144 11.8/12.5 13.5/12.6 15.6/13.0;  2048 -> 1024 13.9/11.0 14.7/11.1 15.6/11.2
//   SiLU * Mul     512 -> 3072 9.2/14.6 10.3/14.9 11.8/15.3;  1024 -> 6144 14.0/15.9 16.1/16.2 19.4/16.4;  1536 -> 11008 19.9/17.5 23.4/17.7 27.4/18.0
//   unaligned int8 256 -> 3072 7.8/10.0 8.7/10.1 10.2/10.2;  512 -> 3072 9.1/10.8 10.1/10.7 11.5/10.9;  512 -> 6144 12.2/10.7 14.4/10.8 17.1/10.9
//   aligned fp32   256 -> 1024 6.7/6.9 7.4/7.0 8.0/7.5;  512 -> 3072 8.1/7.7 8.9/7.8 9.8/8.2;  1024 -> 3072 9.8/8.9 10.7/9.3 11.5/9.4;
//                  1024 -> 6144 12.1/9.0 13.3/9.2 15.5/9.5
// (K above 1536 goes to the paired tiles, in half of the decode kernel's time.)  The last line of the rule, all outputs up
// to K 1024 and N 3072, is older than the fast stores of the aligned ones, which are past their crossing there.
bool decode_past_64_rows(const VxbPlanQuery& q) {
    const uint32_t kpad = round_up(q.k, kKAlign);
    const uint64_t work = (uint64_t)q.rows * ceil_div(ceil_div(q.n, q.sm_count ? q.sm_count : 148u), 32u);
    if (q.rows > 128 || kpad > VXB_WIDE_MAX_KPAD) return false;
    if ((q.fused_tail & 2u) && work <= 192) return true;
    if (!q.out_store_aligned && (q.epilogue == VXB_EPI_I8 ? work <= 128 && q.rows * kpad <= 65536u : work <= 160)) return true;
    return kpad <= 1024 && q.n <= 3072;
}

}  // namespace

extern "C" {

uint32_t vxb_variant_count(void) { return VXB_VARIANT_COUNT; }

const VxbVariant* vxb_variant_info(uint32_t index) { return index < VXB_VARIANT_COUNT ? &kVariants[index] : nullptr; }

int vxb_plan(const VxbPlanQuery* query, VxbLaunchPlan* out, char* why, uint32_t why_bytes) {
    if (why && why_bytes) why[0] = 0;
    if (!query || !out) return refuse(why, why_bytes, "null argument");
    const VxbPlanQuery& q = *query;
    if (!q.rows || !q.k || !q.n) return refuse(why, why_bytes, "empty shape");
    if (q.weight_kind != VXB_WEIGHT_PER_CHANNEL && q.weight_kind != VXB_WEIGHT_GROUPED && q.weight_kind != VXB_WEIGHT_W4_WORDS)
        return refuse(why, why_bytes, "weight kind must be one VXB_WEIGHT_* bit");
    if (q.epilogue != VXB_EPI_ACC && q.epilogue != VXB_EPI_F32 && q.epilogue != VXB_EPI_I8)
        return refuse(why, why_bytes, "epilogue must be one VXB_EPI_* bit");
    const bool grouped = q.weight_kind != VXB_WEIGHT_PER_CHANNEL;
    if (grouped && q.group_size != 32 && q.group_size != 64 && q.group_size != 128 && q.group_size != 256)
        return refuse(why, why_bytes, "group size %u is not 32/64/128/256", q.group_size);
    if ((uint64_t)q.k * 127u * 128u > 2147483647ull) return refuse(why, why_bytes, "d_in %u can overflow the int32 accumulator", q.k);
    if (q.n_peers > 7) return refuse(why, why_bytes, "at most 7 peers");
    const uint32_t sms = q.sm_count ? q.sm_count : 148u;

    memset(out, 0, sizeof *out);
    out->launches = 1;
    int chosen = -1;
    if (q.requested_route != VXB_ROUTE_AUTO) {
        // an explicit route is honoured or refused, never replaced by another kernel
        if (grouped && q.requested_route != VXB_ROUTE_SIMT)
            return refuse(why, why_bytes, "weights with grouped scales take the automatic route only");
        for (int i = 0; i < VXB_VARIANT_COUNT; i++)
            if (kVariants[i].route == q.requested_route && (kVariants[i].weight_mask & q.weight_kind)) { chosen = i; break; }
        if (chosen < 0) return refuse(why, why_bytes, "no kernel variant has route %d", q.requested_route);
        if (!admitted(kVariants[chosen], q, why, why_bytes)) return 0;
    } else if (grouped) {
        if (q.epilogue != VXB_EPI_F32) return refuse(why, why_bytes, "weights with grouped scales produce fp32 output only");
        if (q.fused_tail) return refuse(why, why_bytes, "weights with grouped scales have no fused epilogue");
        // decode: a warp per channel streams the weights once (over the 4-bit words when they were kept); from three rows on
        // the tensor-core kernel is faster at large weights, and at fewer bytes where K is long and the GEMV's blocks are more
        // than half of the SMs (four rows, G = 128, from a graph / in a stream, us, GEMV and tiles: 8192 -> 1024 12.8/13.6 and
        // 14.7/15.4, 8192 -> 2000 18.0/18.6 and 14.8/15.5, 8192 -> 4000 24.0/19.1 and 15.0/15.8, 11008 -> 2048 23.5/17.7 and
        // 18.6/19.3)
        const uint64_t weight_bytes = (uint64_t)round_up(q.k, kKAlign) * q.n;
        if (q.rows <= 2 && q.weight_kind == VXB_WEIGHT_W4_WORDS) chosen = VXB_VARIANT_GEMV_W4_GROUPED;
        else if (q.rows <= 2 || (q.rows <= 4 && weight_bytes <= (32ull << 20) && !(q.k >= 8192 && q.n > 1536))) chosen = VXB_VARIANT_GEMV_GROUPED;
        else chosen = VXB_VARIANT_GROUPED_TCGEN05;
        if (!admitted(kVariants[chosen], q, why, why_bytes)) return 0;
    } else {
        if (q.n_peers) {
            // fused all-gather: the single-CTA kernel with its 128-byte store tiles, unless the launch is clearly
            // MMA-bound (padded K of at least 3424 per peer, 1.6 times the break-even of gather_is_link_bound):
            // then the pairs of CTAs, whose 64-byte store tiles use the links less well, when their tile stores
            // are possible.  Measured: 2 GPUs, K 4096: 174 us paired against 190; 4 GPUs, K 8192 (1.28 times
            // the break-even): 569 us paired against 508.
            const uint32_t tiles = ceil_div(q.rows, 128) * ceil_div(q.n, 256);
            char unused[8];
            chosen = VXB_VARIANT_TCGEN05;
            if (q.rows > 128 && tiles >= 2u * sms && (uint64_t)q.n_peers * 3424u <= round_up(q.k, kKAlign) &&
                admitted(kVariants[VXB_VARIANT_TCGEN05_PAIR], q, unused, sizeof unused)) chosen = VXB_VARIANT_TCGEN05_PAIR;
        }
        else if (q.rows <= 64 || decode_past_64_rows(q)) {
            chosen = VXB_VARIANT_DECODE_ROWS;
            char unused[8];
            // one or two fp32 rows: the single-launch form.  From three rows on every CTA repeating the
            // quantization costs more than the separate cluster quantizer (17.1 against 15.5 us per
            // step at 8 rows, K 4096, N 14336), so the two-launch form stays.
            if (q.fp32_input && q.rows <= tunables().decode_fused_max_rows &&
                admitted(kVariants[VXB_VARIANT_DECODE_FUSED], q, unused, sizeof unused)) chosen = VXB_VARIANT_DECODE_FUSED;
        }
        else {
            // pairs of CTAs on 256 x 256 tiles once there are at least two waves of 128 x 256 tiles
            const uint32_t tiles = ceil_div(q.rows, 128) * ceil_div(q.n, 256);
            chosen = (q.pair_clusters > 0 && tiles >= 2u * sms) ? VXB_VARIANT_TCGEN05_PAIR : VXB_VARIANT_TCGEN05;
            if (q.pair_clusters > 0 && round_up(q.k, kKAlign) > VXB_WIDE_MAX_KPAD) {
                // Long K: a wave of tiles costs its K loop, bound by the operands an SM pulls from L2 per 128 bytes of
                // K (48 KB for 128 x 256 alone, 32 KB in a pair on 256 x 256, 24 KB on 256 x 128) or by the MMAs on
                // them (512, 512, 256 clocks); a pair takes longer to set up.  In clocks, from K = 4096 -> 4096 with
                // fp32 output: 512 rows 16.8 / 16.7 / 13.3 us, 1024 rows 17.1 / 17.8 / -, 2048 rows 29.3 / 27.4 / -
                // (alone / pair / narrow pair).  Held against all three at K 1664 .. 14336, 130 .. 4096 rows and N 1024 ..
                // 11008, fp32 and int8 outputs: 254 of 274 calls get the fastest; the most that one loses is 6 % (int8,
                // 777 x 1664 -> 11008: a pair 26.1 us, alone 24.6).
                const uint32_t pair_rows = ceil_div(q.rows, 256);
                const uint64_t kb = round_up(q.k, kKAlign) / kKAlign;
                const uint64_t alone = 9300ull + 724ull * kb * ceil_div(tiles, sms);
                const uint64_t pair = 14250ull + 594ull * kb * ceil_div(pair_rows * ceil_div(q.n, 256), q.pair_clusters);
                const uint64_t narrow = 13000ull + 386ull * kb * ceil_div(pair_rows * ceil_div(q.n, 128), q.pair_clusters);
                chosen = narrow < pair && narrow < alone ? VXB_VARIANT_TCGEN05_PAIR_NARROW
                       : pair <= alone ? VXB_VARIANT_TCGEN05_PAIR : VXB_VARIANT_TCGEN05;
            }
            // 32-bit outputs at short K are bound by the output, not by the tensor pipe
            char unused[8];
            if (q.epilogue != VXB_EPI_I8 && round_up(q.k, kKAlign) <= VXB_WIDE_MAX_KPAD &&
                admitted(kVariants[VXB_VARIANT_TCGEN05_WIDE], q, unused, sizeof unused)) chosen = VXB_VARIANT_TCGEN05_WIDE;
            // ... and by the tail's arithmetic, from a full wave of tiles on
            if ((q.fused_tail & 2u) && tiles >= sms && round_up(q.k, kKAlign) <= VXB_WIDE_MAX_KPAD &&
                admitted(kVariants[VXB_VARIANT_TCGEN05_WIDE_SILU], q, unused, sizeof unused)) chosen = VXB_VARIANT_TCGEN05_WIDE_SILU;
        }
        if (!admitted(kVariants[chosen], q, why, why_bytes)) return 0;
    }
    if (!geometry((VxbVariantId)chosen, q, out))
        return refuse(why, why_bytes, "no launch shape for %s (rows %u, d_out %u)", kVariants[chosen].id, q.rows, q.n);
    if (q.fp32_input && !(kVariants[chosen].flags & VXB_VF_FUSED_K1)) plan_quantizer(q, out);
    return 1;
}

uint32_t vxb_registry_row(uint32_t index, char* out, uint32_t out_bytes) {
    if (index >= VXB_VARIANT_COUNT || !out || !out_bytes) return 0;
    const VxbVariant& v = kVariants[index];
    const bool grouped = (v.weight_mask & VXB_WEIGHT_PER_CHANNEL) == 0;
    // PackedLinear (R1) is served by every variant; the static QLinear operator (R2) by the
    // per-channel kernels that produce int8
    const char* ops = (!grouped && (v.epilogue_mask & VXB_EPI_I8)) ? "PackedLinear,QLinear" : "PackedLinear";
    const char* phase = v.max_rows && v.max_rows <= 128 ? "decode" : (v.flags & VXB_VF_VERIFY) ? "any" : "prefill";
    const bool tensor = strstr(v.route_label, "tcgen05") != nullptr;
    const int n = snprintf(out, out_bytes,
                           "cuda.packed-linear.%s | native-cuda | %s | w8a8-%s | %s | %s | cuda.sm100a-route-predicate | "
                           "cuda.device-residency,%s | %u",
                           v.route_label, ops, grouped ? "grouped" : "per-channel", phase, v.kernel,
                           tensor ? "cuda.sm100a-tcgen05" : "cuda.sm61-dp4a", v.priority);
    return n > 0 && (uint32_t)n < out_bytes ? (uint32_t)n : 0;
}

}  // extern "C"
