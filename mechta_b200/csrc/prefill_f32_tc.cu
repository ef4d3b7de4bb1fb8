// Prefill attention over the f32 cache, f32-grade arithmetic on the tensor cores: tcgen05.mma by CTA pairs.
//
// Stands in for attn_fa / attn_fd4 + attn_fd_combine of the reference on the f32 cache (W/ops.wgsl:562-651,711-778): token T of the
// block (at pos0 + T) sees first_pos <= key < pos0 + 1 + T. The work is cut as in prefill_tc.cu (prefill_plan.cuh): an item is
// 32 tokens x the 8 query heads of one KV head = 256 rows, 128 in each CTA of a pair, tiles of 128 keys, each CTA loading one
// half of a tile (64 keys of K, 128 of the 256 dims of V); parts of split items are merged by the same kernel.
//
// Arithmetic as in verify_f32_tc.cu: every f32 operand is split into hi = f16(x) and lo = f16(x - hi), a product is
// hi.lo + lo.hi + hi.hi with exact f16 products and f32 accumulators, and every tile's P.V starts from zero and is folded into
// O in registers with rounded adds, because the tensor core's accumulation truncates. Within a tile the two small terms are
// accumulated first, so that the truncations of the long chain happen on small sums.
//
// The f32 prefill used to run as batched 4-token verify items, which read every key once per 4 tokens: 512 tokens over a
// 4,096-token prefix took 567 us a layer, here 120 (8,000: 951 -> 200, 32,768: 3,380 -> 710). A tile takes about 10,400 cycles, of
// which 9,500 are the products: 48 of 256 x 128 x 16 at 128 cycles each (by a pair of CTAs, N = 128 runs at half the rate of N =
// 256) and 24 of 256 x 256 x 16 at 140. The rest is the softmax between a tile's two products: tensor memory has no room for a
// second S, or for one of 256 keys, beside O_t, Q and P. Starting P.V on the first half of the weights was 2 % faster and took
// the error from 6.5e-7 to 7.8e-7. Relative error against f64 over 5 ... 512 tokens and 16 ... 32,768 keys: 3.6e-7 to 6.7e-7
// (2-norm), the verify items 6.5e-7 to 1.1e-6.
//
// Memory. TMA brings a slot [64 keys][128 dims] f32 (32 KB) as two regions of 64 dims, each two boxes of [64 keys][32 dims]
// whose rows are 128 bytes (128-byte swizzle). A converter warp rewrites a row's two 128-byte pieces as the row's 64 hi halves
// (first box) and 64 lo halves (second box): in place, four lanes a row, so a region becomes two f16 operand blocks
// [64 keys][64 dims]. A tile is four slots (K dims 0-127, K dims 128-255, V keys 0-63, V keys 64-127), the ring holds five.
// Queries: hi in tensor memory, lo in shared memory. Weights overwrite their scores in tensor memory: of 16 score columns the
// first 8 become the hi halves of the 16 weights, the others the lo halves (the A operand of P.V).
// TMEM: O_t = columns 0..255, S / P = 256..383, Q hi = 384..511.
//
// Roles (512 threads, register budgets set with setmaxnreg): warp 0 = TMA producer, warp 1 = MMA issuer (one thread, of the
// pair's first CTA) and TMEM owner, warps 4-7 = converters, warps 8-15 = softmax, two threads a row (64 of a tile's keys each)
// which also own 128 dims of the row's O each. Every wait is bounded; TMEM is freed on every path.
#include <stdlib.h>

#include "internal.cuh"
#include "prefill_plan.cuh"
#include "ptx.cuh"

namespace mkv {
using namespace ptx;

constexpr uint32_t PS_NSLOT = 5;
constexpr uint32_t PS_SLOT = 32768;                    // [64 keys][128 dims] f32
constexpr uint32_t PS_REGION = 16384;                  // 64 dims of it; after conversion a hi block and a lo block
constexpr uint32_t PS_BLK = 8192;
constexpr uint32_t PS_OFF_Q = PS_NSLOT * PS_SLOT;      // Q lo: [4 blocks of 64 dims][128 rows][64 dims] f16
constexpr uint32_t PS_QB = 16384;
constexpr uint32_t PS_OFF_RED = PS_OFF_Q + 4 * PS_QB;  // [2 halves][128 rows] floats
constexpr uint32_t PS_OFF_BAR = PS_OFF_RED + 1024;
// barriers: full[NSLOT], conv[NSLOT], empty[NSLOT], s_full, p_full, o_full, q_full
constexpr uint32_t PS_NBAR = 3 * PS_NSLOT + 4;
constexpr uint32_t PS_OFF_MISC = PS_OFF_BAR + PS_NBAR * 8;
constexpr uint32_t PS_SMEM = PS_OFF_MISC + 32 + 1024;
constexpr uint32_t PS_COL_O = 0, PS_COL_S = 256, PS_COL_Q = 384, PS_COLS = 512;
constexpr int PS_THREADS = 512;
constexpr int PS_ROW_OUTSIDE = 1 << 30;                // a row coordinate beyond any cache: TMA fills such a box with zeros
constexpr long long PS_WAIT_LIMIT = 2000000000ll;
constexpr float PS_LOG2E = 1.4426950408889634f;
constexpr float PS_C2 = SCALE * PS_LOG2E;              // scores to base-2 exponents
constexpr float PS_LAZY2 = 8.0f * PS_LOG2E;
constexpr PfCost PS_COST = {1.4f, 0.6f, 0.023f};       // a tile takes about 5.6 us
static_assert(PS_SMEM <= 232448, "shared memory of prefill_f32_tc_kernel");

struct PsShared {
    uint32_t tmem_base;
    volatile uint32_t abort;
};

__device__ __forceinline__ bool ps_wait(uint32_t bar, uint32_t parity, PsShared *sh, uint32_t *status) {
    if (sh->abort) return false;
    if (mbar_wait_bounded(bar, parity, PS_WAIT_LIMIT)) return true;
    sh->abort = 1;
    atomicOr(status, DEV_ERR_WAIT_TIMEOUT);
    return false;
}
// named barrier 5: all warps, at the end of their roles (1..4: the two warps of a group of 32 rows)
__device__ __forceinline__ void ps_bar_roles() { asm volatile("bar.sync 5, 512;" ::: "memory"); }
// hi and lo halves of two floats
__device__ __forceinline__ void ps_split2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ void ps_split8(const float4 &a, const float4 &b, uint4 &hi, uint4 &lo) {
    ps_split2(a.x, a.y, hi.x, lo.x);
    ps_split2(a.z, a.w, hi.y, lo.y);
    ps_split2(b.x, b.y, hi.z, lo.z);
    ps_split2(b.z, b.w, hi.w, lo.w);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PS_THREADS, 1)
prefill_f32_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                      const float *__restrict__ q, float *__restrict__ out, const __grid_constant__ PfPlan plan, uint32_t row0,
                      float *__restrict__ scratch, uint32_t *__restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u; // the same in both CTAs
    uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cta = cluster_ctarank(), pair = blockIdx.x >> 1;
    const uint32_t bar_full = smem_base + PS_OFF_BAR, bar_conv = bar_full + 8u * PS_NSLOT, bar_empty = bar_conv + 8u * PS_NSLOT;
    const uint32_t bar_s_full = bar_empty + 8u * PS_NSLOT, bar_p_full = bar_s_full + 8u, bar_o_full = bar_p_full + 8u;
    const uint32_t bar_q_full = bar_o_full + 8u;
    PsShared *sh = reinterpret_cast<PsShared *>(smem + PS_OFF_MISC);
    pdl_launch_dependents();

    if (tid == 0) {
        for (uint32_t s = 0; s < PS_NSLOT; s++) {
            mbar_init(bar_full + 8u * s, 1);
            mbar_init(bar_conv + 8u * s, 8); // one arrival per converter warp of the pair (counted in the first CTA only)
            mbar_init(bar_empty + 8u * s, 1);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_p_full, 16); // one arrival per softmax warp of the pair
        mbar_init(bar_o_full, 1);
        mbar_init(bar_q_full, 16);
        sh->abort = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc2(smem_base + PS_OFF_MISC, PS_COLS); // writes sh->tmem_base
    tc_fence_before();
    cluster_sync(); // barriers and tensor memory of both CTAs are there
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait(); // nothing global is touched before the kernel in front has finished

    // Every role walks the same segments; g counts the tiles this pair has dealt with so far, across segments. Tile g is the
    // slots 4g .. 4g+3 of the stream, slot n lies in ring position n % NSLOT and is its use n / NSLOT.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            // ---------------- TMA producer: this CTA's halves ----------------
            uint32_t n = 0;
            PfWalk walk(plan, pair);
            PfSegment sg;
            bool ok = true;
            while (ok && walk.next(sg)) {
                const uint32_t end = plan.pos0 + plan.item_end(sg.item); // no key at or past this one is seen by the item's tokens
                for (uint32_t j = sg.a; ok && j < sg.b; j++) {
#pragma unroll 1
                    for (uint32_t part = 0; part < 4u; part++, n++) {
                        const uint32_t s = n % PS_NSLOT, bar = bar_full + 8u * s, dst = smem_base + s * PS_SLOT;
                        if (n >= PS_NSLOT && !(ok = ps_wait(bar_empty + 8u * s, ((n / PS_NSLOT) - 1u) & 1u, sh, status))) break;
                        const bool is_v = part >= 2u;
                        const CUtensorMap *map = is_v ? &vmap : &kmap;
                        const uint32_t key = (plan.t0 + j) * PF_KEYS + 64u * (is_v ? part & 1u : cta);
                        const int x = (int)((sg.item & 1u) * 256u + 128u * (is_v ? cta : part));
                        const int y = key < end ? (int)(key - row0) : PS_ROW_OUTSIDE;
                        mbar_expect_tx(bar, PS_SLOT);
#pragma unroll
                        for (int b = 0; b < 4; b++) tma_load_2d(dst + b * PS_BLK, map, x + 32 * b, y, bar);
                    }
                }
            }
            // the last releases must have arrived here before this CTA may leave: they come from the first CTA's commits
            for (uint32_t i = n > PS_NSLOT ? n - PS_NSLOT : 0u; ok && i < n; i++)
                ok = ps_wait(bar_empty + 8u * (i % PS_NSLOT), (i / PS_NSLOT) & 1u, sh, status);
        } else if (warp == 1 && lane == 0 && cta == 0) {
            // ---------------- MMA issuer ----------------
            constexpr uint32_t IDESC_QK = tc_idesc_f16(256, 128, false);
            constexpr uint32_t IDESC_PV = tc_idesc_f16(256, 256, true);
            const uint32_t qlo = smem_base + PS_OFF_Q, S = tmem + PS_COL_S, O = tmem + PS_COL_O, Q = tmem + PS_COL_Q;
            uint32_t g = 0, nseg = 0;
            auto slot = [&](uint32_t n) { return smem_base + (n % PS_NSLOT) * PS_SLOT; };
            auto slot_wait = [&](uint32_t n) -> bool {
                if (!ps_wait(bar_conv + 8u * (n % PS_NSLOT), (n / PS_NSLOT) & 1u, sh, status)) return false;
                tc_fence_after();
                return true;
            };
            // (the loops stay rolled up: an MMA takes 64 or 128 cycles, and this warpgroup has few registers)
            auto qk = [&]() -> bool { // S = Q K^T for tile g: the small terms of both slots, then the large ones
#pragma unroll 1
                for (uint32_t s = 0; s < 2u; s++) {
                    if (!slot_wait(4u * g + s)) return false;
#pragma unroll 1
                    for (uint32_t r = 0; r < 2u; r++) { // 64 dims of the slot's 128, 16 per MMA
                        const uint32_t b = slot(4u * g + s) + r * PS_REGION, a = qlo + (2u * s + r) * PS_QB, qa = Q + 64u * s + 32u * r;
#pragma unroll
                        for (uint32_t ks = 0; ks < 4u; ks++) {
                            tc_mma2_f16(S, tc_desc_sw128(a + ks * 32u, 16, 1024), tc_desc_sw128(b + ks * 32u, 16, 1024), IDESC_QK, s | r | ks);
                            tc_mma2_f16_ta(S, qa + 8u * ks, tc_desc_sw128(b + PS_BLK + ks * 32u, 16, 1024), IDESC_QK, 1u);
                        }
                    }
                }
#pragma unroll 1
                for (uint32_t s = 0; s < 2u; s++) {
#pragma unroll 1
                    for (uint32_t r = 0; r < 2u; r++) {
                        const uint32_t b = slot(4u * g + s) + r * PS_REGION, qa = Q + 64u * s + 32u * r;
#pragma unroll
                        for (uint32_t ks = 0; ks < 4u; ks++) tc_mma2_f16_ta(S, qa + 8u * ks, tc_desc_sw128(b + ks * 32u, 16, 1024), IDESC_QK, 1u);
                    }
                    tc_commit2(bar_empty + 8u * ((4u * g + s) % PS_NSLOT));
                }
                tc_commit2(bar_s_full);
                return true;
            };
            // O_t = P V for tile g, from zero. mma(a, b, accumulate, key) issues one MMA over the 16 keys from `key`; key0 = the tile's first.
            auto pv = [&](uint32_t key0, auto mma) -> bool {
#pragma unroll 1
                for (uint32_t s = 0; s < 2u; s++) {
                    if (!slot_wait(4u * g + 2u + s)) return false;
                    const uint32_t v = slot(4u * g + 2u + s), p = S + 64u * s, key = key0 + 64u * s;
#pragma unroll
                    for (uint32_t ks = 0; ks < 4u; ks++) { // weights' hi halves in 8 columns, lo halves in the next 8
                        // V slot, N-major: the next 64 dims one region on, the next 8 keys 1024 bytes on
                        mma(p + 16u * ks + 8u, tc_desc_sw128(v + ks * 2048u, PS_REGION, 1024), s | ks, key + 16u * ks);
                        mma(p + 16u * ks, tc_desc_sw128(v + PS_BLK + ks * 2048u, PS_REGION, 1024), 1u, key + 16u * ks);
                    }
                }
#pragma unroll 1
                for (uint32_t s = 0; s < 2u; s++) {
                    const uint32_t v = slot(4u * g + 2u + s), p = S + 64u * s, key = key0 + 64u * s;
#pragma unroll
                    for (uint32_t ks = 0; ks < 4u; ks++) mma(p + 16u * ks, tc_desc_sw128(v + ks * 2048u, PS_REGION, 1024), 1u, key + 16u * ks);
                    tc_commit2(bar_empty + 8u * ((4u * g + 2u + s) % PS_NSLOT));
                }
                tc_commit2(bar_o_full);
                return true;
            };
            PfWalk walk(plan, pair);
            PfSegment sg;
            bool ok = true;
            while (ok && walk.next(sg)) {
                if (!(ok = ps_wait(bar_q_full, nseg & 1u, sh, status))) break; // the segment's queries are in place
                tc_fence_after();
                nseg++;
                const uint32_t tok_pos = plan.pos0 + 32u * plan.group_of(sg.item);
                for (uint32_t j = sg.a; j < sg.b; j++, g++) {
                    // The products run in the order in which they are issued: S of this tile overwrites weights that the product
                    // before has read. The weights of this tile are there once its scores have been read and O_t of the tile
                    // before has been folded (the same threads do all of it, in this order).
                    if (!(ok = qk())) break;
                    if (!(ok = ps_wait(bar_p_full, g & 1u, sh, status))) break;
                    tc_fence_after();
                    const uint32_t key0 = (plan.t0 + j) * PF_KEYS;
                    if (key0 + PF_KEYS <= tok_pos + 1u) // every token sees the whole tile
                        ok = pv(key0, [&](uint32_t a, uint64_t b, uint32_t acc, uint32_t) { tc_mma2_f16_ta(O, a, b, IDESC_PV, acc); });
                    else
                        ok = pv(key0, [&](uint32_t a, uint64_t b, uint32_t acc, uint32_t key) {
                            tc_mma2_f16_ta_off(O, a, b, IDESC_PV, acc, pf_blind_rows(key, tok_pos), pf_blind_rows(key, tok_pos + 16u));
                        });
                    if (!ok) break;
                }
            }
        }
        __syncwarp();
        ps_bar_roles(); // registers come back only after the softmax warps have returned theirs
        asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    } else if (warp < 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // ---------------- converters: f32 rows -> f16 hi and lo rows, in place ----------------
        // Four lanes take a row of a region (16 dims each). The second box's lanes take their chunks in another order, which
        // keeps both the loads and the stores of eight lanes on different banks. Rows no token of the item sees become zero:
        // whatever lies in them, their weights' 0 x V stays finite.
        const uint32_t w = warp - 4u, quarter = lane & 3u, rot = quarter & 2u;
        const uint32_t r_conv = cluster_map(bar_conv, 0);
        uint32_t n = 0;
        PfWalk walk(plan, pair);
        PfSegment sg;
        bool ok = true;
        while (ok && walk.next(sg)) {
            const uint32_t end = plan.pos0 + plan.item_end(sg.item);
            for (uint32_t j = sg.a; ok && j < sg.b; j++) {
#pragma unroll 1
                for (uint32_t part = 0; part < 4u; part++, n++) {
                    const uint32_t s = n % PS_NSLOT;
                    if (!(ok = __all_sync(0xffffffffu, ps_wait(bar_full + 8u * s, (n / PS_NSLOT) & 1u, sh, status)))) break;
                    const uint32_t key0 = (plan.t0 + j) * PF_KEYS + 64u * (part >= 2u ? part & 1u : cta);
#pragma unroll 2
                    for (uint32_t i = 0; i < 4u; i++) {
                        const uint32_t row = (i & 1u) * 32u + w * 8u + (lane >> 2), x = row & 7u, key = key0 + row;
                        uint8_t *hi = smem + s * PS_SLOT + (i >> 1) * PS_REGION + row * 128u, *lo = hi + PS_BLK;
                        const uint8_t *src = (quarter & 2u) ? lo : hi;
                        const uint32_t c0 = 4u * (quarter & 1u);
                        float4 f[4];
#pragma unroll
                        for (uint32_t k = 0; k < 4u; k++) f[k] = *reinterpret_cast<const float4 *>(src + (((c0 + (k ^ rot)) ^ x) << 4));
                        if (key >= end || key < plan.first_pos) {
#pragma unroll
                            for (int k = 0; k < 4; k++) f[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                        uint4 h0, l0, h1, l1;
                        ps_split8(f[0], f[1], h0, l0);
                        ps_split8(f[2], f[3], h1, l1);
                        __syncwarp(); // the row's four lanes have read it
                        const uint32_t o0 = ((2u * quarter + (rot >> 1)) ^ x) << 4, o1 = ((2u * quarter + 1u - (rot >> 1)) ^ x) << 4;
                        *reinterpret_cast<uint4 *>(hi + o0) = h0;
                        *reinterpret_cast<uint4 *>(hi + o1) = h1;
                        *reinterpret_cast<uint4 *>(lo + o0) = l0;
                        *reinterpret_cast<uint4 *>(lo + o1) = l1;
                    }
                    fence_proxy_async(); // the tensor cores read the slot through the async proxy
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(r_conv + 8u * s);
                }
            }
        }
        __syncwarp();
        ps_bar_roles();
        asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        // ---------------- softmax: two threads per row (TMEM lane), 64 keys of a tile and 128 dims of O each ----------------
        const uint32_t q4 = warp & 3u, half = (warp >> 2) & 1u;
        const uint32_t row = 32u * q4 + lane; // the TMEM lanes this warp may access
        const uint32_t lane_addr = (32u * q4) << 16;
        const uint32_t r_p_full = cluster_map(bar_p_full, 0), r_q_full = cluster_map(bar_q_full, 0);
        float *red = reinterpret_cast<float *>(smem + PS_OFF_RED);
        auto arrive = [&](uint32_t bar) { // one arrival per warp, after all its lanes
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bar);
        };
        // This warp's rows of Q lo, dims 128 half .. + 127: two pieces of 4 KB. Between segments they are also where rows change
        // hands between "a lane has a row" (registers, tensor memory) and "a few lanes share a row" (coalesced global accesses).
        uint8_t *qmine = smem + PS_OFF_Q + 2u * half * PS_QB + 4096u * q4;
        auto load_q = [&](const PfSegment &sg) {
            const uint32_t t0 = plan.group_of(sg.item) * 32u + 16u * cta, h0 = 8u * (sg.item & 1u) + 2u * q4;
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < 2u; c0++) { // 64 dims at a time, 16 lanes a row
                float4 v[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const uint32_t r = 2u * i + (lane >> 4), tok = t0 + (r & 15u);
                    v[i] = tok < plan.ntok ? __ldg(reinterpret_cast<const float4 *>(q + (size_t)tok * 4096u + (size_t)(h0 + (r >> 4)) * 256u +
                                                                                   128u * half + 64u * c0 + 4u * (lane & 15u)))
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                uint8_t *blk = qmine + c0 * PS_QB;
                uint2 lo[16];
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    uint2 hi;
                    ps_split2(v[i].x, v[i].y, hi.x, lo[i].x);
                    ps_split2(v[i].z, v[i].w, hi.y, lo[i].y);
                    *reinterpret_cast<uint2 *>(blk + swz128(2u * i + (lane >> 4), (lane & 15u) >> 1) + 8u * (lane & 1u)) = hi;
                }
                __syncwarp();
                uint32_t w[32];
#pragma unroll
                for (uint32_t c = 0; c < 8u; c++) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(blk + swz128(lane, c));
                    w[4 * c] = a.x; w[4 * c + 1] = a.y; w[4 * c + 2] = a.z; w[4 * c + 3] = a.w;
                }
                tmem_st32(tmem + lane_addr + PS_COL_Q + 64u * half + 32u * c0, w);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 16; i++)
                    *reinterpret_cast<uint2 *>(blk + swz128(2u * i + (lane >> 4), (lane & 15u) >> 1) + 8u * (lane & 1u)) = lo[i];
            }
            fence_proxy_async();
            tmem_wait_st();
            tc_fence_before();
            arrive(r_q_full);
        };
        uint32_t g = 0;
        PfWalk walk(plan, pair);
        PfSegment sg;
        bool ok = true;
        while (ok && walk.next(sg)) {
            load_q(sg);
            const uint32_t tok0 = plan.group_of(sg.item) * 32u + 16u * cta, kvh = sg.item & 1u;
            const uint32_t vis = plan.pos0 + 1u + tok0 + (row & 15u); // the row's token sees keys < vis
            const uint32_t full_below = plan.pos0 + 1u + tok0; // keys below this are visible to every row of the CTA
            float m_ref = NEG_BIG, l_run = 0.0f; // l_run: this thread's 64 keys of every tile only
            float acc[128];                      // O of the row, dims 128 half .. + 127
#pragma unroll
            for (int i = 0; i < 128; i++) acc[i] = 0.0f;
            for (uint32_t j = sg.a; j < sg.b; j++, g++) {
                // The warp takes every wait's outcome together: the TMEM accesses below are warp-collective. A wait that ran out
                // goes into the next vote, so that the two warps of these rows leave together.
                ok = __all_sync(0xffffffffu, ps_wait(bar_s_full, g & 1u, sh, status)) && ok;
                tc_fence_after();
                const uint32_t s_addr = tmem + lane_addr + PS_COL_S + 64u * half;
                const uint32_t tile_key = (plan.t0 + j) * PF_KEYS, key_base = tile_key + 64u * half;
                // which of the 64 keys the row sees: all of them off the causal diagonal and the window start
                const bool masked = key_base + 64u > full_below || key_base < plan.first_pos;
                const uint32_t k_lo = plan.first_pos > key_base ? plan.first_pos - key_base : 0u;
                const uint32_t k_hi = vis > key_base ? vis - key_base : 0u;
                float mx = NEG_BIG;
#pragma unroll
                for (uint32_t h = 0; h < 2u; h++) {
                    uint32_t sr[32];
                    tmem_ld32(s_addr + 32u * h, sr);
                    tmem_wait_ld();
                    float mt[4] = {NEG_BIG, NEG_BIG, NEG_BIG, NEG_BIG};
                    if (masked) {
#pragma unroll
                        for (uint32_t c = 0; c < 32u; c++)
                            if (32u * h + c >= k_lo && 32u * h + c < k_hi) mt[c & 3u] = fmaxf(mt[c & 3u], __uint_as_float(sr[c]));
                    } else {
#pragma unroll
                        for (uint32_t c = 0; c < 32u; c++) mt[c & 3u] = fmaxf(mt[c & 3u], __uint_as_float(sr[c]));
                    }
                    mx = fmaxf(mx, fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3])));
                }
                mx = mx > NEG_TEST ? mx * PS_C2 : NEG_BIG; // this half row's tile maximum as a base-2 exponent
                // Lazy reference maximum: it moves only for the first valid tile or when the tile exceeds it by more than 8 (in
                // natural units). The two warps that share these 32 rows vote; only then they exchange maxima.
                if (pair_bar_or(1u + q4, !ok || (mx > NEG_TEST && (m_ref < NEG_TEST || mx > m_ref + PS_LAZY2)))) {
                    red[128u * half + row] = mx;
                    if (pair_bar_or(1u + q4, !ok)) {
                        ok = false;
                        break;
                    }
                    mx = fmaxf(mx, red[128u * (half ^ 1u) + row]);
                    float cf = 1.0f;
                    if (mx > NEG_TEST && (m_ref < NEG_TEST || mx > m_ref + PS_LAZY2)) {
                        const float m_new = fmaxf(m_ref, mx);
                        cf = m_ref > NEG_TEST ? exp2f(m_ref - m_new) : 1.0f;
                        m_ref = m_new;
                    }
                    l_run *= cf;
                    if (__any_sync(0xffffffffu, cf != 1.0f)) {
#pragma unroll
                        for (int i = 0; i < 128; i++) acc[i] *= cf;
                    }
                }
                const float neg_m = m_ref > NEG_TEST ? -m_ref : 0.0f;
                // weights 2^(s - m) as hi + lo halves, in the place of their scores; the row sums run over the f32 weights
                float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                uint32_t sr[2][16];
                tmem_ld16(s_addr, sr[0]);
#pragma unroll
                for (uint32_t c = 0; c < 4u; c++) {
                    tmem_wait_ld();
                    if (c < 3u) tmem_ld16(s_addr + 16u * (c + 1u), sr[(c + 1u) & 1u]);
                    uint32_t p[16];
#pragma unroll
                    for (uint32_t i = 0; i < 16u; i += 2u) {
                        float w0, w1;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w0) : "f"(fmaf(__uint_as_float(sr[c & 1u][i]), PS_C2, neg_m)));
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w1) : "f"(fmaf(__uint_as_float(sr[c & 1u][i + 1u]), PS_C2, neg_m)));
                        if (masked) {
                            if (16u * c + i < k_lo || 16u * c + i >= k_hi) w0 = 0.0f;
                            if (16u * c + i + 1u < k_lo || 16u * c + i + 1u >= k_hi) w1 = 0.0f;
                        }
                        sum[i & 2u] += w0;
                        sum[(i & 2u) + 1u] += w1;
                        ps_split2(w0, w1, p[i >> 1], p[8u + (i >> 1)]);
                    }
                    tmem_st16(s_addr + 16u * c, p);
                }
                l_run += (sum[0] + sum[1]) + (sum[2] + sum[3]);
                tmem_wait_st();
                tc_fence_before();
                arrive(r_p_full);
                // O += O_t, while the next tile's scores are computed
                ok = __all_sync(0xffffffffu, ps_wait(bar_o_full, g & 1u, sh, status));
                tc_fence_after();
                if (ok) {
#pragma unroll
                    for (uint32_t c = 0; c < 4u; c++) {
                        uint32_t o[32];
                        tmem_ld32(tmem + lane_addr + PS_COL_O + 128u * half + 32u * c, o);
                        tmem_wait_ld();
                        if (vis > tile_key) { // (no product has written the row of a token that sees none of the tile)
#pragma unroll
                            for (uint32_t i = 0; i < 32u; i++) acc[32u * c + i] += __uint_as_float(o[i]);
                        }
                    }
                }
                tc_fence_before();
            }
            // ---------------- end of the segment: all its products have completed ----------------
            red[128u * half + row] = l_run;
            if (pair_bar_or(1u + q4, !ok)) {
                ok = false;
                break;
            }
            const float l_all = red[row] + red[128u + row];
            if (sg.npieces == 1u) {
                // the whole item: out[tok][head][:] = O / l
                const float inv = 1.0f / l_all;
#pragma unroll
                for (uint32_t c = 0; c < 4u; c++) {
                    __syncwarp();
#pragma unroll
                    for (uint32_t k = 0; k < 8u; k++)
                        *reinterpret_cast<float4 *>(qmine + swz128(lane, k)) =
                            make_float4(acc[32u * c + 4u * k] * inv, acc[32u * c + 4u * k + 1u] * inv, acc[32u * c + 4u * k + 2u] * inv,
                                        acc[32u * c + 4u * k + 3u] * inv);
                    __syncwarp();
#pragma unroll
                    for (uint32_t i = 0; i < 8u; i++) { // eight lanes write a row's 128 bytes
                        const uint32_t r = 4u * i + (lane >> 3), t = tok0 + (r & 15u), h = 8u * kvh + 2u * q4 + (r >> 4);
                        if (t < plan.ntok)
                            *reinterpret_cast<float4 *>(out + (size_t)t * 4096u + h * 256u + 128u * half + 32u * c + 4u * (lane & 7u)) =
                                *reinterpret_cast<const float4 *>(qmine + swz128(r, lane & 7u));
                    }
                }
            } else {
                // a part of an item: its partial goes to scratch memory for the merge kernel
                float *ps = scratch + pf_slot(pair, sg.piece, cta) * PF_PART;
                const bool real = tok0 + (row & 15u) < plan.ntok; // (rows beyond the block are neither written nor read)
                if (half == 0u && real) *reinterpret_cast<float2 *>(ps + 128u * 256u + 2u * row) = make_float2(m_ref, l_all);
#pragma unroll
                for (uint32_t c = 0; c < 32u; c++)
                    if (real) *reinterpret_cast<float4 *>(ps + ((size_t)(32u * half + c) * 128u + row) * 4u) =
                        make_float4(acc[4u * c], acc[4u * c + 1u], acc[4u * c + 2u], acc[4u * c + 3u]);
            }
            pair_bar_sync(1u + q4); // red[] is free for the next segment
        }
        // The other warpgroups take their registers back behind this barrier only (see verify_f32_tc.cu).
        asm volatile("setmaxnreg.dec.sync.aligned.u32 128;");
        ps_bar_roles();
    }

    // ---------------- teardown: nothing of the pair may still be in flight, then free the tensor memory ----------------
    tc_fence_before();
    __syncwarp();
    if (sh->abort) { // a wait ran out somewhere: give copies already issued into this CTA's shared memory time to land
        const long long t0 = clock64();
        while (clock64() - t0 < 200000000ll) __nanosleep(1000);
    }
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc2(tmem, PS_COLS);
    }
}

mkv_status prefill_f32_tc_setup_device() {
    MKV_CUDA(cudaFuncSetAttribute(prefill_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PS_SMEM));
    return MKV_OK;
}

mkv_status launch_prefill_f32_tc(Ctx *ctx, Cache *c, int layer, uint32_t first_pos, uint32_t pos0, uint32_t ntok, const float *q, float *out) {
    const PfPlan plan = pf_plan(ctx, PS_COST, first_pos, pos0, ntok);
    const CUtensorMap &km = c->maps_host[2 * (c->n_layers + layer)], &vm = c->maps_host[2 * (c->n_layers + layer) + 1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * plan.pairs);
    cfg.blockDim = dim3(PS_THREADS);
    cfg.dynamicSmemBytes = PS_SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MKV_CUDA(cudaLaunchKernelEx(&cfg, prefill_f32_tc_kernel, km, vm, q, out, plan, c->shard_first, ctx->pf_scratch, ctx->dev_status));
    ctx->launches++;
    return launch_prefill_merge(ctx, plan, out);
}

} // namespace mkv
