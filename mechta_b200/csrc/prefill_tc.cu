// Prefill attention over the f16 cache on the 5th-generation tensor cores: tcgen05.mma by CTA pairs, with the S and O
// accumulators and the queries in tensor memory, K/V tiles staged by TMA.
//
// Stands in for q_f16 + attn_fa_mx + attn_fd_combine (W/fa_mx.wgsl:19-115,313-319; M/engine.rs:1215-1226): token T
// of the block (at pos0 + T) sees first_pos <= key < pos0 + 1 + T; the block's K/V rows were appended before
// (M/engine.rs:1213-1214).
//
// A work item is 32 tokens x the 8 query heads of one KV head = 256 rows: the M = 256 of a tcgen05.mma.cta_group::2, 128
// rows in each CTA of a pair (16 tokens a CTA, row = head * 16 + token, the reference's row order, W/fa_mx.wgsl:4). The two
// CTAs share every K/V tile of 128 keys: each loads one half of it (64 keys of K, 128 of the 256 dims of V) into its own
// shared memory and the tensor cores of both read both halves. With one CTA per 128 rows the kernel was bound by the L2 ->
// SM traffic of the tiles (9.1 GB a layer at 2,048 tokens over a 32,768-token prefix, 8.7 TB/s with the products switched
// off) and by the issue of products with N = 64; a pair needs half the traffic, and its products are 256x128x16 and
// 256x256x16. Measured, ten layers of 2,048 tokens over 32,768: 12.3 -> 9.7 ms (1,170 TFLOP/s under the power cap; a few layers
// in a burst run at 1,345). The waits use mbarrier.try_wait and the remote arrivals mbarrier.arrive at their default scope: with
// .acquire.cluster, which costs a cache invalidation each time, the same kernel took 1,032 us a layer instead of 843. No thread
// loads what a thread of the other CTA stored: what crosses the pair are tiles, weights and accumulators, which TMA and the tensor
// cores read and write (each writer's fence.proxy.async or tcgen05 fence in front of its arrival, tcgen05.commit or complete_tx
// behind the asynchronous ones).
//
// Scheduling. The grid is at most one pair of CTAs per two SMs; pf_plan decides what each pair takes: whole items, equal parts
// of items, or equal ranges of the tiles of all items laid end to end (prefill_plan.cuh). A pair walks its work segment by
// segment; a segment that covers its whole item writes the output, a part of an item writes its un-normalised partial
// (reference maximum, sum, O) to scratch memory, and a second small kernel merges the parts in index order over the whole chip
// (the reference splits long prefills over chunks and merges with attn_fd_combine in the same way, M/engine.rs:1219-1225). 200
// tokens over 9,001: 256 -> 40 us a layer (one CTA per split item used to merge it alone, with uncoalesced loads).
//
// Roles (320 threads): warp 0 = TMA producer, warp 1 = MMA issuer (one thread, of the pair's first CTA only) and TMEM owner,
// warps 2..9 = softmax, two threads per row (64 of a tile's 128 keys each). Per tile: S = Q K^T (16 MMAs, A = Q from tensor
// memory); the row's threads read S, release it (so that the next tile's S is computed while this one is in softmax), scale,
// mask, exponentiate against a reference maximum that only moves when the tile exceeds it by more than 8 (the reference's
// lazy maximum, M/dmx.rs:80 and W/fa_mx.wgsl:120: a matrix accumulator cannot be rescaled per row cheaply), write P as f16 to
// shared memory; O += P V (8 MMAs, V used N-major straight from its TMA tile). Rows that see none of an MMA's 16 keys are left out of
// it (pf_blind_rows); a row that sees no key of a segment has l = 0 there and its O, which no product has written, is not used.
// TMEM: O = columns 0..255, S = 256..383, Q (f16) = 384..511. Every wait is bounded; TMEM is freed on every path.
#include <stdlib.h>

#include <algorithm>

#include "internal.cuh"
#include "prefill_plan.cuh"
#include "ptx.cuh"

namespace mkv {
using namespace ptx;

constexpr int TC_NST = 3;                              // ring depth, K and V each
constexpr uint32_t TC_BOX = 8192;                      // one TMA box [64 keys][64 dims] f16 (PF_TILE rows)
constexpr uint32_t TC_HALF = 32768;                    // a CTA's half of a K or V tile
constexpr uint32_t TC_OFF_V = TC_NST * TC_HALF;
constexpr uint32_t TC_OFF_P = 2 * TC_NST * TC_HALF;    // [2 key blocks][128 rows][64 keys] f16
constexpr uint32_t TC_OFF_RED = TC_OFF_P + 32768;      // [2 halves][128 rows] floats
constexpr uint32_t TC_OFF_BAR = TC_OFF_RED + 1024;
// barriers: k_full[NST], v_full[NST], k_empty[NST], v_empty[NST], s_full, s_free, p_full, pv_done, q_full
constexpr uint32_t TC_NBAR = 4 * TC_NST + 5;
constexpr uint32_t TC_OFF_MISC = TC_OFF_BAR + TC_NBAR * 8; // TcShared
constexpr uint32_t TC_SMEM = TC_OFF_MISC + 32 + 1024;
constexpr uint32_t TC_COL_O = 0, TC_COL_S = 256, TC_COL_Q = 384, TC_COLS = 512;
constexpr int TC_THREADS = 320;
constexpr int TC_ROW_OUTSIDE = 1 << 30;                // a row coordinate beyond any cache: TMA fills such a box with zeros
constexpr long long TC_WAIT_LIMIT = 2000000000ll;
constexpr float TC_LOG2E = 1.4426950408889634f;
constexpr float TC_LAZY2 = 8.0f * TC_LOG2E;
constexpr float TC_C2 = SCALE * TC_LOG2E;              // scores to base-2 exponents
constexpr PfCost TC_COST = {2.8f, 1.7f, 0.075f};     // a tile takes about 1.75 us
static_assert(TC_SMEM <= 232448, "shared memory of prefill_f16_tc_kernel");

struct TcShared {
    uint32_t tmem_base;
    volatile uint32_t abort;
};

// Bounded wait shared by all roles: returns false (and raises the CTA's abort flag) when it runs out or when
// another thread already gave up.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, TcShared *sh, uint32_t *status) {
    if (sh->abort) return false;
    if (mbar_wait_bounded(bar, parity, TC_WAIT_LIMIT)) return true;
    sh->abort = 1;
    atomicOr(status, DEV_ERR_WAIT_TIMEOUT);
    return false;
}

// QF16: the queries come as f16 [ntok][16][256] (the output of the reference's q_f16 pass) instead of f32.
template <bool QF16>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
prefill_f16_tc_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                      const void *__restrict__ q, float *__restrict__ out, const __grid_constant__ PfPlan plan, uint32_t row0,
                      float *__restrict__ scratch, uint32_t *__restrict__ status, uint32_t phase_arg) {
    // phase (builds with -DMKV_MEASURE only): 0 = everything, 1 = tile loads only, 2 = loads and MMAs without the softmax math
#ifdef MKV_MEASURE
    const uint32_t phase = phase_arg;
#else
    constexpr uint32_t phase = 0u;
    (void)phase_arg;
#endif
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u; // the same in both CTAs
    uint8_t *smem = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cta = cluster_ctarank(), pair = blockIdx.x >> 1;
    const uint32_t bar0 = smem_base + TC_OFF_BAR;
    const uint32_t bar_k_full = bar0, bar_v_full = bar0 + 8u * TC_NST, bar_k_empty = bar0 + 16u * TC_NST, bar_v_empty = bar0 + 24u * TC_NST;
    const uint32_t bar_s_full = bar0 + 32u * TC_NST, bar_s_free = bar_s_full + 8u, bar_p_full = bar_s_free + 8u;
    const uint32_t bar_pv_done = bar_p_full + 8u, bar_q_full = bar_pv_done + 8u;
    TcShared *sh = reinterpret_cast<TcShared *>(smem + TC_OFF_MISC);
    pdl_launch_dependents();

    if (tid == 0) {
        for (int s = 0; s < 4 * TC_NST; s++) mbar_init(bar0 + 8u * s, 1);
        mbar_init(bar_s_full, 1);
        mbar_init(bar_s_free, 16); // one arrival per softmax warp of the pair (counted in the first CTA only)
        mbar_init(bar_p_full, 16);
        mbar_init(bar_pv_done, 1);
        mbar_init(bar_q_full, 16);
        sh->abort = 0;
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc2(smem_base + TC_OFF_MISC, TC_COLS); // writes sh->tmem_base
    tc_fence_before();
    cluster_sync(); // barriers and tensor memory of both CTAs are there
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait(); // nothing global is touched before the kernel in front has finished

    // Every role walks the same segments; g counts the tiles this pair has dealt with so far, across segments: ring
    // stage g % NST and the parities of the barriers follow from it.
    if (warp == 0) {
        // ---------------- TMA producer: runs ahead of the other roles, also across segment borders ----------------
        if (lane == 0) {
            uint32_t g = 0;
            PfWalk walk(plan, pair);
            PfSegment sg;
            bool ok = true;
            while (ok && walk.next(sg)) {
                const int x = (int)((sg.item & 1u) * 256u);
                const uint32_t end = plan.pos0 + plan.item_end(sg.item); // no key at or past this one is seen by the item's tokens
                for (uint32_t j = sg.a; j < sg.b; j++, g++) {
                    const uint32_t s = g % TC_NST, key0 = (plan.t0 + j) * PF_KEYS;
                    // A half tile without a key for any of the item's tokens is not read: its weights are zero, but zero times
                    // an infinity or NaN left in such a V row is not. (The first half can only lie below first_pos.)
                    const int y[2] = {key0 + 64u > plan.first_pos ? (int)(key0 - row0) : TC_ROW_OUTSIDE,
                                      key0 + 64u < end ? (int)(key0 + 64u - row0) : TC_ROW_OUTSIDE};
                    const uint32_t par = ((g / TC_NST) - 1u) & 1u;
                    if (g >= (uint32_t)TC_NST && !(ok = tc_wait(bar_k_empty + 8u * s, par, sh, status))) break;
                    // both CTAs' halves are counted on the first CTA's barrier: its MMA thread is the one that waits
                    uint32_t dst = smem_base + s * TC_HALF, bar = cluster_map(bar_k_full + 8u * s, 0);
                    if (cta == 0) mbar_expect_tx(bar_k_full + 8u * s, 2u * TC_HALF);
#pragma unroll
                    for (int db = 0; db < 4; db++) tma_load_2d_pair(dst + db * TC_BOX, &kmap, x + 64 * db, y[cta], bar);
                    if (g >= (uint32_t)TC_NST && !(ok = tc_wait(bar_v_empty + 8u * s, par, sh, status))) break;
                    dst = smem_base + TC_OFF_V + s * TC_HALF;
                    bar = cluster_map(bar_v_full + 8u * s, 0);
                    if (cta == 0) mbar_expect_tx(bar_v_full + 8u * s, 2u * TC_HALF);
#pragma unroll
                    for (int db = 0; db < 2; db++)
#pragma unroll
                        for (int kb = 0; kb < 2; kb++)
                            tma_load_2d_pair(dst + (2 * db + kb) * TC_BOX, &vmap, x + 128 * (int)cta + 64 * db, y[kb], bar);
                }
            }
            // the last releases must have arrived here before this CTA may leave: they come from the other CTA's commits
            for (uint32_t i = g > (uint32_t)TC_NST ? g - TC_NST : 0u; ok && i < g; i++)
                ok = tc_wait(bar_k_empty + 8u * (i % TC_NST), (i / TC_NST) & 1u, sh, status) &&
                     tc_wait(bar_v_empty + 8u * (i % TC_NST), (i / TC_NST) & 1u, sh, status);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0 && cta == 0) {
            constexpr uint32_t IDESC_QK = tc_idesc_f16(256, 128, false);
            constexpr uint32_t IDESC_PV = tc_idesc_f16(256, 256, true);
            uint32_t g = 0, nseg = 0;
            auto qk = [&](uint32_t gg) -> bool { // S = Q K^T for tile gg
                const uint32_t s = gg % TC_NST;
                if (gg > 0u && !tc_wait(bar_s_free, (gg - 1u) & 1u, sh, status)) return false;
                if (!tc_wait(bar_k_full + 8u * s, (gg / TC_NST) & 1u, sh, status)) return false;
                tc_fence_after();
                const uint32_t kb = smem_base + s * TC_HALF;
#pragma unroll
                for (uint32_t ks = 0; ks < 16u; ks++) { // 16 dims per MMA; 4 per 64-dim box
                    const uint64_t b = tc_desc_sw128(kb + (ks >> 2) * TC_BOX + (ks & 3u) * 32u, 16, 1024);
                    if (phase != 1u) tc_mma2_f16_ta(tmem + TC_COL_S, tmem + TC_COL_Q + 8u * ks, b, IDESC_QK, ks > 0 ? 1u : 0u);
                }
                tc_commit2(bar_k_empty + 8u * s);
                tc_commit2(bar_s_full);
                return true;
            };
            PfWalk walk(plan, pair);
            PfSegment sg;
            bool ok = true;
            while (ok && walk.next(sg)) {
                // the segment's Q is in tensor memory (the softmax threads put it there once the scores of the segment
                // before it were all there)
                if (!(ok = tc_wait(bar_q_full, nseg & 1u, sh, status))) break;
                tc_fence_after();
                nseg++;
                const uint32_t n = sg.b - sg.a, tok_pos = plan.pos0 + 32u * plan.group_of(sg.item);
                if (!(ok = qk(g))) break;
                // Tiles of which every token sees all keys, then the one or two at the item's end, where an MMA leaves out the rows
                // that see none of its 16 keys and MMAs that no row has a share in are not issued. (With one loop for both, ten layers
                // of 2,048 tokens over 32,768 took 1.5 % longer; leaving rows out in every MMA, 7 %.)
                const uint32_t whole = min(n, max((tok_pos + 1u) / PF_KEYS, plan.t0 + sg.a) - (plan.t0 + sg.a));
                uint32_t j = 0;
                for (; j < whole; j++, g++) {
                    if (j + 1u < n && !(ok = qk(g + 1u))) break; // the next tile's scores while this one is in softmax
                    const uint32_t s = g % TC_NST;
                    if (!(ok = tc_wait(bar_v_full + 8u * s, (g / TC_NST) & 1u, sh, status))) break;
                    if (!(ok = tc_wait(bar_p_full, g & 1u, sh, status))) break;
                    tc_fence_after();
                    const uint32_t vb = smem_base + TC_OFF_V + s * TC_HALF, pb = smem_base + TC_OFF_P;
#pragma unroll
                    for (uint32_t ks = 0; ks < 8u; ks++) { // 16 keys per MMA
                        const uint64_t a = tc_desc_sw128(pb + (ks >> 2) * 16384u + (ks & 3u) * 32u, 16, 1024);
                        // V half [2 blocks of 64 dims][128 keys], N-major: the next 64 dims 16 KB on, the next 8 keys 1024 bytes
                        const uint64_t b = tc_desc_sw128(vb + ks * 2048u, 2u * TC_BOX, 1024);
                        if (phase != 1u) tc_mma2_f16(tmem + TC_COL_O, a, b, IDESC_PV, (j > 0 || ks > 0) ? 1u : 0u);
                    }
                    tc_commit2(bar_v_empty + 8u * s);
                    tc_commit2(bar_pv_done); // O holds the segment's tiles so far; P may be overwritten
                }
                for (; ok && j < n; j++, g++) {
                    if (j + 1u < n && !(ok = qk(g + 1u))) break;
                    const uint32_t s = g % TC_NST;
                    if (!(ok = tc_wait(bar_v_full + 8u * s, (g / TC_NST) & 1u, sh, status))) break;
                    if (!(ok = tc_wait(bar_p_full, g & 1u, sh, status))) break;
                    tc_fence_after();
                    const uint32_t vb = smem_base + TC_OFF_V + s * TC_HALF, pb = smem_base + TC_OFF_P;
#pragma unroll 1
                    for (uint32_t ks = 0; ks < 8u; ks++) {
                        const uint32_t key = (plan.t0 + sg.a + j) * PF_KEYS + 16u * ks;
                        if (key > tok_pos + 31u) break;
                        const uint32_t off0 = pf_blind_rows(key, tok_pos), off1 = pf_blind_rows(key, tok_pos + 16u);
                        const uint64_t a = tc_desc_sw128(pb + (ks >> 2) * 16384u + (ks & 3u) * 32u, 16, 1024);
                        const uint64_t b = tc_desc_sw128(vb + ks * 2048u, 2u * TC_BOX, 1024);
                        const uint32_t acc = (j > 0 || ks > 0) ? 1u : 0u;
                        if (phase == 1u) continue;
                        if ((off0 | off1) == 0u) tc_mma2_f16(tmem + TC_COL_O, a, b, IDESC_PV, acc);
                        else tc_mma2_f16_off(tmem + TC_COL_O, a, b, IDESC_PV, acc, off0, off1);
                    }
                    tc_commit2(bar_v_empty + 8u * s);
                    tc_commit2(bar_pv_done);
                }
            }
        }
    } else {
        // ---------------- softmax: two threads per row (TMEM lane), 64 keys of a tile and 128 dims of O each ----------------
        const uint32_t q4 = warp & 3u, half = (warp - 2u) >> 2;
        const uint32_t row = 32u * q4 + lane; // the TMEM lanes this warp may access
        const uint32_t lane_addr = (32u * q4) << 16;
        const uint32_t r_s_free = cluster_map(bar_s_free, 0), r_p_full = cluster_map(bar_p_full, 0), r_q_full = cluster_map(bar_q_full, 0);
        float *red = reinterpret_cast<float *>(smem + TC_OFF_RED);
        auto arrive = [&](uint32_t bar) { // one arrival per warp, after all its lanes
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(bar);
        };
        // This warp's own 4 KB of the P buffer (its rows, its 64 keys) is where rows change hands between "a lane has a row" (tensor
        // memory) and "a few lanes share a row" (coalesced global accesses): free whenever the products so far have completed.
        uint8_t *stage = smem + TC_OFF_P + 16384u * half + 4096u * q4;
        // Q of an item goes to tensor memory as the A operand of S = Q K^T (q_f16 of the reference, W/fa_mx.wgsl:313-319), as
        // f16, two values per 32-bit column: the warp loads 64 dims of its 32 rows at a time, whole lines, and a lane stores its
        // row. (With every lane loading its own row straight from global memory this took 8 us of a segment for f32 queries
        // and 3 us for f16 ones.) Rows of tokens past the block are not loaded, which one token over 16 keys feels: 10.3 us a layer
        // with such rows loaded from the last token's and then zeroed, 9.2 without (f16 queries: 8.9 and 8.6).
        auto load_q = [&](const PfSegment &sg) {
            const uint32_t t0 = plan.group_of(sg.item) * 32u + 16u * cta, h0 = 8u * (sg.item & 1u) + 2u * q4;
            auto src_of = [&](uint32_t r) { // element offset of the warp's row r (= head * 16 + token), this half's first dim
                return (size_t)(t0 + (r & 15u)) * 4096u + (size_t)(h0 + (r >> 4)) * 256u + 128u * half;
            };
            constexpr int NL = QF16 ? 8 : 16; // 16-byte loads of a lane per 64 dims
            uint4 v[2][NL];
#pragma unroll
            for (int c0 = 0; c0 < 2; c0++)
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const uint32_t r = QF16 ? 4u * i + (lane >> 3) : 2u * i + (lane >> 4);
                    const void *src = QF16 ? static_cast<const void *>(static_cast<const __half *>(q) + src_of(r) + 64u * c0 + 8u * (lane & 7u))
                                           : static_cast<const void *>(static_cast<const float *>(q) + src_of(r) + 64u * c0 + 4u * (lane & 15u));
                    v[c0][i] = t0 + (r & 15u) < plan.ntok ? __ldg(static_cast<const uint4 *>(src)) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
            for (int c0 = 0; c0 < 2; c0++) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < NL; i++) {
                    const uint4 a = v[c0][i];
                    if constexpr (QF16) {
                        *reinterpret_cast<uint4 *>(stage + swz128(4u * i + (lane >> 3), lane & 7u)) = a;
                    } else {
                        const __half2 h0 = __floats2half2_rn(__uint_as_float(a.x), __uint_as_float(a.y));
                        const __half2 h1 = __floats2half2_rn(__uint_as_float(a.z), __uint_as_float(a.w));
                        *reinterpret_cast<uint2 *>(stage + swz128(2u * i + (lane >> 4), (lane & 15u) >> 1) + 8u * (lane & 1u)) =
                            make_uint2(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1));
                    }
                }
                __syncwarp();
                uint32_t w[32];
#pragma unroll
                for (uint32_t c = 0; c < 8u; c++) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(stage + swz128(lane, c));
                    w[4 * c] = a.x; w[4 * c + 1] = a.y; w[4 * c + 2] = a.z; w[4 * c + 3] = a.w;
                }
                tmem_st32(tmem + lane_addr + TC_COL_Q + 64u * half + 32u * c0, w);
            }
            tmem_wait_st();
            tc_fence_before();
            arrive(r_q_full);
        };
        uint32_t g = 0;
        PfWalk walk(plan, pair);
        PfSegment sg, nx;
        bool more = walk.next(sg), ok = true;
        if (more) load_q(sg);
        while (more) {
            const uint32_t tok0 = plan.group_of(sg.item) * 32u + 16u * cta, kvh = sg.item & 1u;
            const uint32_t vis = plan.pos0 + 1u + tok0 + (row & 15u); // the row's token sees keys < vis
            const uint32_t full_below = plan.pos0 + 1u + tok0; // keys below this are visible to every row of the CTA
            float m_ref = NEG_BIG, l_run = 0.0f; // l_run: this thread's 64 keys of every tile only
            const uint32_t n = sg.b - sg.a;
            for (uint32_t j = 0; j < n; j++, g++) {
                // The warp takes every wait's outcome together: the TMEM loads below are warp-collective. A wait that ran out
                // goes into the next vote, so that the two warps of these rows leave together.
                ok = __all_sync(0xffffffffu, tc_wait(bar_s_full, g & 1u, sh, status)) && ok;
                tc_fence_after();
                if (phase != 0u) { // measurement: no softmax math, P left as it is
                    tc_fence_before();
                    arrive(r_s_free);
                    if (j > 0) ok = __all_sync(0xffffffffu, tc_wait(bar_pv_done, (g - 1u) & 1u, sh, status)) && ok;
                    if (!ok) break; // (no vote in this mode before the segment's end)
                    arrive(r_p_full);
                    continue;
                }
                uint32_t sr[2][32];
                tmem_ld32(tmem + lane_addr + TC_COL_S + 64u * half, sr[0]);
                tmem_ld32(tmem + lane_addr + TC_COL_S + 64u * half + 32u, sr[1]);
                tmem_wait_ld();
                tc_fence_before();
                arrive(r_s_free); // the next tile's scores may be computed
                const uint32_t key_base = (plan.t0 + sg.a + j) * PF_KEYS + 64u * half;
                // work in base-2 exponents: exp(s / 16 - m) = 2^(s * C - m2), C = log2(e) / 16, one FFMA + one ex2 per score
                float mt[4] = {NEG_BIG, NEG_BIG, NEG_BIG, NEG_BIG};
                if (key_base + 64u > full_below || key_base < plan.first_pos) { // the causal diagonal or the window start (W/fa_mx.wgsl:62)
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int c = 0; c < 32; c++) {
                            const uint32_t key = key_base + 32u * h + c;
                            const float v = (key >= plan.first_pos && key < vis) ? __uint_as_float(sr[h][c]) : NEG_BIG;
                            sr[h][c] = __float_as_uint(v);
                            mt[c & 3] = fmaxf(mt[c & 3], v);
                        }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int c = 0; c < 32; c++) mt[c & 3] = fmaxf(mt[c & 3], __uint_as_float(sr[h][c]));
                }
                float mx = fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3]));
                mx = mx > NEG_TEST ? mx * TC_C2 : NEG_BIG; // this half row's tile maximum as a base-2 exponent
                // Lazy reference maximum: it moves only for the first valid tile or when the tile exceeds it by more than 8 (in
                // natural units, as the reference). The two warps that share these 32 rows vote; only then they exchange maxima.
                float cf = 1.0f;
                if (pair_bar_or(1u + q4, !ok || (mx > NEG_TEST && (m_ref < NEG_TEST || mx > m_ref + TC_LAZY2)))) {
                    red[128u * half + row] = mx;
                    if (pair_bar_or(1u + q4, !ok)) {
                        ok = false;
                        break;
                    }
                    mx = fmaxf(mx, red[128u * (half ^ 1u) + row]);
                    if (mx > NEG_TEST && (m_ref < NEG_TEST || mx > m_ref + TC_LAZY2)) {
                        const float m_new = fmaxf(m_ref, mx);
                        cf = m_ref > NEG_TEST ? exp2f(m_ref - m_new) : 1.0f;
                        m_ref = m_new;
                    }
                }
                const float neg_m = m_ref > NEG_TEST ? -m_ref : 0.0f; // masked scores stay at -3e38 * C: 2^that = 0
                float sum[2] = {0.0f, 0.0f};
                uint32_t ph[32]; // 64 weights as f16 pairs
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        float w0, w1;
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w0) : "f"(fmaf(__uint_as_float(sr[h][c]), TC_C2, neg_m)));
                        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w1) : "f"(fmaf(__uint_as_float(sr[h][c + 1]), TC_C2, neg_m)));
                        sum[0] += w0;
                        sum[1] += w1;
                        const __half2 hp = __floats2half2_rn(w0, w1);
                        ph[16 * h + (c >> 1)] = *reinterpret_cast<const uint32_t *>(&hp);
                    }
                l_run = l_run * cf + (sum[0] + sum[1]);
                // P and O belong to the MMAs of the tile before until those have completed
                if (j > 0) ok = __all_sync(0xffffffffu, tc_wait(bar_pv_done, (g - 1u) & 1u, sh, status));
                tc_fence_after();
                if (j > 0 && __any_sync(0xffffffffu, cf != 1.0f)) { // rescale this warp's rows and dims of O (rare)
#pragma unroll 1
                    for (uint32_t c0 = 0; c0 < 128u; c0 += 32u) {
                        uint32_t orow[32];
                        tmem_ld32(tmem + lane_addr + TC_COL_O + 128u * half + c0, orow);
                        tmem_wait_ld();
#pragma unroll
                        for (int c = 0; c < 32; c++) orow[c] = __float_as_uint(__uint_as_float(orow[c]) * cf);
                        tmem_st32(tmem + lane_addr + TC_COL_O + 128u * half + c0, orow);
                    }
                    tmem_wait_st();
                }
                uint8_t *prow = smem + TC_OFF_P + 16384u * half;
#pragma unroll
                for (uint32_t c = 0; c < 8u; c++) // 8 chunks of 8 keys
                    *reinterpret_cast<uint4 *>(prow + swz128(row, c)) = make_uint4(ph[4 * c], ph[4 * c + 1], ph[4 * c + 2], ph[4 * c + 3]);
                fence_proxy_async();
                tc_fence_before();
                arrive(r_p_full);
            }
            // ---------------- end of the segment: all its MMAs have completed ----------------
            ok = ok && __all_sync(0xffffffffu, tc_wait(bar_pv_done, (g - 1u) & 1u, sh, status));
            tc_fence_after();
            more = ok && walk.next(nx);
            if (more) load_q(nx); // the next segment's first scores are computed while this one's epilogue runs
            red[128u * half + row] = l_run;
            if (pair_bar_or(1u + q4, !ok)) break;
            const float l_all = red[row] + red[128u + row];
            if (sg.npieces == 1u) {
                // the whole item: out[tok][head][:] = O / l
                const float inv = 1.0f / l_all;
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < 128u; c0 += 32u) {
                    uint32_t orow[32];
                    tmem_ld32(tmem + lane_addr + TC_COL_O + 128u * half + c0, orow);
                    tmem_wait_ld();
                    __syncwarp();
#pragma unroll
                    for (uint32_t c = 0; c < 8u; c++)
                        *reinterpret_cast<float4 *>(stage + swz128(lane, c)) =
                            make_float4(__uint_as_float(orow[4 * c]) * inv, __uint_as_float(orow[4 * c + 1]) * inv,
                                        __uint_as_float(orow[4 * c + 2]) * inv, __uint_as_float(orow[4 * c + 3]) * inv);
                    __syncwarp();
#pragma unroll
                    for (uint32_t i = 0; i < 8u; i++) { // eight lanes write a row's 128 bytes
                        const uint32_t r = 4u * i + (lane >> 3), t = tok0 + (r & 15u), h = 8u * kvh + 2u * q4 + (r >> 4);
                        if (t < plan.ntok)
                            *reinterpret_cast<float4 *>(out + (size_t)t * 4096u + h * 256u + 128u * half + c0 + 4u * (lane & 7u)) =
                                *reinterpret_cast<const float4 *>(stage + swz128(r, lane & 7u));
                    }
                }
            } else {
                // a part of an item: its partial goes to scratch memory for the merge kernel
                float *ps = scratch + pf_slot(pair, sg.piece, cta) * PF_PART;
                const bool real = tok0 + (row & 15u) < plan.ntok; // (rows beyond the block are neither written nor read)
                if (half == 0u && real) *reinterpret_cast<float2 *>(ps + 128u * 256u + 2u * row) = make_float2(m_ref, l_all);
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < 128u; c0 += 32u) {
                    uint32_t orow[32];
                    tmem_ld32(tmem + lane_addr + TC_COL_O + 128u * half + c0, orow);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; c += 4)
                        if (real) *reinterpret_cast<uint4 *>(ps + ((size_t)((128u * half + c0 + c) >> 2) * 128u + row) * 4u) =
                            make_uint4(orow[c], orow[c + 1], orow[c + 2], orow[c + 3]);
                }
            }
            tc_fence_before();
            pair_bar_sync(1u + q4); // red[] is free for the next segment
            sg = nx;
        }
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
        tmem_dealloc2(tmem, TC_COLS);
    }
}

// The pair that has an item's first part, and the number of its parts.
__device__ __forceinline__ void pf_parts(const PfPlan &plan, uint32_t item, uint32_t &p0, uint32_t &np) {
    const uint32_t n = plan.tiles_of(item);
    if (plan.per > 0u) {
        p0 = item * plan.per;
        np = (n + plan.part_len(n) - 1u) / plan.part_len(n);
    } else {
        uint32_t base = 0;
        for (uint32_t i = 0; i < item; i++) base += plan.tiles_of(i);
        p0 = base / plan.len;
        np = (base + n - 1u) / plan.len - p0 + 1u;
    }
}

// Merges the parts of split items: out = sum_s e^(m_s - M) O_s / sum_s e^(m_s - M) l_s, in a fixed order, so that the result
// does not depend on timing. One block = 32 rows (one per lane) and an eighth of the dims of one CTA's half of an item; four
// groups of two warps take every fourth part each (with the maximum of their own parts; the loads of four parts are in flight
// at once, which is what bounds this kernel: an item of few tokens over a long prefix has dozens of parts) and meet in shared
// memory, from where the output rows leave as whole lines.
__global__ void __launch_bounds__(256)
prefill_merge_kernel(const __grid_constant__ PfPlan plan, const float *__restrict__ scratch, float *__restrict__ out) {
    __shared__ float2 ml_s[4][32];
    __shared__ float4 acc_s[4][32][9];
    pdl_launch_dependents();
    const uint32_t item = blockIdx.y, cta = blockIdx.x >> 5, q4 = (blockIdx.x >> 3) & 3u, eighth = blockIdx.x & 7u;
    const uint32_t lane = threadIdx.x & 31u, grp = threadIdx.x >> 6, ch = (threadIdx.x >> 5) & 1u, row = 32u * q4 + lane;
    uint32_t p0, np;
    pf_parts(plan, item, p0, np);
    const uint32_t tok0 = plan.group_of(item) * 32u + 16u * cta;
    if (np == 1u || tok0 >= plan.ntok) return; // written by the attention kernel, or padding
    const bool real = tok0 + (row & 15u) < plan.ntok;
    pdl_wait();
    float M = NEG_BIG, l = 0.0f;
    float4 acc[4];
#pragma unroll
    for (int i = 0; i < 4; i++) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t s0 = grp; s0 < np; s0 += 16u) {
        float2 ml[4];
        float4 v[4][4];
#pragma unroll
        for (uint32_t k = 0; k < 4u; k++) {
            const uint32_t s = s0 + 4u * k;
            const float *ps = scratch + pf_slot(p0 + min(s, np - 1u), s, cta) * PF_PART; // (s > 0 from the second part on)
            ml[k] = s < np && real ? __ldcg(reinterpret_cast<const float2 *>(ps + 128u * 256u + 2u * row)) : make_float2(NEG_BIG, 0.0f);
#pragma unroll
            for (uint32_t i = 0; i < 4u; i++)
                v[k][i] = s < np && real ? __ldcg(reinterpret_cast<const float4 *>(ps + ((size_t)(8u * eighth + 4u * ch + i) * 128u + row) * 4u))
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (ml[k].y == 0.0f) { // the row's token sees no key of the part: no product has written its O
#pragma unroll
                for (int i = 0; i < 4; i++) v[k][i] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        const float mx = fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x));
        if (mx > M) {
            const float f = M > NEG_TEST ? exp2f(M - mx) : 0.0f;
            l *= f;
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i] = make_float4(acc[i].x * f, acc[i].y * f, acc[i].z * f, acc[i].w * f);
            M = mx;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float e = ml[k].x > NEG_TEST ? exp2f(ml[k].x - M) : 0.0f;
            l = fmaf(e, ml[k].y, l);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i].x = fmaf(e, v[k][i].x, acc[i].x);
                acc[i].y = fmaf(e, v[k][i].y, acc[i].y);
                acc[i].z = fmaf(e, v[k][i].z, acc[i].z);
                acc[i].w = fmaf(e, v[k][i].w, acc[i].w);
            }
        }
    }
    if (ch == 0u) ml_s[grp][lane] = make_float2(M, l);
#pragma unroll
    for (uint32_t i = 0; i < 4u; i++) acc_s[grp][lane][4u * ch + i] = acc[i];
    __syncthreads();
    const uint32_t r = threadIdx.x >> 3, c = threadIdx.x & 7u, rr = 32u * q4 + r, tok = tok0 + (rr & 15u);
    if (tok >= plan.ntok) return;
    const float Mr = fmaxf(fmaxf(ml_s[0][r].x, ml_s[1][r].x), fmaxf(ml_s[2][r].x, ml_s[3][r].x));
    float L = 0.0f;
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int g = 0; g < 4; g++) {
        const float e = ml_s[g][r].x > NEG_TEST ? exp2f(ml_s[g][r].x - Mr) : 0.0f;
        const float4 a = acc_s[g][r][c];
        L = fmaf(e, ml_s[g][r].y, L);
        y.x = fmaf(e, a.x, y.x);
        y.y = fmaf(e, a.y, y.y);
        y.z = fmaf(e, a.z, y.z);
        y.w = fmaf(e, a.w, y.w);
    }
    const float inv = 1.0f / L;
    *reinterpret_cast<float4 *>(out + (size_t)tok * 4096u + (8u * (item & 1u) + (rr >> 4)) * 256u + 32u * eighth + 4u * c) =
        make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
}

// The same for items of at most PF_FEW parts (equal parts of many items, cuts of long items): a thread takes four dims of a row
// through all parts, four loads in flight; the rows leave through shared memory as whole lines. prefill_merge_kernel's four groups
// would be idle or half so, at 121 registers a thread: ten layers, 512 tokens over 4,096 on the f32 cache (2 parts) 1,317 ->
// 1,248 us, 200 over 9,001 on the f16 cache (5 parts) 442 -> 428. us a layer, this kernel never / up to 8 parts / up to 16: 512 tokens
// over 32,768 (2 parts) 222 / 215 / 215, 200 over 9,001 41.6 / 39.4 / 39.4, 128 over 9,001 (9 parts) 30.2 / 30.2 / 29.5, 96 over 9,001
// (12 parts) 27.0 / 27.0 / 26.6; the line at 8 leaves those last 2 % where they are. With up to 4 items both kernels' blocks are one
// wave and it makes no difference (6 tokens over 849 14.4 and 14.5, 64 over 9,001 23.0 and 23.0).
constexpr uint32_t PF_FEW = 8;
__global__ void __launch_bounds__(256)
prefill_merge_few_kernel(const __grid_constant__ PfPlan plan, const float *__restrict__ scratch, float *__restrict__ out) {
    __shared__ float4 y_s[32][9];
    pdl_launch_dependents();
    const uint32_t item = blockIdx.y, cta = blockIdx.x >> 5, q4 = (blockIdx.x >> 3) & 3u, eighth = blockIdx.x & 7u;
    const uint32_t lane = threadIdx.x & 31u, ch = threadIdx.x >> 5, row = 32u * q4 + lane;
    uint32_t p0, np;
    pf_parts(plan, item, p0, np);
    const uint32_t tok0 = plan.group_of(item) * 32u + 16u * cta;
    if (np == 1u || tok0 >= plan.ntok) return; // written by the attention kernel, or padding
    const bool real = tok0 + (row & 15u) < plan.ntok;
    pdl_wait();
    float M = NEG_BIG, l = 0.0f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t s0 = 0; s0 < np; s0 += 4u) {
        float2 ml[4];
        float4 v[4];
#pragma unroll
        for (uint32_t k = 0; k < 4u; k++) {
            const uint32_t s = s0 + k;
            const float *ps = scratch + pf_slot(p0 + min(s, np - 1u), s, cta) * PF_PART; // (s > 0 from the second part on)
            ml[k] = s < np && real ? __ldcg(reinterpret_cast<const float2 *>(ps + 128u * 256u + 2u * row)) : make_float2(NEG_BIG, 0.0f);
            v[k] = s < np && real ? __ldcg(reinterpret_cast<const float4 *>(ps + ((size_t)(8u * eighth + ch) * 128u + row) * 4u))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (ml[k].y == 0.0f) v[k] = make_float4(0.f, 0.f, 0.f, 0.f); // the row's token sees no key of the part: no product has written its O
        const float mx = fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x));
        if (mx > M) {
            const float f = M > NEG_TEST ? exp2f(M - mx) : 0.0f;
            l *= f;
            acc = make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
            M = mx;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float e = ml[k].x > NEG_TEST ? exp2f(ml[k].x - M) : 0.0f;
            l = fmaf(e, ml[k].y, l);
            acc.x = fmaf(e, v[k].x, acc.x);
            acc.y = fmaf(e, v[k].y, acc.y);
            acc.z = fmaf(e, v[k].z, acc.z);
            acc.w = fmaf(e, v[k].w, acc.w);
        }
    }
    const float inv = 1.0f / l;
    y_s[lane][ch] = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    __syncthreads();
    const uint32_t r = threadIdx.x >> 3, c = threadIdx.x & 7u, rr = 32u * q4 + r, tok = tok0 + (rr & 15u);
    if (tok < plan.ntok)
        *reinterpret_cast<float4 *>(out + (size_t)tok * 4096u + (8u * (item & 1u) + (rr >> 4)) * 256u + 32u * eighth + 4u * c) = y_s[r][c];
}

mkv_status prefill_tc_setup_device() {
    MKV_CUDA(cudaFuncSetAttribute(prefill_f16_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
    MKV_CUDA(cudaFuncSetAttribute(prefill_f16_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
    return MKV_OK;
}

static bool pf_splits(const PfPlan &plan) {
    if (plan.per > 1u) return plan.part_len(plan.tiles_of(0)) < plan.tiles_of(0);
    for (uint32_t i = 0, base = 0; plan.per == 0u && i < plan.nitems; i++) {
        const uint32_t n = plan.tiles_of(i);
        if (base / plan.len != (base + n - 1u) / plan.len) return true;
        base += n;
    }
    return false;
}

void prefill_reserve(Ctx *ctx) {
    if (ctx->pf_scratch) return;
    if (cudaMalloc(&ctx->pf_scratch, 2u * (size_t)ctx->sm_count * PF_PART * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        ctx->pf_scratch = nullptr;
    }
}

// Chooses the way of the three that the cost model expects to be the fastest. Whole items need no merge but leave pairs idle
// when there are few; equal parts are one segment a pair; the end-to-end cut is even for any number of items but gives a pair
// several segments. Measured against the
// end-to-end cut alone (us a layer): 1,226 tokens over 91 77 -> 29 and 1,121 over 1,779 96 -> 51 (whole items), 200 over 9,001 45.3
// -> 40.2 (five parts an item), 32 over 9,001 24.6 -> 20.1, 5 over 16 18.5 -> 11.6; 2,048 over 32,768 is still cut end to end.
PfPlan pf_plan(Ctx *ctx, const PfCost &cost, uint32_t first_pos, uint32_t pos0, uint32_t ntok) {
    PfPlan plan;
    plan.first_pos = first_pos; plan.pos0 = pos0; plan.ntok = ntok;
    plan.ngroups = (ntok + 31u) / 32u;
    plan.nitems = 2u * plan.ngroups;
    plan.t0 = first_pos / PF_KEYS;
    plan.total = 0;
    for (uint32_t i = 0; i < plan.nitems; i += 2u) plan.total += 2u * plan.tiles_of(i);
    const uint32_t npairs = (uint32_t)ctx->sm_count / 2u, n = plan.nitems, longest = plan.tiles_of(0), shortest = plan.tiles_of(n - 1u);
    plan.len = (plan.total + npairs - 1u) / npairs;
    // end to end
    float best = (float)plan.len + (1.0f + (float)plan.len / (float)shortest) * cost.segment + cost.merge + cost.part * (float)(npairs + n);
    plan.per = 0;
    plan.pairs = (plan.total + plan.len - 1u) / plan.len;
    { // whole items: the pair that gets the most
        const uint32_t rounds = (n + npairs - 1u) / npairs;
        uint32_t most = longest;
        for (uint32_t p = 0; rounds > 1u && p < npairs; p++) {
            uint32_t t = 0;
            for (uint32_t k = 0; k < rounds; k++) {
                const uint32_t u = k * npairs + ((k & 1u) ? npairs - 1u - p : p);
                if (u < n) t += plan.tiles_of(u);
            }
            most = std::max(most, t);
        }
        const float t = (float)most + (float)rounds * cost.segment;
        if (t <= best) {
            best = t;
            plan.per = 1;
            plan.pairs = std::min(n, npairs);
        }
    }
    for (uint32_t per = 2; per * n <= npairs && per <= longest; per++) { // equal parts
        const float t = (float)((longest + per - 1u) / per) + cost.segment + cost.merge + cost.part * (float)(per * n);
        if (t < best) {
            best = t;
            plan.per = per;
            plan.pairs = per * n;
        }
    }
    if (!ctx->pf_scratch && pf_splits(plan)) {
        plan.per = 1;
        plan.pairs = std::min(n, npairs);
    }
    return plan;
}

mkv_status launch_prefill_merge(Ctx *ctx, const PfPlan &plan, float *out) {
    if (!pf_splits(plan)) return MKV_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64u, plan.nitems);
    cfg.blockDim = dim3(256);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const uint32_t most = plan.per > 0u ? plan.per : (plan.tiles_of(0) + plan.len - 1u) / plan.len + 1u; // parts of an item
    MKV_CUDA(cudaLaunchKernelEx(&cfg, most <= PF_FEW && plan.nitems > 4u ? prefill_merge_few_kernel : prefill_merge_kernel, plan, (const float *)ctx->pf_scratch, out));
    ctx->launches++;
    return MKV_OK;
}

mkv_status launch_prefill_f16_tc(Ctx *ctx, Cache *c, int layer, uint32_t first_pos, uint32_t pos0, uint32_t ntok,
                                 const void *q, bool q_is_f16, float *out) {
#ifdef MKV_MEASURE
    static const uint32_t phase = [] { const char *e = getenv("MKV_PHASE"); return e ? (uint32_t)atoi(e) : 0u; }();
#else
    const uint32_t phase = 0u;
#endif
    const PfPlan plan = pf_plan(ctx, TC_COST, first_pos, pos0, ntok);
    const CUtensorMap &km = c->maps_host[2 * (c->n_layers + layer)], &vm = c->maps_host[2 * (c->n_layers + layer) + 1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * plan.pairs);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = TC_SMEM;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (q_is_f16)
        MKV_CUDA(cudaLaunchKernelEx(&cfg, prefill_f16_tc_kernel<true>, km, vm, q, out, plan, c->shard_first, ctx->pf_scratch, ctx->dev_status, phase));
    else
        MKV_CUDA(cudaLaunchKernelEx(&cfg, prefill_f16_tc_kernel<false>, km, vm, q, out, plan, c->shard_first, ctx->pf_scratch, ctx->dev_status, phase));
    ctx->launches++;
    return launch_prefill_merge(ctx, plan, out);
}

} // namespace mkv
