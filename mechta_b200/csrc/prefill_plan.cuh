// How a prefill launch is cut into work for pairs of CTAs, shared by the kernels of both cache formats (prefill_tc.cu,
// prefill_f32_tc.cu) and the kernel that merges the parts of split items.
#pragma once
#include "internal.cuh"

namespace mkv {

constexpr uint32_t PF_KEYS = 128;   // keys per tile
// One partial of a CTA: O as [64 chunks of 4 dims][128 rows][4] (a warp's rows store and load 512 contiguous bytes), then
// [128 rows][m, l]
constexpr size_t PF_PART = 128u * 256u + 128u * 2u;

// The work of one launch. Items are numbered longest first: item i = (group of 32 tokens ngroups - 1 - i / 2, KV head i % 2);
// its tiles are the 128-key tiles from first_pos / 128 up to the last key its last token sees. Pairs of CTAs take
//   per = 1: whole items, item after item to and fro over the pairs;
//   per > 1: one of `per` equal parts of an item each;
//   per = 0: the tiles [p * len, (p + 1) * len) of all items laid end to end.
struct PfPlan {
    uint32_t first_pos, pos0, ntok;
    uint32_t ngroups, nitems, t0;
    uint32_t per, pairs;
    uint32_t total, len; // per = 0
    __host__ __device__ uint32_t group_of(uint32_t item) const { return ngroups - 1u - (item >> 1); }
    __host__ __device__ uint32_t item_end(uint32_t item) const { // the token after the item's last one
        const uint32_t e = group_of(item) * 32u + 32u;
        return e < ntok ? e : ntok;
    }
    __host__ __device__ uint32_t tiles_of(uint32_t item) const {
        return (pos0 + item_end(item) + PF_KEYS - 1u) / PF_KEYS - t0;
    }
    __host__ __device__ uint32_t part_len(uint32_t n) const { return (n + per - 1u) / per; } // per > 0: tiles of a part of an item of n tiles
};
struct PfSegment {
    uint32_t item, a, b;     // tiles [a, b) of the item
    uint32_t piece, npieces; // which part of the item this is, of how many
};
// Walks the segments of one pair.
struct PfWalk {
    const PfPlan &p;
    uint32_t pair, lo, hi, item, base; // per > 0: base = rounds over the pairs so far
    __device__ __forceinline__ PfWalk(const PfPlan &plan, uint32_t pair_) : p(plan), pair(pair_), item(0), base(0) {
        lo = min(pair * p.len, p.total);
        hi = min(lo + p.len, p.total);
    }
    __device__ __forceinline__ bool next(PfSegment &s) {
        if (p.per > 0u) {
            const uint32_t u = base * p.pairs + ((base & 1u) ? p.pairs - 1u - pair : pair);
            base++;
            if (u >= p.nitems * p.per) return false;
            const uint32_t it = u / p.per, piece = u % p.per, n = p.tiles_of(it), l = p.part_len(n);
            if (piece * l >= n) return false; // (per > 1, where a pair has one part: an item of so few tiles has fewer parts)
            s = {it, piece * l, min(piece * l + l, n), piece, (n + l - 1u) / l};
            return true;
        }
        while (item < p.nitems && base < hi) {
            const uint32_t n = p.tiles_of(item), a = max(base, lo), b = min(base + n, hi);
            if (b > a) {
                const uint32_t c0 = base / p.len;
                s = {item, a - base, b - base, pair - c0, (base + n - 1u) / p.len - c0 + 1u};
            }
            const bool found = b > a;
            base += n;
            item++;
            if (found) return true;
        }
        return false;
    }
};
// The rows of a CTA whose tokens see none of the keys from `key` on, as lanes of a group of 32 (rows are head * 16 + token, so a group
// is two heads of the same 16 tokens); tok_pos = position of the CTA's first token. P V leaves these rows out, 16 keys at a time
// (the K of one MMA): their weights are zero, but zero times an infinity or NaN in a later token's V row, or in a row past the
// block, is not.
__device__ __forceinline__ uint32_t pf_blind_rows(uint32_t key, uint32_t tok_pos) {
    const uint32_t m = (1u << (key > tok_pos ? min(key - tok_pos, 16u) : 0u)) - 1u;
    return m | m << 16;
}
// Where a pair's CTA keeps the partial of a part: a pair has at most one segment that continues an item begun by the pair
// before it (slot 0) and at most one that begins an item it does not finish (slot 1).
__host__ __device__ inline size_t pf_slot(uint32_t pair, uint32_t piece, uint32_t cta) {
    return ((size_t)pair * 2u + (piece == 0u ? 1u : 0u)) * 2u + cta;
}

// What parts cost a kernel, in units of its time for a tile: a segment (queries, pipeline, outputs or partial), the launch of the
// merge, and a part's way through memory.
struct PfCost {
    float segment, merge, part;
};
// The plan of a launch. Without the partials' scratch (prefill_reserve) items stay whole.
PfPlan pf_plan(Ctx *ctx, const PfCost &cost, uint32_t first_pos, uint32_t pos0, uint32_t ntok);
// Merges the split items of the launch in front, if it has any.
mkv_status launch_prefill_merge(Ctx *ctx, const PfPlan &plan, float *out);

} // namespace mkv
