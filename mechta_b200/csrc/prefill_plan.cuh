// How a prefill launch is cut into work for pairs of CTAs, shared by the kernels of both cache formats (prefill_tc.cu,
// prefill_f32_tc.cu) and the kernel that merges the parts of split items.
#pragma once
#include "internal.cuh"

namespace mkv {

constexpr uint32_t PF_KEYS = 128;   // keys per tile
constexpr uint32_t PF_MIN_LEN = 2;  // tiles a pair takes at least: a shorter range costs more in partials than it saves
// One partial of a CTA: O as [64 chunks of 4 dims][128 rows][4] (a warp's rows store and load 512 contiguous bytes), then
// [128 rows][m, l]
constexpr size_t PF_PART = 128u * 256u + 128u * 2u;

// The work of one launch. Items are numbered longest first: item i = (group of 32 tokens ngroups - 1 - i / 2, KV head i % 2);
// its tiles are the 128-key tiles from first_pos / 128 up to the last key its last token sees. Pair p takes the tiles
// [p * len, (p + 1) * len) of all items laid end to end.
struct PfPlan {
    uint32_t first_pos, pos0, ntok;
    uint32_t ngroups, nitems, t0;
    uint32_t total, len;
    __host__ __device__ uint32_t group_of(uint32_t item) const { return ngroups - 1u - (item >> 1); }
    __host__ __device__ uint32_t item_end(uint32_t item) const { // the token after the item's last one
        const uint32_t e = group_of(item) * 32u + 32u;
        return e < ntok ? e : ntok;
    }
    __host__ __device__ uint32_t tiles_of(uint32_t item) const {
        return (pos0 + item_end(item) + PF_KEYS - 1u) / PF_KEYS - t0;
    }
};
struct PfSegment {
    uint32_t item, a, b;     // tiles [a, b) of the item
    uint32_t piece, npieces; // which part of the item this is, of how many
};
// Walks the segments of one pair.
struct PfWalk {
    const PfPlan &p;
    uint32_t pair, lo, hi, item, base;
    __device__ __forceinline__ PfWalk(const PfPlan &plan, uint32_t pair_) : p(plan), pair(pair_), item(0), base(0) {
        lo = min(pair * p.len, p.total);
        hi = min(lo + p.len, p.total);
    }
    __device__ __forceinline__ bool next(PfSegment &s) {
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
// Where a pair's CTA keeps the partial of a part: a pair has at most one segment that continues an item begun by the pair
// before it (slot 0) and at most one that begins an item it does not finish (slot 1).
__host__ __device__ inline size_t pf_slot(uint32_t pair, uint32_t piece, uint32_t cta) {
    return ((size_t)pair * 2u + (piece == 0u ? 1u : 0u)) * 2u + cta;
}

PfPlan pf_plan(Ctx *ctx, uint32_t first_pos, uint32_t pos0, uint32_t ntok);
inline uint32_t pf_pairs(const PfPlan &p) { return (p.total + p.len - 1u) / p.len; }
// Scratch of the split items: two partials per CTA, allocated with the context's first prefill launch and kept until the
// context goes.
mkv_status prefill_scratch(Ctx *ctx);
// Merges the split items of the launch in front, if it has any.
mkv_status launch_prefill_merge(Ctx *ctx, const PfPlan &plan, float *out);

} // namespace mkv
