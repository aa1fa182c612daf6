// Shared by the two forms of the block-select score/top-k stage (select.cu, select_gemm.cu): order-preserving
// score keys and the per-row selection.
#pragma once
#include "common.cuh"

namespace lcbsa {
namespace sel {

// First step of the search for the threshold of a row of 16-bit keys (select_row_regs): an octave of scores
template <typename T> struct FirstStep { static constexpr uint32_t value = 0; };
template <> struct FirstStep<__nv_bfloat16> { static constexpr uint32_t value = 1u << 7; };
template <> struct FirstStep<__half> { static constexpr uint32_t value = 1u << 10; };
constexpr int kRegWords = 24;  // 32-bit words of a 16-bit key row that a lane may keep in registers (select_row_regs: rows up to 1536 keys)

template <typename T> struct KeyOf { using type = uint16_t; };
template <> struct KeyOf<float> { using type = uint32_t; };

// Order-preserving key: a larger key is a larger score; -0 equals +0; NaN ranks above +inf.
__device__ __forceinline__ uint16_t make_key(__nv_bfloat16 v) {
    uint16_t u = __bfloat16_as_ushort(v);
    if ((u & 0x7fffu) > 0x7f80u) return 0xffffu;
    if (u == 0x8000u) u = 0;
    return (u & 0x8000u) ? (uint16_t)~u : (uint16_t)(u | 0x8000u);
}
__device__ __forceinline__ uint16_t make_key(__half v) {
    uint16_t u = __half_as_ushort(v);
    if ((u & 0x7fffu) > 0x7c00u) return 0xffffu;
    if (u == 0x8000u) u = 0;
    return (u & 0x8000u) ? (uint16_t)~u : (uint16_t)(u | 0x8000u);
}
__device__ __forceinline__ uint32_t make_key(float v) {
    uint32_t u = __float_as_uint(v);
    if ((u & 0x7fffffffu) > 0x7f800000u) return 0xffffffffu;
    if (u == 0x80000000u) u = 0;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ int warp_sum(int v) { return __reduce_add_sync(0xffffffffu, v); }

// Number of keys of a row that are >= cand (gt == false) or > cand (gt == true).
__device__ __forceinline__ int count_row(const uint16_t* row, int nk_pad, uint32_t cand, bool gt, int lane) {
    const uint32_t* r32 = reinterpret_cast<const uint32_t*>(row);
    const uint32_t c = gt ? cand + 1u : cand;  // cand + 1 may be 0x10000: no 16-bit key reaches it
    int n = 0;
    for (int p = lane; p < nk_pad / 2; p += 32) {
        const uint32_t kk = r32[p];
        n += ((kk & 0xffffu) >= c) + ((kk >> 16) >= c);
    }
    return warp_sum(n);
}
__device__ __forceinline__ int count_row(const uint32_t* row, int nk_pad, uint32_t cand, bool gt, int lane) {
    int n = 0;
    for (int p = lane; p < nk_pad; p += 32) {
        const uint32_t kk = row[p];
        n += gt ? (kk > cand) : (kk >= cand);
    }
    return warp_sum(n);
}

// Which key blocks a row may select from.  Blocks are numbered frame-major (t, then h, then w); a block belongs to the
// "first part" when (its frame-block index % period) < split -- period = all frame blocks and split = the conditioning
// frame blocks for a single grid, period = the frame blocks of one rank for the rank-major grid of a context-parallel
// group.  period == 0: every block is allowed.
struct KeyMask {
    int hw, period, split;
    __device__ __forceinline__ bool operator()(int j) const { return period == 0 || ((j / hw) % period) < split; }
};

// The nsel largest keys of one row of 16-bit keys (ties at the threshold broken towards the lower block index), emitted as
// ascending block indices by one warp; the cap - nsel trailing entries are set to -1.  nk_pad (a multiple of 64, at most
// 64 * NW) entries are readable and those past Nk hold key 0, which no block that may be selected has.
//
// n_keys: keys the row may select from (it decides how the threshold is looked for, not the result).
//
// Issue bound: the row is read once (2 bytes per key) and then counted some seven times (16 bits of a plain bisection take 12
// to 17).  Every lane keeps its share of the row in registers (word i: keys 2 (lane + 32 i) and the one behind it), the low key
// of a word shifted up in a register of its own, so that a count is a compare and an add per key; NW follows the row (a fixed 24
// words spent 60 % of the work of a 624-key row on padding); the search ends as soon as a candidate is reached by exactly
// nsel keys; and the indices are emitted from the registers.  Before, with 24 words for every row, five shuffles per count, all
// 17 counts and a second read of the row: 19 968 rows of 624 keys 76 us, then 33 us; 46 080 rows of 1440 keys 199 us, then 185 us
// (there 23 of the 24 words were needed all along).
//
// Where the threshold is looked for.  Fewer than half of the keys selected: a little below the largest key.  Half or more: it
// may lie on the other side of zero, half of all 16-bit values away, so it is bisected between the smallest and the largest key.
// Scores and selection, us: always from 16 bits down (with a score kernel some 25 us slower) / always from the largest key, by an
// octave of bf16 / as here:
//   46 080 rows of 1440 keys, bf16, head_dim 128: 1/16 selected 630 / 556 / 556, half 595 / 607 / 575, three quarters 632 / 673 / 608
//   the same in fp16, head_dim 64:                1/16 selected 423 / 400 / 380, half 389 / 423 / 380, three quarters 425 / 478 / 415
template <int NW>
__device__ __forceinline__ void select_row_regs(const uint16_t* row, int n_keys, int nk_pad, int nsel, int cap, uint32_t first_step, int32_t* out,
                                                int32_t* cnt_out, int lane, const KeyMask mask = KeyMask{1, 0, 0}) {
    if (lane == 0) *cnt_out = nsel;
    if (nsel > 0) {
        const uint32_t* r32 = reinterpret_cast<const uint32_t*>(row);
        const int nwords = nk_pad / 2;
        uint32_t hi[NW], lo[NW];  // hi: the word itself (its upper key decides a comparison with c << 16), lo: the lower key << 16
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            uint32_t w = (lane + 32 * i < nwords) ? r32[lane + 32 * i] : 0u;  // key 0 is never counted
            if (mask.period != 0) {  // keys of blocks this row may not select become key 0
                const int j = 2 * (lane + 32 * i);
                if (!mask(j)) w &= 0xffff0000u;
                if (!mask(j + 1)) w &= 0x0000ffffu;
            }
            hi[i] = w;
            lo[i] = w << 16;
        }
        auto count = [&](uint32_t c) {  // keys >= c, 1 <= c <= 0xffff
            int n = 0;
            const uint32_t cc = c << 16;
#pragma unroll
            for (int i = 0; i < NW; ++i) n += (int)(hi[i] >= cc) + (int)(lo[i] >= cc);
            return warp_sum(n);
        };
        // Few keys: steps down from the largest one, of an octave of scores at first, then twice as long each time, until nsel keys are
        // reached, and bisects the last step.  Many: bisects from the smallest key up.  count(below) >= nsel > count(above) throughout.
        uint32_t top = 0;
#pragma unroll
        for (int i = 0; i < NW; ++i) top = max(top, max(hi[i], lo[i]));
        uint32_t below = 0, above = (__reduce_max_sync(0xffffffffu, top) >> 16) + 1u, reach = first_step;
        int n_above = 0;     // keys that reach `above`
        bool exact = false;  // exactly nsel keys reach the threshold
        if (2 * nsel >= n_keys) {
            uint32_t low = 0xffffffffu;  // key 0 is no key
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                low = min(low, hi[i] >= 0x10000u ? hi[i] : 0xffffffffu);
                low = min(low, lo[i] != 0u ? lo[i] : 0xffffffffu);
            }
            below = __reduce_min_sync(0xffffffffu, low) >> 16;
            exact = nsel >= n_keys && count(below) == nsel;  // all of them
        }
#pragma unroll 1
        while (!exact && above - below > 1u) {
            uint32_t cand = (below + above) >> 1;
            if (below == 0u) {
                cand = above > reach ? above - reach : 1u;
                if (n_above > 0) reach *= 2u;
            }
            const int n = count(cand);
            if (n >= nsel) {
                below = cand;
                exact = n == nsel;
            } else {
                above = cand;
                n_above = n;
            }
        }
        // otherwise the threshold is the nsel-th largest key and more than nsel keys reach it
        const uint32_t thr = below;
        const int take_eq = exact ? 0 : nsel - n_above;  // ties to keep, lowest block index first
        const uint32_t tt = thr << 16;
        const unsigned lt_mask = (1u << lane) - 1u;
        int n_out = 0, n_eq = 0;
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            if (64 * i >= nk_pad) break;
            bool t0 = lo[i] >= tt, t1 = hi[i] >= tt;
            if (!exact) {
                const bool e0 = lo[i] == tt, e1 = (hi[i] & 0xffff0000u) == tt;
                const unsigned m0 = __ballot_sync(0xffffffffu, e0), m1 = __ballot_sync(0xffffffffu, e1);
                const int before = n_eq + __popc(m0 & lt_mask) + __popc(m1 & lt_mask);
                if (e0) t0 = before < take_eq;
                if (e1) t1 = before + (int)e0 < take_eq;
                n_eq += __popc(m0) + __popc(m1);
            }
            const unsigned s0 = __ballot_sync(0xffffffffu, t0), s1 = __ballot_sync(0xffffffffu, t1);
            const int at = n_out + __popc(s0 & lt_mask) + __popc(s1 & lt_mask);
            if (t0) out[at] = 2 * (lane + 32 * i);
            if (t1) out[at + (int)t0] = 2 * (lane + 32 * i) + 1;
            n_out += __popc(s0) + __popc(s1);
        }
    }
    for (int j = nsel + lane; j < cap; j += 32) out[j] = -1;
}

// The same for a row of any length and either key type, counted where it lies: `row` may be shared or global memory.
template <typename Key>
__device__ __forceinline__ void select_row(const Key* row, int Nk, int nk_pad, int nsel, int cap, int32_t* out, int32_t* cnt_out,
                                           int lane) {
    constexpr int kKeyBits = sizeof(Key) * 8;
    if (lane == 0) *cnt_out = nsel;
    if (nsel > 0) {
        uint32_t thr = 0;
        for (int bit = kKeyBits - 1; bit >= 0; --bit) {
            const uint32_t cand = thr | (1u << bit);
            if (count_row(row, nk_pad, cand, false, lane) >= nsel) thr = cand;
        }
        const int above = count_row(row, nk_pad, thr, true, lane);
        const int take_eq = nsel - above;  // ties at the threshold to keep, lowest block index first
        int n_out = 0, n_eq = 0;
        const unsigned lt_mask = (1u << lane) - 1u;
        for (int j0 = 0; j0 < Nk; j0 += 32) {
            const int j = j0 + lane;
            const bool ok = j < Nk;
            const uint32_t key = ok ? (uint32_t)row[j] : 0u;
            const bool gt = key > thr;
            const bool eq = (key == thr) && ok;
            const unsigned eq_mask = __ballot_sync(0xffffffffu, eq);
            const bool take = gt || (eq && (n_eq + __popc(eq_mask & lt_mask) < take_eq));
            const unsigned take_mask = __ballot_sync(0xffffffffu, take);
            if (take) out[n_out + __popc(take_mask & lt_mask)] = j;
            n_out += __popc(take_mask);
            n_eq += __popc(eq_mask);
        }
    }
    for (int j = nsel + lane; j < cap; j += 32) out[j] = -1;
}

}  // namespace sel
}  // namespace lcbsa
