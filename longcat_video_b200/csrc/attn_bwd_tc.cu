// Block-sparse attention backward on TMA + tcgen05 + TMEM for head_dim 128: the dQ pass and the dK/dV pass, after the delta
// kernel and the transposition of the block lists of attn_bwd.cu (which keeps head_dim 64, and ragged grids in fp16 or with
// blocks above 64 tokens, on warp-level MMAs).  A CTA owns a block of 64 or 128 tokens (kM rows: M=64 or M=128 MMAs) and
// streams 64-token tiles; attn_bwd.cu writes the lists in those terms (larger blocks are taken as 64-token units).
// Stands in for the Triton kernels _attn_bwd_dq_bsa_varlen_align and _attn_bwd_dkdv_bsa_varlen_align
// (longcat_video/block_sparse_attention/flash_attn_bsa_varlen_mask.py:289-945).
//
// Both passes are one kernel with the roles of the operands exchanged.  A CTA owns one tile pair (A1, A2) of kM rows and
// walks a list of 64-row tile pairs (B1, B2); per list entry
//
//   dQ pass   (CTA = query block i, list = its key blocks j):  A1 = Q_i  A2 = dO_i  B1 = K_j  B2 = V_j
//       S  = A1 B1^T        dP  = A2 B2^T        dS  = P o (dP - delta_i) * scale        dQ_i += dS B1
//   dK/dV pass (CTA = key block j, list = the query blocks i that selected it):  A1 = K_j  A2 = V_j  B1 = Q_i  B2 = dO_i
//       S^T = A1 B1^T       dP^T = A2 B2^T       P^T, dS^T as above, transposed          dV_j += P^T B2   dK_j += dS^T B1
//
// with P = exp2(S * scale * log2(e) - lse * log2(e)).  S and dP are (M = kM) N64 K128 MMAs, own tile from TMEM,
// streamed tile from shared memory, fp32 result in TMEM (kM = 128, dK/dV pass: V too comes from shared memory); P and dS are written back to TMEM in the input dtype and are the A operands of the N128 K64 MMAs
// that accumulate the gradients in TMEM over the whole list, with the streamed tile as MN-major B operand: a tile is
// loaded once (two 5-D TMA boxes of 64 columns, 128-byte swizzle) and serves as K-major operand of the first
// contraction and as MN-major operand of the last.  Nothing is recomputed within a pass, nothing goes through shared
// memory between the contractions, and no gradient is accumulated with atomics.
//
// Ragged grids (64-token blocks, bf16): the boxes of partial blocks are zero-filled by TMA outside the grid; a key outside
// the grid then has K = V = 0 and a query row outside has Q = dO = 0, so every term they enter is a number times zero and
// needs no mask as long as that number is finite.  A streamed query row outside the grid has P = 1 and dS = 0.  A streamed key
// outside the grid (dQ pass) has S = dP = 0, hence P = 2^(-lse * log2 e), which overflows for rows whose scores are all far
// below zero: where the key grid has partial blocks the exponent is capped (kCap).  A dS of fp16 overflows long before
// that, so fp16 keeps ragged grids on the warp-level kernels, which mask such keys.  Rows outside the grid are not stored.
//
//   warps 0-7 : arithmetic.  kM = 128: a thread serves one TMEM lane = one row of the 128 x 64 tile.  kM = 64: the tile occupies lanes
//               0-15 of every 32-lane quadrant, and a warp takes its 16 rows with all threads, two rows and 32 values each
//   warps 8, 11 : TMA producers of B1 and of B2 into a ring of five (four for kM = 128) slots; warp 8 also brings the CTA's
//               own tiles once, and in the dK/dV pass the query block's 64 (lse * log2 e) and 64 delta values per slot, by a
//               bulk copy onto the same barrier (bwd_stats_kernel lays them out, negated, per block)
//   warp 9    : issues S and dP    warp 10 : issues the gradient MMAs; one elected lane each
//
// TMEM and the order of the MMAs (see Cols).  P and dS (16-bit pairs) have columns of their own; those of entry s are overwritten
// once the gradient MMAs of s have read them (ts_done).
//   kM = 64, both passes: two buffers of everything; warps 0-3 take the even entries, warps 4-7 the odd ones.
//   kM = 128, dQ pass: two buffers of S and of dS, one of dP; the same split of the entries.
//   kM = 128, dK/dV pass (two accumulators): ONE buffer each of S^T, dP^T, P^T and dS^T; all eight warps work on every entry
//       (warps 0-3 columns 0-31, warps 4-7 columns 32-63).
//   S and dP of the entry that takes a buffer next wait until the arithmetic warps hold the last ones in registers (s_free), and the
//   gradient MMAs of s for x_full(s), its P and dS.
// The own tiles are moved to TMEM once, where they are the A operands of every S and dP (kM = 128, dK/dV pass: only K, TMEM is
// full): an M=64 S with both operands in shared memory reads 128 bytes a cycle of it, all that it gives, beside the incoming
// tiles.  At kM = 64 the second of two things sits in the lanes 16-31 that an M=64 tile leaves free (see Cols).
// What bounds it: the tensor pipe, 512 + 256 cycles per entry in the dQ pass and 512 + 512 in the dK/dV pass whether M is 64 or
// 128.  Measured per entry (in-kernel time stamps; 64-token blocks of the 480p grid, 128-token blocks of 24x32x56), before with
// one issuer and one producer and both operands in shared memory, and now: dQ 1071 -> 948 and 1200 -> 958 cycles, dK/dV
// 1336 -> 1165.
// Persistent, one CTA per SM: a CTA per block spent some 10000 cycles before its first and behind its last entry, on barriers, TMEM,
// its list, its first tiles and its gradients; now the own tiles, the list and the row values of the next block are fetched
// under the entries of this one, and some 3500 are left.  The blocks are taken off a counter, since the transposed lists differ in
// length.  Backward of 8 heads, 39 of 624 64-token blocks: 1889 -> 1704 us; 16 of 832: 570 -> 445 us.  With 128-token blocks, 42
// of 336, the step took 2497 -> 2590 us (2653 us before the issuer's look-ahead, 2470 to 2540 us now); short calls of a few blocks
// are some 3 us slower for it.
// Counters over whole launches (8 heads, 480p grids): tensor pipe 82 % (dQ) and 88 % (dK/dV) with 64-token blocks, 957 and 1190 cycles
// per entry; 70 % and 73 % with 128-token blocks, 1126 and 1431 cycles.
// Every mbarrier wait is bounded; when one runs out the CTA flags the status word, drains its copies, frees TMEM, returns.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "tc_common.cuh"

namespace lcbsa {

namespace {

using namespace tc;

constexpr int kD = 128;
constexpr int kBlk = 64;
constexpr int kTileBytes = kBlk * kD * 2;   // 16 KiB
constexpr int kHalfBytes = kTileBytes / 2;  // one 64-column half: 64 rows x 128 B, 128B-swizzled
constexpr int kSlotBytes = 2 * kTileBytes;  // a ring slot: the (B1, B2) tiles of one list entry
constexpr int kStatsFloats = 2 * kBlk;      // per 64-token query block: lse * log2(e) [64], delta [64]
constexpr int kStatsBytes = kStatsFloats * 4;
constexpr int kThreads = 384;
constexpr int kRegsMath = 200, kRegsOther = 104;  // setmaxnreg: (200 + 200 + 104) * 128 = the 63 K registers of the launch

constexpr int kItemRing = 4;  // items announced ahead

// Shared memory, for own tiles of kM = 64 or 128 rows (the streamed tiles always have 64).
template <int kM> struct Lay {
    static constexpr int aTile = kM * kD * 2;        // 16 or 32 KiB: A1, A2
    static constexpr int aHalf = aTile / 2;          // one 64-column half: kM rows x 128 B, 128B-swizzled
    static constexpr int slots = kM == 64 ? 5 : 4;   // ring of (B1, B2) tile pairs
    static constexpr int offA = 0;
    static constexpr int offB = offA + 2 * aTile;
    static constexpr int offStats = offB + slots * kSlotBytes;  // per slot: -lse2[64], -delta[64] of the streamed query block
    static constexpr int offBar = offStats + slots * kStatsBytes;
    // barriers: full[slots], empty[slots], s_full[2], s_free[2], x_full[2], ts_done[2], a_full, a_empty, at_full, at_free, acc_done,
    //           acc_free, item_full[kItemRing], item_empty[kItemRing]
    static constexpr int numBars = 2 * slots + 8 + 6 + 2 * kItemRing;
    static constexpr int offMisc = (offBar + numBars * 8 + 15) / 16 * 16;  // abort flag, TMEM base
    static constexpr int offItems = offMisc + 64;                          // [kItemRing] (item, entries, first entry of its list, -)
    static constexpr int smem = offItems + kItemRing * 16;
};

// Where things are in TMEM: column plus (lane offset << 16).  own1, own2: the CTA's own tiles as 16-bit pairs (64 columns);
// s, dp: fp32, 64 columns; xp, xd: P and dS as 16-bit pairs, 32 columns; acc1, acc2: fp32, 128 columns.  sbufs: buffers of S, xbufs: of P
// and dS; split: both warpgroups work on every entry (half the columns each) instead of on every other one.
//
// An M=64 tile takes lanes 0-15 of every 32-lane quadrant, so at kM = 64 two things share their columns: S and dP, P and dS, dV and
// dK, A1 and A2, the second of each 16 lanes up (the A operand and the result of an MMA are always in the same lanes).
constexpr uint32_t kUp = 16u << 16;
template <int kMode, int kM> struct Cols;
template <int kMode> struct Cols<kMode, 64> {
    static constexpr uint32_t acc2 = 0, acc1 = kMode == 0 ? 0 : kUp;
    static constexpr uint32_t own1 = 320, own2 = 320 + kUp;
    static constexpr int sbufs = 2, xbufs = 2;
    static constexpr bool split = false;
    __device__ static __forceinline__ uint32_t s(int buf) { return 128u + 64u * buf; }
    __device__ static __forceinline__ uint32_t dp(int buf) { return 128u + 64u * buf + kUp; }
    __device__ static __forceinline__ uint32_t xp(int buf) { return 256u + 32u * buf; }
    __device__ static __forceinline__ uint32_t xd(int buf) { return 256u + 32u * buf + (kMode == 0 ? 0u : kUp); }
};
// kM = 128, dQ pass: dQ 0, S 128 and 192, dP 256 (one buffer), dS 320 and 352, Q 384, dO 448
template <> struct Cols<0, 128> {
    static constexpr uint32_t acc1 = 0, acc2 = 0, own1 = 384, own2 = 448;
    static constexpr int sbufs = 2, xbufs = 2;
    static constexpr bool split = false;
    __device__ static __forceinline__ uint32_t s(int buf) { return 128u + 64u * buf; }
    __device__ static __forceinline__ uint32_t dp(int) { return 256u; }
    __device__ static __forceinline__ uint32_t xp(int) { return 0u; }  // unused in this pass
    __device__ static __forceinline__ uint32_t xd(int buf) { return 320u + 32u * buf; }
};
// kM = 128, dK/dV pass: dK 0, dV 128, S^T 256, dP^T 320, P^T 384, dS^T 416 (one buffer each), K 448; V stays in shared memory
template <> struct Cols<1, 128> {
    static constexpr uint32_t acc1 = 0, acc2 = 128, own1 = 448, own2 = 0;
    static constexpr int sbufs = 1, xbufs = 1;
    static constexpr bool split = true;
    __device__ static __forceinline__ uint32_t s(int) { return 256u; }
    __device__ static __forceinline__ uint32_t dp(int) { return 320u; }
    __device__ static __forceinline__ uint32_t xp(int) { return 384u; }
    __device__ static __forceinline__ uint32_t xd(int) { return 416u; }
};

struct BwdTcParams {
    CUtensorMap tm_a1, tm_a2, tm_b1, tm_b2;
    const int32_t* list;   // dQ pass: [BH][n_own][cap] key units per own block; dK/dV pass: [BH][list_stride] query units, by toff
    const int32_t* cnt;    // dQ pass: [BH][n_own]
    const int32_t* toff;   // dK/dV pass: [BH][n_own + 1]
    long long list_stride;
    const float* stats;    // dK/dV pass: [BH][n_stream][2][64] of the streamed 64-token query blocks: -lse * log2(e), -delta
    const float* lse;      // dQ pass: [BH][Sq] natural log, of the own rows
    const float* delta;    // dQ pass: [BH][Sq]
    long long Sq;
    unsigned int* status;
    void* out1;            // dQ pass: dq; dK/dV pass: dk
    void* out2;            // dK/dV pass: dv
    long long o1_sb, o1_sh, o1_ss, o2_sb, o2_sh, o2_ss;  // element strides
    int cap, n_own, n_stream, heads;
    int n_items;           // own blocks of all heads: item = bh * n_own + own block
    int* next_item;        // counter of the items taken behind the first of each CTA, zero at the start
    int merge_a1, merge_a2, merge_b1, merge_b2;  // how the batch axis is folded into each map
    Geom ga, gb;           // grid of the CTA's own tiles (blocks of 64 or 128 tokens), grid of the streamed 64-token tiles
    float scale, scale2;   // sm_scale, sm_scale * log2(e)
};

// Cap of the exponents on ragged key grids.  A present key has S * scale <= lse, so its exponent is at most rounding above 0 (2^-22
// of |lse|: the cap is out of its reach below |lse| = 2^27); a key outside the grid gets P <= 2^64, whose dS = -P * delta * scale is
// finite in fp32 and bf16.  A NaN stays a NaN.
constexpr float kMaxExponent = 64.f;
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// called by a whole converged warp with warp-uniform operands, like the _elect copies of tc_common.cuh
__device__ __forceinline__ void bulk_load_elect(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}

// -lse * log2(e) and -delta of every query row, laid out per 64-token block in slot order, so that a block's 128 values are
// one contiguous 512-byte piece.  Slots of a partial block that lie outside the grid get zeros (their q and dO rows are
// zero-filled by TMA, so that P is 1 and dS 0, and every term they enter is zero).
__global__ void __launch_bounds__(256) bwd_stats_kernel(const float* lse, const float* delta, Geom g, long long Sq, long long total,
                                                        float* stats, int* next_item) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < 2) next_item[p] = 0;  // the item counters of the two passes that follow
    if (p >= total) return;
    const int r = (int)(p % kBlk);
    const long long rest = p / kBlk;
    const int blk = (int)(rest % g.nblk);
    const long long bh = rest / g.nblk;
    int lt, lh, lw, bt, bhh, bw;
    slot_coords(g, r, lt, lh, lw);
    block_coords(g, blk, bt, bhh, bw);
    const int tt = bt * g.ct + lt, hh = bhh * g.ch + lh, ww = bw * g.cw + lw;
    const bool inside = tt < g.T && hh < g.H && ww < g.W;
    const long long tok = ((long long)tt * g.H + hh) * g.W + ww;
    float* dst = stats + (bh * g.nblk + blk) * kStatsFloats;
    dst[r] = inside ? -(lse[bh * Sq + tok] * 1.4426950408889634f) : 0.f;
    dst[kBlk + r] = inside ? -delta[bh * Sq + tok] : 0.f;
}

// 64 columns of this thread's accumulator row -> 128 bytes of the row in global memory (input dtype)
template <bool kBf16>
__device__ __forceinline__ void store_row64(unsigned char* row_ptr, int col0, const uint32_t (&r)[64]) {
#pragma unroll
    for (int q8 = 0; q8 < 8; ++q8) {
        uint4 pk;
        pk.x = pack2(kBf16, __uint_as_float(r[q8 * 8 + 0]), __uint_as_float(r[q8 * 8 + 1]));
        pk.y = pack2(kBf16, __uint_as_float(r[q8 * 8 + 2]), __uint_as_float(r[q8 * 8 + 3]));
        pk.z = pack2(kBf16, __uint_as_float(r[q8 * 8 + 4]), __uint_as_float(r[q8 * 8 + 5]));
        pk.w = pack2(kBf16, __uint_as_float(r[q8 * 8 + 6]), __uint_as_float(r[q8 * 8 + 7]));
        *reinterpret_cast<uint4*>(row_ptr + (col0 + q8 * 8) * 2) = pk;
    }
}

// kMode 0: dQ pass, 1: dK/dV pass.  kCap: dQ pass over a key grid with partial blocks.  Persistent, one CTA per SM.
template <bool kBf16, int kMode, int kM, bool kCap>
__global__ void __launch_bounds__(kThreads, 1) bwd_tc_kernel(const __grid_constant__ BwdTcParams P) {
    using C = Cols<kMode, kM>;
    using Ly = Lay<kM>;
    constexpr int kSlots = Ly::slots, kOffA = Ly::offA, kOffB = Ly::offB, kOffStats = Ly::offStats, kOffBar = Ly::offBar, kOffMisc = Ly::offMisc;
    constexpr int kATile = Ly::aTile, kAHalf = Ly::aHalf;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = sbase + kOffBar;
    // Entries are numbered over the whole kernel: entry s uses ring slot s % kSlots, S and dP of buffer s % kSBufs, P and dS of
    // buffer s % kXBufs.  Items with a list that is not empty are numbered too, for the barriers that turn once an item.
    constexpr int kB = 2 * kSlots, kSBufs = C::sbufs, kXBufs = C::xbufs;
    auto bar_full = [&](int s) { return bar0 + 8u * s; };
    auto bar_empty = [&](int s) { return bar0 + 8u * (kSlots + s); };
    constexpr bool kSplit = C::split;
    constexpr bool kOneDp = kM == 128 && kMode == 0;  // two buffers of S, one of dP
    constexpr bool kOwn2Smem = kM == 128 && kMode == 1;  // A2 is read from shared memory
    auto bar_s_full = [&](int sbuf) { return bar0 + 8u * (kB + sbuf); };
    auto bar_s_free = [&](int sbuf) { return bar0 + 8u * (kB + 2 + sbuf); };
    auto bar_x_full = [&](int buf) { return bar0 + 8u * (kB + 4 + buf); };
    auto bar_ts_done = [&](int buf) { return bar0 + 8u * (kB + 6 + buf); };
    const uint32_t bar_a_full = bar0 + 8u * (kB + 8), bar_a_empty = bar0 + 8u * (kB + 9), bar_at_full = bar0 + 8u * (kB + 10);
    const uint32_t bar_at_free = bar0 + 8u * (kB + 11), bar_acc_done = bar0 + 8u * (kB + 12), bar_acc_free = bar0 + 8u * (kB + 13);
    auto bar_item_full = [&](int k) { return bar0 + 8u * (kB + 14 + k); };
    auto bar_item_empty = [&](int k) { return bar0 + 8u * (kB + 14 + kItemRing + k); };
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kOffMisc);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffMisc + 8);
    int4* items = reinterpret_cast<int4*>(smem + Ly::offItems);
    const Ctl ctl{abort_flag, P.status};

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // provably warp-uniform
    if (tid == 0) {
        ctl_init(ctl);
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(bar_full(s), 2);  // one arrival per producer
            mbar_init(bar_empty(s), 1);
        }
        for (int buf = 0; buf < 2; ++buf) {
            mbar_init(bar_s_full(buf), 1);
            mbar_init(bar_s_free(buf), kSplit ? 8 : 4);  // one elected arrival per warp that works on an entry
            mbar_init(bar_x_full(buf), kSplit ? 8 : 4);
            mbar_init(bar_ts_done(buf), 1);
        }
        mbar_init(bar_a_full, 1);
        mbar_init(bar_a_empty, kOwn2Smem ? 9 : 8);  // the arithmetic warps have moved it; kOwn2Smem: and the last dP has read A2
        mbar_init(bar_at_full, 8);
        mbar_init(bar_at_free, 1);
        mbar_init(bar_acc_done, 1);
        mbar_init(bar_acc_free, 8);
        for (int k = 0; k < kItemRing; ++k) {
            mbar_init(bar_item_full(k), 1);
            mbar_init(bar_item_empty(k), 11);  // every warp but the one that announces
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the tiles are 128B-swizzled, which ties their layout to address bits 7-9: refuse to run on an unaligned base
        if (sbase & 1023u) {
            *abort_flag = 1;
            if (atomicCAS(P.status, 0u, 1u) == 0u) {
                P.status[1] = blockIdx.x;
                P.status[2] = sbase;
                P.status[3] = 0;
            }
        }
    }
    if (warp == 9) {  // TMEM: all 512 columns, allocated and freed by the issuing warp
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const bool start_ok = *abort_flag == 0;  // else nothing runs, nothing is written

    // The items of a CTA are announced by warp 8, which takes them off a counter: lists differ in length, in the dK/dV pass by a lot.
    struct Item {
        int id, n, lo;  // n entries, from position lo of the list array of its head (dK/dV pass)
    };
    // Item number k of this CTA, for every warp but warp 8.  id < 0: there is none, or the kernel is giving up.
    auto take_item = [&](unsigned k) {
        Item it{-1, 0, 0};
        if (!mbar_wait_warp(bar_item_full(k % kItemRing), (k / kItemRing) & 1, ctl, 200, k)) return it;
        const int4 v = items[k % kItemRing];
        __syncwarp();
        mbar_arrive_elect(bar_item_empty(k % kItemRing));
        it.id = v.x;
        it.n = v.y;
        it.lo = v.z;
        return it;
    };
    auto list_of = [&](const Item& it) {
        return kMode == 0 ? P.list + (long long)it.id * P.cap : P.list + (long long)(it.id / P.n_own) * P.list_stride + it.lo;
    };

    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
        if (!start_ok) {
        } else if (warp == 8 || warp == 11) {
            // ================================================================== TMA producers: warp 8 B1, the own tiles and the stats, warp 11 B2
            const bool is_b1 = warp == 8;
            const CUtensorMap* tm = is_b1 ? &P.tm_b1 : &P.tm_b2;
            const int mrg = is_b1 ? P.merge_b1 : P.merge_b2;
            bool ok = true;
            unsigned s = 0, kk = 0;  // entries, items with entries
            // Warp 8 works two items ahead on the announcements: `ahead2` is the number taken off the counter for the item behind the
            // next, `ahead` the next item, whose list length is on its way.  The first item of a CTA is its own number: a call with
            // an item per CTA would wait for two trips to the counter before its first copy (8 heads of 4x8x16 tokens, 128-token blocks,
            // backward 31.2 -> 30.4 us; with a CTA per block, as it was once, 27.3 us: no announcements and no move to TMEM).
            int ahead2 = 0;
            Item ahead{-1, 0, 0};
            auto take = [&]() { return lane == 0 ? (int)gridDim.x + atomicAdd(P.next_item, 1) : 0; };
            auto look = [&](int id) {
                Item it{id < P.n_items ? id : -1, 0, 0};
                if (it.id >= 0) {
                    if (kMode == 0) {
                        it.n = min(max(P.cnt[it.id], 0), P.cap);
                    } else {
                        const int32_t* to = P.toff + (long long)(it.id / P.n_own) * (P.n_own + 1) + it.id % P.n_own;
                        it.lo = to[0];
                        it.n = max(to[1] - it.lo, 0);
                    }
                }
                return it;
            };
            if (is_b1) {
                ahead = look(blockIdx.x);
                ahead2 = take();
            }
            auto step = [&]() {
                ahead = look(__shfl_sync(0xffffffffu, ahead2, 0));
                ahead2 = take();
            };
            for (unsigned k = 0;; ++k) {
                Item it;
                if (is_b1) {
                    it = ahead;
                    ok = mbar_wait_warp(bar_item_empty(k % kItemRing), ((k / kItemRing) & 1) ^ 1, ctl, 201, k);
                    if (!ok) break;
                    if (lane == 0) items[k % kItemRing] = make_int4(it.id, it.n, it.lo, 0);
                    __syncwarp();
                    mbar_arrive_elect(bar_item_full(k % kItemRing));
                } else {
                    it = take_item(k);
                }
                if (it.id < 0) break;
                const int n = it.n;
                if (n == 0) {
                    if (is_b1) step();
                    continue;
                }
                const int bh = it.id / P.n_own, own = it.id % P.n_own, b = bh / P.heads, h = bh % P.heads;
                const int c3 = mrg ? b * P.gb.T : 0, c4 = mrg ? h : b * P.heads + h;
                const int32_t* list = list_of(it);
                // The list is fetched and decoded by the whole warp, 32 entries at a time and one window ahead: lane L holds entry
                // 32 w + L as the block's first token packed t << 20 | h << 10 | w.
                auto fetch = [&](int e) { return e < n ? list[e] : 0; };
                auto decode = [&](int blk) {
                    // an entry outside the grid never becomes an address: the box is placed at w = W, wholly outside the map, and
                    // TMA fills the tiles with zeros (the list transposition has flagged the call)
                    if ((unsigned)blk >= (unsigned)P.gb.nblk) return P.gb.W;
                    int bt, bhh, bw;
                    block_coords(P.gb, blk, bt, bhh, bw);
                    return ((bt * P.gb.ct) << 20) | ((bhh * P.gb.ch) << 10) | (bw * P.gb.cw);
                };
                int blk = fetch(lane), blk_n = fetch(32 + lane);
                if (is_b1) {
                    // one box of kM rows per 64-column half (the own grid's block is the box)
                    ok = mbar_wait_warp(bar_a_empty, (kk & 1) ^ 1, ctl, 202, kk);
                    if (!ok) break;
                    mbar_arrive_tx_elect(bar_a_full, 2 * kATile);
                    const Coord a1 = block_coord(P.ga, own, b, h, P.heads, P.merge_a1, P.ga.T), a2 = block_coord(P.ga, own, b, h, P.heads, P.merge_a2, P.ga.T);
                    tma_load_5d_elect(sbase + kOffA, &P.tm_a1, bar_a_full, 0, a1.c1, a1.c2, a1.c3, a1.c4);
                    tma_load_5d_elect(sbase + kOffA + kAHalf, &P.tm_a1, bar_a_full, 64, a1.c1, a1.c2, a1.c3, a1.c4);
                    tma_load_5d_elect(sbase + kOffA + kATile, &P.tm_a2, bar_a_full, 0, a2.c1, a2.c2, a2.c3, a2.c4);
                    tma_load_5d_elect(sbase + kOffA + kATile + kAHalf, &P.tm_a2, bar_a_full, 64, a2.c1, a2.c2, a2.c3, a2.c4);
                }
                ++kk;
                int pos = decode(blk);
                for (int e = 0; e < n; ++e) {
                    const int slot = s % kSlots;
                    ok = mbar_wait_warp(bar_empty(slot), ((s / kSlots) & 1) ^ 1, ctl, 210 + kMode, s);
                    if (!ok) break;
                    ++s;
                    const int pk = __shfl_sync(0xffffffffu, pos, e & 31);
                    const bool stats = kMode == 1 && is_b1;
                    mbar_arrive_tx_elect(bar_full(slot), kTileBytes + (stats ? kStatsBytes : 0));
                    const uint32_t dst = sbase + kOffB + slot * kSlotBytes + (is_b1 ? 0 : kTileBytes);
                    tma_load_5d_elect(dst, tm, bar_full(slot), 0, pk & 1023, (pk >> 10) & 1023, (pk >> 20) + c3, c4);
                    tma_load_5d_elect(dst + kHalfBytes, tm, bar_full(slot), 64, pk & 1023, (pk >> 10) & 1023, (pk >> 20) + c3, c4);
                    if (stats) {  // transposed lists only hold blocks of the grid
                        const int bk = __shfl_sync(0xffffffffu, blk, e & 31);
                        bulk_load_elect(sbase + kOffStats + slot * kStatsBytes, P.stats + ((long long)bh * P.n_stream + bk) * kStatsFloats, kStatsBytes,
                                        bar_full(slot));
                    }
                    // Behind the item's last copies, none of which waits for the counter; the ring holds some 5000 cycles of work
                    // then, so the next item's length and list arrive under it.  Asked earlier, a CTA commits itself to an item
                    // it will not come to for long: 3 heads of 8x32x32 tokens, 32 of 128 blocks, 171 us instead of 155 us.
                    if (is_b1 && e == n - 1) step();
                    if ((e & 31) == 31) {
                        blk = blk_n;
                        pos = decode(blk);
                        blk_n = fetch(e + 33 + lane);
                    }
                }
                if (!ok) break;
            }
            if ((!ok || *abort_flag != 0) && lane == 0) {
                // drain: give the copies this warp issued a bounded time to land before the CTA exits
                const long long t0 = clock64();
                while (is_b1 && kk > 0 && !mbar_try(bar_a_full, (kk - 1) & 1) && clock64() - t0 < 40000000ll) {
                }
                for (unsigned r = s > kSlots ? s - kSlots : 0; r < s; ++r)
                    while (!mbar_try(bar_full(r % kSlots), (r / kSlots) & 1) && clock64() - t0 < 40000000ll) {
                    }
            }
        } else if (warp == 9) {
            // ================================================================== issuer of S and dP (S^T and dP^T)
            const uint32_t idesc_ss = instr_desc(kBf16, kM, 64, 0);
            const uint64_t a2d = smem_desc(sbase + kOffA + kATile, 16, 1024);  // kOwn2Smem
            bool ok = true;
            unsigned s = 0, kk = 0;
            for (unsigned k = 0; ok; ++k) {
                const Item it = take_item(k);
                if (it.id < 0) break;
                if (it.n == 0) continue;
                ok = mbar_wait_warp(bar_at_full, kk & 1, ctl, 220 + kMode, kk);  // the own tiles are in TMEM
                ++kk;
                bool pre = false;
                for (int e = 0; e < it.n && ok; ++e, ++s) {
                    const int slot = s % kSlots, sbuf = s % kSBufs;
                    if (!pre) {  // not already seen ready by the look-ahead of the entry before
                        ok = mbar_wait_warp(bar_full(slot), (s / kSlots) & 1, ctl, 222 + kMode, s);
                        // the arithmetic warps hold the buffer's last S and dP in registers (kOneDp: seen before the dP of entry s - 1)
                        if (ok && !kOneDp) ok = mbar_wait_warp(bar_s_free(sbuf), ((s / kSBufs) & 1) ^ 1, ctl, 226, s);
                        if (!ok) break;
                    }
                    tc_fence_after();
                    const uint32_t tile = sbase + kOffB + slot * kSlotBytes;
                    const uint64_t b1d = smem_desc(tile, 16, 1024), b2d = smem_desc(tile + kTileBytes, 16, 1024);
#pragma unroll
                    for (int j = 0; j < kD / 16; ++j) {
                        // 32 bytes per 16-column step inside a 64-column half, the halves 8 KiB apart; 8 TMEM columns per step
                        const uint64_t off = (uint64_t)(((j >> 2) * kHalfBytes + (j & 3) * 32) >> 4);
                        tc_mma_ts(tmem + C::s(sbuf), tmem + C::own1 + 8u * j, b1d + off, idesc_ss, j > 0);
                    }
                    // Look ahead: probe the next entry's barriers between the two contractions and read the answer after them.  Before the
                    // first one the arithmetic warps do not have the S and dP of the entry before yet.  (8 heads, 39 of 624 blocks: 1705 us
                    // with the probe in front, 1662 us.)
                    bool nf = false, ns = kOneDp;
                    if (e + 1 < it.n) {
                        nf = mbar_test(bar_full((s + 1) % kSlots), ((s + 1) / kSlots) & 1);
                        if (!kOneDp) ns = mbar_test(bar_s_free((s + 1) % kSBufs), (((s + 1) / kSBufs) & 1) ^ 1);
                    }
                    tc_fence_after();
                    if (kOneDp && s > 0) {  // dP of the entry before is in registers
                        ok = mbar_wait_warp(bar_s_free((s - 1) & 1), ((s - 1) >> 1) & 1, ctl, 227, s);
                        if (!ok) break;
                        tc_fence_after();
                    }
#pragma unroll
                    for (int j = 0; j < kD / 16; ++j) {
                        const uint64_t off = (uint64_t)(((j >> 2) * kHalfBytes + (j & 3) * 32) >> 4);
                        const uint64_t aoff = (uint64_t)(((j >> 2) * kAHalf + (j & 3) * 32) >> 4);  // the halves of an own tile are kM x 128 B apart
                        if (kOwn2Smem) tc_mma(tmem + C::dp(sbuf), a2d + aoff, b2d + off, idesc_ss, j > 0);
                        else tc_mma_ts(tmem + C::dp(sbuf), tmem + C::own2 + 8u * j, b2d + off, idesc_ss, j > 0);
                    }
                    tc_commit(bar_s_full(sbuf));
                    if (e == it.n - 1) {  // the own tiles have been read
                        tc_commit(bar_at_free);
                        if (kOwn2Smem) tc_commit(bar_a_empty);
                    }
                    __syncwarp();
                    pre = __all_sync(0xffffffffu, nf && ns);
                }
            }
        } else if (warp == 10) {
            // ================================================================== issuer of the gradient MMAs: A from TMEM (8 columns
            // per 16-row step), B the streamed tile, MN-major (64-column halves 8 KiB apart = LBO, 8-row groups 1 KiB apart =
            // SBO, 16 rows = 2 KiB per step)
            const uint32_t idesc_ts = instr_desc(kBf16, kM, 128, 1);
            bool ok = true;
            unsigned s = 0, kk = 0;
            for (unsigned k = 0; ok; ++k) {
                const Item it = take_item(k);
                if (it.id < 0) break;
                if (it.n == 0) continue;
                ok = mbar_wait_warp(bar_acc_free, (kk & 1) ^ 1, ctl, 244, kk);  // the gradients of the item before have been read
                ++kk;
                bool pre = false;
                for (int e = 0; e < it.n && ok; ++e, ++s) {
                    const int slot = s % kSlots, buf = s % kXBufs;
                    if (!pre) {
                        ok = mbar_wait_warp(bar_full(slot), (s / kSlots) & 1, ctl, 228 + kMode, s);
                        if (ok) ok = mbar_wait_warp(bar_x_full(buf), (s / kXBufs) & 1, ctl, 224 + kMode, s);
                        if (!ok) break;
                    }
                    bool nf = false, nx = false;
                    if (e + 1 < it.n) {
                        nf = mbar_test(bar_full((s + 1) % kSlots), ((s + 1) / kSlots) & 1);
                        nx = mbar_test(bar_x_full((s + 1) % kXBufs), ((s + 1) / kXBufs) & 1);
                    }
                    tc_fence_after();
                    const uint32_t tile = sbase + kOffB + slot * kSlotBytes;
                    const uint64_t b1m = smem_desc(tile, kHalfBytes, 1024), b2m = smem_desc(tile + kTileBytes, kHalfBytes, 1024);
                    if (kMode == 1) {
#pragma unroll
                        for (int j = 0; j < kBlk / 16; ++j)  // dV += P^T dO
                            tc_mma_ts(tmem + C::acc2, tmem + C::xp(buf) + 8u * j, b2m + (uint64_t)((j * 2048) >> 4), idesc_ts, (e > 0 || j > 0) ? 1u : 0u);
                    }
#pragma unroll
                    for (int j = 0; j < kBlk / 16; ++j)  // dQ += dS K, or dK += dS^T Q
                        tc_mma_ts(tmem + C::acc1, tmem + C::xd(buf) + 8u * j, b1m + (uint64_t)((j * 2048) >> 4), idesc_ts, (e > 0 || j > 0) ? 1u : 0u);
                    tc_commit(bar_empty(slot));  // the streamed tiles are free once these MMAs have read them
                    tc_commit(bar_ts_done(buf)); // and so are P and dS
                    if (e == it.n - 1) tc_commit(bar_acc_done);
                    __syncwarp();
                    pre = __all_sync(0xffffffffu, nf && nx);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsMath));
        // ================================================================== arithmetic warps
        const int wg = warp >> 2;  // dQ pass: entries wg, wg + 2, ...; dK/dV pass: columns 32 wg .. 32 wg + 31 of every entry
        const int wq = warp & 3;   // TMEM quadrant of this warp
        // row of the own tile = TMEM lane.  An M=128 accumulator has row r in lane r; an M=64 one occupies lanes 0-15 of every
        // 32-lane quadrant, and what shares its columns the lanes 16-31
        const int row = kM == 128 ? wq * 32 + lane : wq * 16 + (lane & 15);
        const uint32_t t_lane = (uint32_t)(wq * 32) << 16;
        bool ok = start_ok;
        unsigned s0 = 0, kk = 0;  // entries before the current item, items with entries before it
        // The own tiles go from shared memory to TMEM, where they are the A operands of every S and dP: with both operands in shared
        // memory an M=64 S reads as many bytes of the own tile as of the streamed one.  A thread moves (half of) a row.
        auto own_to_tmem = [&](unsigned item) -> bool {
            if (!mbar_wait_warp(bar_a_full, item & 1, ctl, 242, item)) return false;
            if (item > 0 && !mbar_wait_warp(bar_at_free, (item - 1) & 1, ctl, 243, item)) return false;
            tc_fence_after();
            // kM = 64: warpgroup g moves half g of A1 (lanes 0-15) and of A2 (lanes 16-31); kM = 128: A1 and A2, or half g of A1
            const int tile = kM == 64 ? lane >> 4 : (kOwn2Smem ? 0 : wg);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if ((kM == 64 || kOwn2Smem) && half != wg) continue;
                const unsigned char* src = smem + kOffA + tile * kATile + half * kAHalf + row * 128;
                uint32_t ar[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(src + ((c ^ (row & 7)) << 4));
                    ar[4 * c + 0] = v.x;
                    ar[4 * c + 1] = v.y;
                    ar[4 * c + 2] = v.z;
                    ar[4 * c + 3] = v.w;
                }
                tc_st32(tmem + (kM == 128 && tile == 1 ? C::own2 : C::own1) + 32u * half + t_lane, ar);
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            mbar_arrive_elect(bar_at_full);
            mbar_arrive_elect(bar_a_empty);
            return true;
        };
        // Two columns of S and dP -> one 16-bit pair of P and one of dS, two columns per instruction where the machine has packed
        // fp32 forms.  nl, nd: -lse * log2(e) and -delta.
        const float2 sc2 = make_float2(P.scale2, P.scale2), sc = make_float2(P.scale, P.scale);
        auto pair = [&](uint32_t s0, uint32_t s1, uint32_t d0, uint32_t d1, float2 nl, float2 nd, uint32_t& xp, uint32_t& xd) {
            float2 x = __ffma2_rn(make_float2(__uint_as_float(s0), __uint_as_float(s1)), sc2, nl);
            if (kCap) x = make_float2(min_nan(x.x, kMaxExponent), min_nan(x.y, kMaxExponent));
            const float2 p = make_float2(ex2(x.x), ex2(x.y));
            const float2 t = __fadd2_rn(make_float2(__uint_as_float(d0), __uint_as_float(d1)), nd);
            const float2 g = __fmul2_rn(__fmul2_rn(p, t), sc);
            if (kMode == 1) xp = pack2(kBf16, p.x, p.y);
            xd = pack2(kBf16, g.x, g.y);
        };
        // The token of row r of an item (rows of a block are its tokens in t, h, w order), -1 outside the grid: such a row of a
        // partial block is computed on zero-filled operands and never stored.
        auto token = [&](const Item& it, int r) -> long long {
            int lt, lh, lw, bt, bhh, bw;
            slot_coords(P.ga, r, lt, lh, lw);
            block_coords(P.ga, it.id % P.n_own, bt, bhh, bw);
            const int tt = bt * P.ga.ct + lt, hh = bhh * P.ga.ch + lh, ww = bw * P.ga.cw + lw;
            return tt < P.ga.T && hh < P.ga.H && ww < P.ga.W ? ((long long)tt * P.ga.H + hh) * P.ga.W + ww : -1;
        };
        // dQ pass: -lse * log2(e) and -delta of this thread's query rows, one pair for the whole list; rows outside the grid: 0
        auto row_stats = [&](const Item& it, int r, float2& nl, float2& nd) {
            nl = nd = make_float2(0.f, 0.f);
            if (kMode != 0) return;
            const long long tok = token(it, r);
            if (tok < 0) return;
            const long long at = (long long)(it.id / P.n_own) * P.Sq + tok;
            const float l2 = -(P.lse[at] * 1.4426950408889634f), dl = -P.delta[at];
            nl = make_float2(l2, l2);
            nd = make_float2(dl, dl);
        };
        auto entries = [&](unsigned n, const float2 (&st)[4]) {
        if constexpr (kM == 64) {
            // A warp takes its quadrant's 16 rows with all lanes: rows lane / 4 and lane / 4 + 8, columns 8 k + 2 (lane % 4) + 0, 1.
            float2 nl0 = st[0], nd0 = st[1], nl1 = st[2], nd1 = st[3];
            for (unsigned i = s0 + ((s0 ^ wg) & 1); i < s0 + n && ok; i += 2) {  // buffer i & 1 = wg
                const unsigned r = i >> 1;
                const int slot = i % kSlots;
                // dK/dV pass: the slot's lse and delta values came with its tiles
                if (kMode == 1) ok = mbar_wait_warp(bar_full(slot), (i / kSlots) & 1, ctl, 234 + wg, i);
                if (ok) ok = mbar_wait_warp(bar_s_full(wg), r & 1, ctl, 230 + wg, i);
                if (!ok) break;
                tc_fence_after();
                uint32_t xp[16], xd[16], sr[32], dr[32];
                tc_ld_half64(tmem + C::s(wg) + t_lane, sr);
                tc_ld_half64(tmem + C::dp(wg) + t_lane, dr);
                tc_wait_ld();
                tc_fence_before();
                mbar_arrive_elect(bar_s_free(wg));  // S and dP may be overwritten by those of entry i + 2
                const float2* st2 = reinterpret_cast<const float2*>(smem + kOffStats + slot * kStatsBytes) + (lane & 3);
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (kMode == 1) {  // columns are query rows
                        nl0 = nl1 = st2[4 * k];
                        nd0 = nd1 = st2[4 * k + kBlk / 2];
                    }
                    pair(sr[4 * k], sr[4 * k + 1], dr[4 * k], dr[4 * k + 1], nl0, nd0, xp[2 * k], xd[2 * k]);
                    pair(sr[4 * k + 2], sr[4 * k + 3], dr[4 * k + 2], dr[4 * k + 3], nl1, nd1, xp[2 * k + 1], xd[2 * k + 1]);
                }
                // TS of entry i - 2 has read the columns
                ok = mbar_wait_warp(bar_ts_done(wg), (r & 1) ^ 1, ctl, 236 + wg, i);
                if (!ok) break;
                tc_fence_after();
                if (kMode == 1) tc_st_half32(tmem + C::xp(wg) + t_lane, xp);
                tc_st_half32(tmem + C::xd(wg) + t_lane, xd);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_elect(bar_x_full(wg));
            }
        } else if constexpr (kMode == 0) {
            const float2 nl = st[0], nd = st[1];
            for (unsigned i = s0 + ((s0 ^ wg) & 1); i < s0 + n && ok; i += 2) {  // buffer i & 1 = wg
                const unsigned r = i >> 1;
                ok = mbar_wait_warp(bar_s_full(wg), r & 1, ctl, 230 + wg, i);
                if (!ok) break;
                tc_fence_after();
                uint32_t xp[1], xd[32], sr[64], dr[64];
                tc_ld64(tmem + C::s(wg) + t_lane, sr);
                tc_ld64(tmem + C::dp(wg) + t_lane, dr);
                tc_wait_ld();
                tc_fence_before();
                mbar_arrive_elect(bar_s_free(wg));  // dP may be overwritten by that of entry i + 1, S by that of entry i + 2
#pragma unroll
                for (int k = 0; k < 32; ++k) pair(sr[2 * k], sr[2 * k + 1], dr[2 * k], dr[2 * k + 1], nl, nd, xp[0], xd[k]);
                // TS of entry i - 2 has read the columns
                ok = mbar_wait_warp(bar_ts_done(wg), (r & 1) ^ 1, ctl, 236 + wg, i);
                if (!ok) break;
                tc_fence_after();
                tc_st32(tmem + C::xd(wg) + t_lane, xd);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_elect(bar_x_full(wg));
            }
        } else {
            for (unsigned i = s0; i < s0 + n && ok; ++i) {  // columns 32 wg .. 32 wg + 31 of every entry
                const int slot = i % kSlots;
                // the slot's lse and delta values came with its tiles
                ok = mbar_wait_warp(bar_full(slot), (i / kSlots) & 1, ctl, 234 + wg, i);
                if (ok) ok = mbar_wait_warp(bar_s_full(0), i & 1, ctl, 232 + wg, i);
                if (!ok) break;
                tc_fence_after();
                uint32_t sr[32], dr[32];
                tc_ld32(tmem + C::s(0) + 32u * wg + t_lane, sr);
                tc_ld32(tmem + C::dp(0) + 32u * wg + t_lane, dr);
                tc_wait_ld();
                tc_fence_before();
                mbar_arrive_elect(bar_s_free(0));  // S^T and dP^T may be overwritten by the next entry's
                const float2* st2 = reinterpret_cast<const float2*>(smem + kOffStats + slot * kStatsBytes) + 16 * wg;
                uint32_t xp[16], xd[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) pair(sr[2 * k], sr[2 * k + 1], dr[2 * k], dr[2 * k + 1], st2[k], st2[k + kBlk / 2], xp[k], xd[k]);
                // TS of entry i - 1 has read the columns
                ok = mbar_wait_warp(bar_ts_done(0), (i & 1) ^ 1, ctl, 236 + wg, i);
                if (!ok) break;
                tc_fence_after();
                // 32 columns of the tile are 16 columns of 16-bit pairs
                tc_st16(tmem + C::xp(0) + 16u * wg + t_lane, xp);
                tc_st16(tmem + C::xd(0) + 16u * wg + t_lane, xd);
                tc_wait_st();
                tc_fence_before();
                mbar_arrive_elect(bar_x_full(0));
            }
        }
            s0 += n;
        };
        // The accumulated gradients of an item's rows: TMEM -> registers, which frees the accumulators -> global memory (rows in T,H,W order)
        auto store_item = [&](const Item& it, unsigned item) {
            const int bh = it.id / P.n_own, b = bh / P.heads, h = bh % P.heads;
            const long long tok = token(it, row);
            // Warpgroup g stores columns 64 g .. 64 g + 63 of dQ, or (kM = 64) of dV from lanes 0-15 and of dK from lanes 16-31;
            // dK/dV pass with kM = 128: warpgroup 0 stores dK, 1 dV.
            const bool whole = kMode == 1 && kM == 128;
            const bool second = kMode == 1 && (kM == 128 ? wg == 1 : lane < 16);
            unsigned char* base = static_cast<unsigned char*>(second ? P.out2 : P.out1);
            const long long sb = second ? P.o2_sb : P.o1_sb, sh = second ? P.o2_sh : P.o1_sh, ss = second ? P.o2_ss : P.o1_ss;
            unsigned char* row_ptr = base + ((long long)b * sb + (long long)h * sh + tok * ss) * 2;
            const uint32_t t_acc = tmem + (whole && second ? C::acc2 : 0u) + t_lane;
            const int col_lo = whole ? 0 : 64 * wg;
            const bool live = (kM == 128 || kMode == 1 || lane < 16) && tok >= 0;
            if (it.n > 0) {
                if (!mbar_wait_warp(bar_acc_done, item & 1, ctl, 240 + kMode, item)) return false;
            }
            tc_fence_after();
#pragma unroll
            for (int part = 0; part < (whole ? 2 : 1); ++part) {
                uint32_t acc[64];
                if (it.n > 0) {
                    tc_ld64(t_acc + col_lo + 64 * part, acc);
                    tc_wait_ld();
                    if (part == (whole ? 1 : 0)) {
                        tc_fence_before();
                        mbar_arrive_elect(bar_acc_free);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 64; ++j) acc[j] = 0u;  // nothing selected this block: its gradient is zero
                }
                if (live) store_row64<kBf16>(row_ptr, col_lo + 64 * part, acc);
            }
            return true;
        };
        // Item by item; the own tiles and row values of the next one are fetched before the gradients of this one are stored.
        unsigned k = 0;
        Item cur{-1, 0, 0};
        if (ok) cur = take_item(k++);
        bool moved = false;
        float2 st[4], st_n[4];
        while (ok && cur.id >= 0) {
            if (cur.n > 0 && !moved) {
                row_stats(cur, kM == 64 ? wq * 16 + (lane >> 2) : row, st[0], st[1]);
                if (kM == 64) row_stats(cur, wq * 16 + (lane >> 2) + 8, st[2], st[3]);
                ok = own_to_tmem(kk);
                if (!ok) break;
            }
            if (cur.n > 0) {
                entries(cur.n, st);
                if (!ok) break;
            }
            const Item nx = take_item(k++);
            moved = cur.n > 0 && nx.id >= 0 && nx.n > 0;
            if (moved) {
                row_stats(nx, kM == 64 ? wq * 16 + (lane >> 2) : row, st_n[0], st_n[1]);
                if (kM == 64) row_stats(nx, wq * 16 + (lane >> 2) + 8, st_n[2], st_n[3]);
                ok = own_to_tmem(kk + 1);
                if (!ok) break;
            }
            ok = store_item(cur, kk);
            if (cur.n > 0) ++kk;
            if (moved) {
#pragma unroll
                for (int j = 0; j < 4; ++j) st[j] = st_n[j];
            }
            cur = nx;
        }
    }

    // ---- teardown
    tc_fence_before();
    __syncthreads();
    if (tid == 0) ctl_report(ctl);
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

template <bool kBf16, int kMode, int kM, bool kCap = false>
cudaError_t launch_pass(const BwdTcParams& P, cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::atomic<int>& sms = device_states()[dev].sm_count;
    int sm_count = sms.load(std::memory_order_relaxed);
    if (sm_count == 0) {
        e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        sms.store(sm_count, std::memory_order_relaxed);
    }
    // the attribute is per device and per kernel; setting it on every call costs a microsecond and keeps this stateless
    e = cudaFuncSetAttribute(bwd_tc_kernel<kBf16, kMode, kM, kCap>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay<kM>::smem);
    if (e != cudaSuccess) return e;
    // a CTA holds its SM for the whole pass: those that the caller keeps free for other streams stay free here too
    const int usable = std::max(sm_count - attn_sm_reserve(), 1);
    bwd_tc_kernel<kBf16, kMode, kM, kCap><<<(unsigned)std::min(P.n_items, usable), kThreads, Lay<kM>::smem, st>>>(P);
    return cudaGetLastError();
}

template <int kMode>
cudaError_t launch_pass_any(bool bf16, int rows, const BwdTcParams& P, cudaStream_t st) {
    if constexpr (kMode == 0)
        if (P.gb.ragged) return rows == 128 ? launch_pass<true, 0, 128, true>(P, st) : launch_pass<true, 0, 64, true>(P, st);  // bf16 only
    if (rows == 128) return bf16 ? launch_pass<true, kMode, 128>(P, st) : launch_pass<false, kMode, 128>(P, st);
    return bf16 ? launch_pass<true, kMode, 64>(P, st) : launch_pass<false, kMode, 64>(P, st);
}

bool grid_fits(const Geom& g, int rows) { return g.bs == rows && g.ct <= 256 && g.ch <= 256 && g.cw <= 256; }

}  // namespace

bool attn_bwd_tc_supported(const BwdArgs& a, const BwdTcPlan& p) {
    const char* force = std::getenv("LCBSA_BWD_IMPL");  // "mma" keeps the warp-level kernels (for comparisons)
    if (force && std::strcmp(force, "mma") == 0) return false;
    if (a.dtype != LCBSA_BF16 && a.dtype != LCBSA_FP16) return false;
    if (a.D != kD) return false;
    if (!grid_fits(p.unit_q, 64) || !grid_fits(p.unit_k, 64)) return false;
    if ((p.unit_q.ragged || p.unit_k.ragged) && a.dtype != LCBSA_BF16) return false;  // see the note on ragged grids above
    if (!grid_fits(p.own_q, 64) && !grid_fits(p.own_q, 128)) return false;
    if (!grid_fits(p.own_k, 64) && !grid_fits(p.own_k, 128)) return false;
    if (encode_fn() == nullptr) return false;
    if ((long long)a.B * a.H * std::max(p.own_q.nblk, p.own_k.nblk) > 0x7fff0000ll) return false;  // items are counted in 32 bits
    const View* vs[4] = {&a.q, &a.dout, &a.k, &a.v};
    const Geom* gs[8] = {&p.own_q, &p.own_q, &p.own_k, &p.own_k, &p.unit_q, &p.unit_q, &p.unit_k, &p.unit_k};
    for (int i = 0; i < 8; ++i) {
        const View& v = *vs[i % 4];
        if (merge_mode(v, a.B, a.H, *gs[i]) < 0) return false;
        if (v.ss * 2 >= (1ll << 40) || v.sh * 2 >= (1ll << 40)) return false;
    }
    return true;
}

// a.delta, the lists of the plan and (for the dK/dV pass) their transposition are ready on the stream; a.stats is scratch
// of two floats per slot of every query block (B*H*Sq*2 floats on whole grids, more on ragged ones)
cudaError_t launch_attn_bwd_tc(const BwdArgs& a, const BwdTcPlan& p, cudaStream_t st, const char** why) {
    const long long Sq = (long long)a.gq.T * a.gq.H * a.gq.W;
    const long long BH = (long long)a.B * a.H;
    {
        const long long total = BH * p.unit_q.nblk * kBlk;  // every slot of every 64-token query unit
        bwd_stats_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a.lse, a.delta, p.unit_q, Sq, total, a.stats, a.next_item);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // maps: q and dout with the boxes of the dQ pass's own blocks and of the streamed query units; k and v likewise
    const int m_q_own = merge_mode(a.q, a.B, a.H, p.own_q), m_do_own = merge_mode(a.dout, a.B, a.H, p.own_q);
    const int m_q_u = merge_mode(a.q, a.B, a.H, p.unit_q), m_do_u = merge_mode(a.dout, a.B, a.H, p.unit_q);
    const int m_k_own = merge_mode(a.k, a.B, a.H, p.own_k), m_v_own = merge_mode(a.v, a.B, a.H, p.own_k);
    const int m_k_u = merge_mode(a.k, a.B, a.H, p.unit_k), m_v_u = merge_mode(a.v, a.B, a.H, p.unit_k);
    BwdTcParams P;
    std::memset(&P, 0, sizeof(P));
    P.stats = a.stats;
    P.lse = a.lse;
    P.delta = a.delta;
    P.Sq = Sq;
    P.status = a.status;
    P.heads = a.H;
    P.scale = a.sm_scale;
    P.scale2 = a.sm_scale * 1.4426950408889634f;
    const bool bf16 = a.dtype == LCBSA_BF16;

    // dQ pass: own tiles Q_i, dO_i (a query block of 64 or 128 tokens); streamed K_j, V_j (64-token units)
    if (!make_map(&P.tm_a1, a.dtype, a.q, a.B, a.H, p.own_q, m_q_own) || !make_map(&P.tm_a2, a.dtype, a.dout, a.B, a.H, p.own_q, m_do_own) ||
        !make_map(&P.tm_b1, a.dtype, a.k, a.B, a.H, p.unit_k, m_k_u) || !make_map(&P.tm_b2, a.dtype, a.v, a.B, a.H, p.unit_k, m_v_u)) {
        *why = "cuTensorMapEncodeTiled rejected a tensor";
        return cudaErrorInvalidValue;
    }
    P.merge_a1 = m_q_own; P.merge_a2 = m_do_own; P.merge_b1 = m_k_u; P.merge_b2 = m_v_u;
    P.ga = p.own_q; P.gb = p.unit_k;
    P.list = p.list_q; P.cnt = p.cnt_q; P.cap = p.cap_q; P.toff = nullptr; P.list_stride = 0;
    P.n_own = p.own_q.nblk; P.n_stream = p.unit_k.nblk;
    P.n_items = (int)(BH * p.own_q.nblk); P.next_item = a.next_item;
    P.out1 = const_cast<void*>(a.dq.data); P.o1_sb = a.dq.sb; P.o1_sh = a.dq.sh; P.o1_ss = a.dq.ss;
    P.out2 = nullptr;
    cudaError_t e = launch_pass_any<0>(bf16, p.own_q.bs, P, st);
    if (e != cudaSuccess) return e;

    // dK/dV pass: own tiles K_j, V_j (a key block of 64 or 128 tokens); streamed Q_i, dO_i (64-token units)
    if (!make_map(&P.tm_a1, a.dtype, a.k, a.B, a.H, p.own_k, m_k_own) || !make_map(&P.tm_a2, a.dtype, a.v, a.B, a.H, p.own_k, m_v_own) ||
        !make_map(&P.tm_b1, a.dtype, a.q, a.B, a.H, p.unit_q, m_q_u) || !make_map(&P.tm_b2, a.dtype, a.dout, a.B, a.H, p.unit_q, m_do_u)) {
        *why = "cuTensorMapEncodeTiled rejected a tensor";
        return cudaErrorInvalidValue;
    }
    P.merge_a1 = m_k_own; P.merge_a2 = m_v_own; P.merge_b1 = m_q_u; P.merge_b2 = m_do_u;
    P.ga = p.own_k; P.gb = p.unit_q;
    P.list = p.tidx; P.cnt = nullptr; P.cap = 0; P.toff = p.toff; P.list_stride = p.tidx_stride;
    P.n_own = p.own_k.nblk; P.n_stream = p.unit_q.nblk;
    P.n_items = (int)(BH * p.own_k.nblk); P.next_item = a.next_item + 1;
    P.out1 = const_cast<void*>(a.dk.data); P.o1_sb = a.dk.sb; P.o1_sh = a.dk.sh; P.o1_ss = a.dk.ss;
    P.out2 = const_cast<void*>(a.dv.data); P.o2_sb = a.dv.sb; P.o2_sh = a.dv.sh; P.o2_ss = a.dv.ss;
    return launch_pass_any<1>(bf16, p.own_k.bs, P, st);
}

}  // namespace lcbsa
