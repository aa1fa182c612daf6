// Block-sparse flash-attention forward for sm_100a: TMA + tcgen05 + TMEM.
//
// Stands in for the Triton kernel _attn_fwd_bsa_varlen_align
// (longcat_video/block_sparse_attention/flash_attn_bsa_varlen_mask.py:172-285) together with the
// three rearrange copies before it and the one after it (bsa_interface.py:650-659): the 3-D token
// blocks are fetched and the output is written by 5-D TMA boxes straight from/to T,H,W order.
//
// Shape handled: head_dim 128 or 64, query and key blocks of 64 tokens, bf16 or fp16.  The figures below are those of
// head_dim 128; at 64 a tile is one 64-column half, the rings have six slots, an S is half as many MMAs and a P V half as wide
// (2 x 16 heads of a 12x16x24 grid in fp16, 18 of 72 blocks, whole call: 130 us, 151 us with the merge on the softmax warps).
//
// One persistent CTA per SM.  A work item is a pair of consecutive query blocks of one head.  Each
// query block is a 64-row tile, i.e. an M=64 tcgen05 MMA whose accumulator occupies 16 lanes of every
// 32-lane TMEM quadrant; the two tiles of the pair sit in the lower and the upper 16 lanes of the same
// columns, so that a softmax warpgroup (128 threads, one TMEM lane each) serves both with every lane busy.
//
// The selected K/V blocks of the pair are dealt alternately to two softmax warpgroups (even blocks to
// warpgroup 0, odd blocks to warpgroup 1).  Each keeps its own running maximum, row sum and O accumulator,
// and the two partial results are merged once at the end of the work item (as in split-KV decoding) by four warps of
// their own, so the warpgroups never synchronise with each other inside the loop and one computes while the other waits.
//
//   warps 0-3, 4-7 : softmax warpgroups 0 and 1     warp 8  : TMA producer of Q and K
//   warp 9         : S = Q K^T issuer               warp 10 : O += P V issuer
//   warp 11        : TMA producer of V               warps 12-15 : Q to TMEM, merge and store of O (epilogue warps)
//
// Once per item the epilogue warps move the Q rows from shared memory to TMEM, where they are the A operand of
// every S of the item: with Q in shared memory an S reads as many bytes of Q as of K for every block.
// Per block i (warpgroup g = i & 1):  S = Q K^T  (M64 N64 K128, A from TMEM, fp32 result in the warpgroup's S columns)
// ->  the warpgroup reads S into registers with tcgen05.ld and releases the columns, so that the S of its next block is
// computed under its arithmetic  ->  exp2 online softmax in registers, P in the input dtype into the warpgroup's P columns
// with tcgen05.st, once its PV of the block before has finished  ->  O_g += P V  (M64 N128 K64, A operand from TMEM).
// With P written over S, S of a block could not start before the PV of an earlier block was through.
// K and V have a ring of three slots each (a slot = the tiles of both query blocks).  Each ring has a producer warp of
// its own, and the copies are issued by one elected lane of the converged warp: one warp for both rings, issuing from a
// divergent branch, needed about 950 cycles per ring slot and was what the rest waited for (V was requested 1700 cycles
// after its P was ready).
// What bounds it: M=64 MMAs, 16 x 32 + 8 x 64 = 1024 cycles of tensor pipe per block of a pair (an M=64 tile occupies the
// pipe like an M=128 one); inside an item a block takes 1025 to 1040 cycles.  K and V of the block come in at 64 bytes per
// cycle and SM meanwhile; tiles at the full rate would ask L2 for twice that (what it can deliver has not been measured).  An item
// boundary costs some 2700 cycles more (480p grid, 39 blocks per item: 42700 cycles per item by time stamps): PV of the next item
// waits for the epilogue warps to have read O.
// It was 8000 when the softmax warps merged and stored O before they took up the next item and the kernel had 162 KB of code, more than
// the instruction caches hold (68 KB now).  480p, 39 of 624 blocks, whole call with 8 heads: 565 us with both, 549 us with
// the smaller code, 532 us with epilogue warps; 720p grid of 45 rows (ragged, masks in the softmax warps), 32 heads: 13095,
// 12880, 11560 us.
//
// The MMAs are issued by whole converged warps with one elected lane (about 23 cycles per MMA for the
// warp; a single lane inside a divergent branch needs 50 and more).
//
// head_dim 128: the running maximum baked into O is only refreshed when the row maximum grows by more than 2^8
// (the accumulated values stay finite and the result is unchanged after the final division), so O is
// rarely rescaled in TMEM.  head_dim 64 takes every new maximum, for its precision (see the softmax loop).
//
// TMEM columns: O of warpgroup g at 128 * g (128 columns), its S at 256 + 64 * g, its P at 384 + 32 * g (two 16-bit
// values per column), Q at 448 (64 columns of 16-bit pairs); the second tile of the pair 16 lanes up in each.
//
// At the end of a work item the softmax warpgroups leave (maximum, row sum) in shared memory and go on with the next item, whose
// Q the epilogue warps have moved to TMEM as soon as the last S of the item was computed.  The epilogue warps then merge and
// normalise O, stage it in the Q buffer (which that Q has just left) and send it off by TMA store, after which the buffer
// takes the Q of the item after the next.  PV of the next item starts when they have O in registers.
//
// Every wait on an mbarrier is bounded: when a wait runs out the CTA records where, raises an abort
// flag that all roles poll, drains its outstanding bulk copies, frees its TMEM and returns.
#include "tc_common.cuh"


namespace lcbsa {

namespace {

using namespace tc;

constexpr int kBlk = 64;                    // tokens per query / key block
constexpr int kHalfBytes = kBlk * 128;      // one 64-column half of a tile: 64 rows x 128 B, 128B-swizzled
constexpr int kTilesPerWork = 2;            // the two query blocks of a pair
constexpr int kThreads = 512;
// Reference of a row whose blocks so far scored -inf throughout: finite, so that their probabilities are 0 and not NaN, and far
// enough below every score that the first one above -inf replaces it.
constexpr float kNoScore = -1e30f;
// setmaxnreg per warpgroup: (168 + 168 + 48 + 128) * 128 threads = the 64 K registers of the SM, 128 per thread at launch.  The
// epilogue warps hold 32 columns of both accumulators: with 96 registers (and 184 for the softmax warps) the 720p grid takes 11300 us
// instead of 11070.  ptxas reports 88 bytes of spill stores and 164 of loads per thread (ragged head_dim 128: 56 and 120), whatever
// the split of the budgets: 64 for the producers or 144 for the epilogue warps leave them much the same.
constexpr int kRegsSoftmax = 168, kRegsOther = 48, kRegsEpilogue = 128;

// TMEM columns: O accumulator of warpgroup g at 128 * g, its S at 256 + 64 * g, its P (16-bit pairs) at 384 + 32 * g; Q (16-bit pairs)
constexpr uint32_t kTmO = 0, kTmS = 256, kTmP = 384, kTmQ = 448;

// shared memory map (offsets from the 1024-byte aligned base of dynamic shared memory)
// Ring of the key masks of ragged grids, indexed by block number.  The K producer writes the masks of a block before it
// requests its tiles, at most six (the K ring) ahead of an S that waited for a softmax warpgroup to have read the masks of
// a block at most three further back: sixteen entries are never overwritten unread.
// They become visible through threads' arrivals alone: the producer's on k_full, then the S issuer's on s_full.
constexpr int kMaskRing = 16;
template <int kD> struct Lay {
    static constexpr int halves = kD / 64;
    static constexpr int tile = halves * kHalfBytes;     // one Q, K, V or O tile: 16 KiB at head_dim 128
    static constexpr int slot = kTilesPerWork * tile;    // a ring slot holds the K (or V) tiles of both query blocks
    static constexpr int slots = kD == 128 ? 3 : 6;      // of the K ring and of the V ring: 96 KiB each
    static constexpr int offQ = 0;
    static constexpr int offK = offQ + kTilesPerWork * tile;
    static constexpr int offV = offK + slots * slot;
    static constexpr int offBar = offV + slots * slot;
    // barriers: k_full[slots] k_empty[slots] v_full[slots] v_empty[slots] q_full q_free s_full[2] s_free[2] p_full[2] pv_done[2]
    //           ml_ready o_free o_staged qt_full qt_free
    static constexpr int numBars = 4 * slots + 2 + 8 + 5;
    static constexpr int offMisc = offBar + numBars * 8;  // abort flag, TMEM base
    static constexpr int offMl = offMisc + 64;            // [2 warpgroups][128 lanes] (maximum, row sum)
    static constexpr int offMask = offMl + 2 * 128 * 8;   // ragged grids: [kMaskRing][2 tiles] which keys of a block are present
    static constexpr int smem = offMask + kMaskRing * 16;
};

struct TcParams {
    CUtensorMap tm_q, tm_kv[2];  // [0]: K, [1]: V
    // Output maps.  Normally one (tm_o[0]).  With o_frames > 0 the query grid is the rank-major grid of a
    // context-parallel group: frames [r * o_frames, (r + 1) * o_frames) are the tokens of rank r, and the rows of a
    // query block are stored straight into rank r's result buffer (its own map, over this GPU's or a peer's memory).
    CUtensorMap tm_o[kMaxOutDst];
    int o_frames;
    const int32_t* idx;
    const int32_t* cnt;
    float* lse;
    unsigned int* status;
    int cap;
    int nq;         // query blocks per head
    int bh_total;   // B*H
    int heads;      // H
    int merge_q, merge_k, merge_v, merge_o;  // 0: batch folded into the head axis of the map, 1: into the T axis
    int Tq, Tk;     // frames (for merge == 1 coordinates)
    Geom gq, gk;
    float scale2;   // sm_scale * log2(e)
    int is_bf16;
};

// ------------------------------------------------------------------------------------------ kernel

__device__ __forceinline__ int clamp_cnt(const TcParams& P, int bh, int qt) {
    return qt < P.nq ? min(max(P.cnt[(long long)bh * P.nq + qt], 0), P.cap) : 0;
}

// kRagged: the key grid has partial blocks.  The masking code exists only in that instantiation, which keeps the
// instruction stream of the softmax loop of whole grids short (the loop is sensitive to instruction fetch).
template <bool kBf16, bool kRagged, int kD>
__global__ void __launch_bounds__(kThreads, 1) attn_tc_kernel(const __grid_constant__ TcParams P) {
    using Ly = Lay<kD>;
    constexpr int kHalves = Ly::halves, kTileBytes = Ly::tile, kSlotBytes = Ly::slot, kKSlots = Ly::slots, kVSlots = Ly::slots;
    constexpr int kOffQ = Ly::offQ, kOffK = Ly::offK, kOffV = Ly::offV, kOffBar = Ly::offBar, kOffMisc = Ly::offMisc, kOffMl = Ly::offMl;
    constexpr int kOffMask = Ly::offMask;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar0 = sbase + kOffBar;
    auto bar_k_full = [&](int s) { return bar0 + 8u * s; };
    auto bar_k_empty = [&](int s) { return bar0 + 8u * (kKSlots + s); };
    auto bar_v_full = [&](int s) { return bar0 + 8u * (2 * kKSlots + s); };
    auto bar_v_empty = [&](int s) { return bar0 + 8u * (2 * kKSlots + kVSlots + s); };
    constexpr int kB0 = 2 * kKSlots + 2 * kVSlots;
    const uint32_t bar_q_full = bar0 + 8u * kB0, bar_q_free = bar0 + 8u * (kB0 + 1);
    auto bar_s_full = [&](int wg) { return bar0 + 8u * (kB0 + 2 + wg); };
    auto bar_s_free = [&](int wg) { return bar0 + 8u * (kB0 + 4 + wg); };
    auto bar_p_full = [&](int wg) { return bar0 + 8u * (kB0 + 6 + wg); };
    auto bar_pv_done = [&](int wg) { return bar0 + 8u * (kB0 + 8 + wg); };
    constexpr int kB1 = kB0 + 10;
    const uint32_t bar_ml_ready = bar0 + 8u * kB1, bar_o_free = bar0 + 8u * (kB1 + 1), bar_o_staged = bar0 + 8u * (kB1 + 2);
    const uint32_t bar_qt_full = bar0 + 8u * (kB1 + 3), bar_qt_free = bar0 + 8u * (kB1 + 4);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kOffMisc);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffMisc + 8);
    float2* ml = reinterpret_cast<float2*>(smem + kOffMl);  // [2][128]
    unsigned long long* masks = reinterpret_cast<unsigned long long*>(smem + kOffMask);  // [kMaskRing][2]
    const Ctl ctl{abort_flag, P.status};

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // the same value, but provably warp-uniform

    if (tid == 0) {
        ctl_init(ctl);
        for (int s = 0; s < kKSlots; ++s) {
            mbar_init(bar_k_full(s), 1);
            mbar_init(bar_k_empty(s), 1);
        }
        for (int s = 0; s < kVSlots; ++s) {
            mbar_init(bar_v_full(s), 1);
            mbar_init(bar_v_empty(s), 1);
        }
        mbar_init(bar_q_full, 1);
        mbar_init(bar_q_free, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar_s_full(b), kRagged ? 2 : 1);  // the MMAs; ragged grids: and the issuer, for the masks
            mbar_init(bar_s_free(b), 4);
            mbar_init(bar_p_full(b), 4);  // one elected arrival per softmax warp
            mbar_init(bar_pv_done(b), 1);
        }
        mbar_init(bar_qt_full, 4);
        mbar_init(bar_qt_free, 1);
        mbar_init(bar_ml_ready, 8);
        mbar_init(bar_o_free, 4);
        mbar_init(bar_o_staged, 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // The tiles are 128B-swizzled, which ties their layout to address bits 7-9: without a 1024-byte aligned
        // base nothing below is valid.  The declaration asks for it; refuse to run if it was not honoured.
        if (sbase & 1023u) {
            *abort_flag = 1;
            if (atomicCAS(P.status, 0u, 1u) == 0u) {
                P.status[1] = blockIdx.x;
                P.status[2] = sbase;
                P.status[3] = 0;
            }
        }
    }
    if (warp == 9) {  // TMEM: all 512 columns, allocated and freed by the S issuer
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const bool start_ok = *abort_flag == 0;

    const int groups = (P.nq + kTilesPerWork - 1) / kTilesPerWork;
    const int total_work = start_ok ? P.bh_total * groups : 0;  // q alone has 32 KB per item, so this is far below 2^31
    // The CTA's items are blockIdx.x, blockIdx.x + gridDim.x, ...; every role steps through them as (head, group) pairs, since a
    // 64-bit division per role and item costs more than a round.
    const int first_bh = (int)(blockIdx.x / (unsigned)groups), first_g = (int)(blockIdx.x % (unsigned)groups);
    const int step_bh = (int)(gridDim.x / (unsigned)groups), step_g = (int)(gridDim.x % (unsigned)groups);
    auto next_item = [&](int& bh, int& g) {
        bh += step_bh;
        g += step_g;
        if (g >= groups) {
            g -= groups;
            ++bh;
        }
    };
    constexpr bool bf16 = kBf16;

    // All roles walk the same list of work items and blocks.  Block number gb (counted over the whole kernel)
    // uses slot gb % slots of the K ring and of the V ring.  Within an item block i belongs to warpgroup i & 1, which numbers its own rounds rr
    // over the whole kernel.
    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
        // ================================================================== epilogue warps
        // Between two items: Q of the next one from shared memory to TMEM as soon as the last S of the current one has read
        // the columns, then the merge of the two partial results, staged in the Q buffer that has just become free (a thread
        // writes the row that it read Q from) and sent off by TMA store.  The softmax warps meanwhile go on with the next item.
        const int wq = warp & 3;          // TMEM quadrant of this warp
        const int hf = lane >> 4;         // tile of the pair this lane serves
        const int row = wq * 16 + (lane & 15);  // row of that tile
        const uint32_t t_lane = (uint32_t)(wq * 32) << 16;
        const int ml_idx = wq * 32 + lane;
        unsigned char* const buf = smem + kOffQ + hf * kTileBytes + row * 128;  // this thread's row: chunk c at 16 * (c ^ (row & 7)), halves kHalfBytes apart
        unsigned wk = 0, rr0 = 0, rr1 = 0;  // rounds of the two softmax warpgroups over the whole kernel
        bool ok = true;
        auto q_to_tmem = [&](unsigned item) -> bool {  // Q of the CTA's work item number `item`
            // the last S of the item before has read the columns
            if (item > 0 && !mbar_wait_warp(bar_qt_free, (item - 1) & 1, ctl, 106, item)) return false;
            if (!mbar_wait_warp(bar_q_full, item & 1, ctl, 108, item)) return false;
            tc_fence_after();
#pragma unroll 1
            for (int half = 0; half < kHalves; ++half) {
                uint32_t qr[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(buf + half * kHalfBytes + ((c ^ (row & 7)) << 4));
                    qr[4 * c + 0] = v.x;
                    qr[4 * c + 1] = v.y;
                    qr[4 * c + 2] = v.z;
                    qr[4 * c + 3] = v.w;
                }
                tc_st32(tmem + kTmQ + 32u * half + t_lane, qr);
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            mbar_arrive_elect(bar_qt_full);
            return true;
        };
        int bh = 0, g = 0, nx_bh = first_bh, nx_g = first_g, my_n = 0, other_n = 0;
        auto peek = [&](bool there) {  // list lengths of item nx, read one item ahead
            if (there) {
                my_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork + hf);
                other_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork + (hf ^ 1));
            }
        };
        peek(blockIdx.x < total_work);
        int my_cnt = 0, n_iter = 0;
        for (int w = blockIdx.x;; w += gridDim.x) {  // item w gets its Q, the one before (number wk) is finished
            const bool there = w < total_work;
            const bool start = w == blockIdx.x;
            if (there && !q_to_tmem(start ? 0 : wk + 1)) break;
            // Behind the last item comes no Q, whose arrival would mean that the store of the item before has left the buffer.
            if (!there && wk > 0 && !mbar_wait_warp(bar_q_free, (wk - 1) & 1, ctl, 112, wk)) break;
            if (!start) {
            rr0 += (n_iter + 1) >> 1;
            rr1 += n_iter >> 1;

            // Both warpgroups have stored their last P, hence seen every PV but their last finish; no PV of the next item starts
            // before o_free, so the waits below are for exactly the item's last PVs.
            ok = mbar_wait_warp(bar_ml_ready, wk & 1, ctl, 104, wk);
            if (!ok) break;
            const float2 ml0 = ml[ml_idx], ml1 = ml[128 + ml_idx];
            // merged scale of both partial sums: everything relative to the larger reference maximum.  A row with a NaN or an
            // infinite score has a NaN sum and comes out as NaN, like on the warp-level kernel; a warpgroup that saw no block has
            // the maximum -inf, hence the weight 0.
            const float m_all = fmaxf(ml0.x, ml1.x), m_base = m_all == -INFINITY ? 0.f : m_all;
            const float w0 = ex2(ml0.x - m_base), w1 = ex2(ml1.x - m_base);
            // the accumulator of a warpgroup that saw no block holds garbage and is not used
            const bool saw0 = my_cnt > 0, saw1 = my_cnt > 1;
            const bool rd0 = __any_sync(0xffffffffu, saw0), rd1 = __any_sync(0xffffffffu, saw1);
            const bool both = __all_sync(0xffffffffu, saw1);  // the usual case: no lane has to be masked
            const float l_all = ml0.y * w0 + ml1.y * w1;
            const float inv = l_all == 0.f ? 0.f : 1.f / l_all;
            const float f0 = w0 * inv, f1 = w1 * inv;
            const float2 f0_2 = make_float2(f0, f0), f1_2 = make_float2(f1, f1);
            ok = mbar_wait_warp(bar_pv_done(0), (rr0 - 1) & 1, ctl, 100, wk);
            if (ok && n_iter > 1) ok = mbar_wait_warp(bar_pv_done(1), (rr1 - 1) & 1, ctl, 101, wk);
            if (!ok) break;
            tc_fence_after();
            const uint32_t tm_o = tmem + kTmO + t_lane;
#pragma unroll 1
            for (int cch = 0; cch < kD / 32; ++cch) {
                uint32_t oa[32], ob[32];
                if (rd0) tc_ld32(tm_o + 32 * cch, oa);
                if (rd1) tc_ld32(tm_o + 128 + 32 * cch, ob);
                tc_wait_ld();
                if (cch == kD / 32 - 1) {  // both O accumulators may be overwritten by the next item's first PVs
                    tc_fence_before();
                    __syncwarp();
                    mbar_arrive_elect(bar_o_free);
                }
                if (LCBSA_UNLIKELY(!both)) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (!saw0) oa[j] = 0u;
                        if (!saw1) ob[j] = 0u;
                    }
                }
                // the rows of a second tile that does not exist are written too; nobody stores them
                unsigned char* const half = buf + (cch >> 1) * kHalfBytes;
#pragma unroll
                for (int q8 = 0; q8 < 4; ++q8) {
                    uint32_t pw[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = q8 * 8 + 2 * j;
                        const float2 a2 = __fmul2_rn(make_float2(__uint_as_float(oa[e]), __uint_as_float(oa[e + 1])), f0_2);
                        const float2 v2 = __ffma2_rn(make_float2(__uint_as_float(ob[e]), __uint_as_float(ob[e + 1])), f1_2, a2);
                        pw[j] = pack2(bf16, v2.x, v2.y);
                    }
                    const int chunk = (cch & 1) * 4 + q8;
                    *reinterpret_cast<uint4*>(half + ((chunk ^ (row & 7)) << 4)) = make_uint4(pw[0], pw[1], pw[2], pw[3]);
                }
            }
            fence_proxy_async();
            __syncwarp();
            mbar_arrive_elect(bar_o_staged);
            const int qt = g * kTilesPerWork + hf;
            if (P.lse != nullptr && qt < P.nq) {
                int lt, lh, lw, bt, bhh, bw;
                slot_coords(P.gq, row, lt, lh, lw);
                block_coords(P.gq, qt, bt, bhh, bw);
                const int tt = bt * P.gq.ct + lt, hh = bhh * P.gq.ch + lh, ww = bw * P.gq.cw + lw;
                if (tt < P.gq.T && hh < P.gq.H && ww < P.gq.W) {
                    const long long Sq = (long long)P.gq.T * P.gq.H * P.gq.W;
                    const long long tok = ((long long)tt * P.gq.H + hh) * P.gq.W + ww;
                    P.lse[(long long)bh * Sq + tok] = l_all > 0.f ? (m_all + log2f(l_all)) * 0.6931471805599453f : -INFINITY;
                }
            }
            if (warp == 12) {  // the rows of all four warps are staged: off they go, then the buffer takes the Q after the next
                ok = mbar_wait_warp(bar_o_staged, wk & 1, ctl, 110, wk);
                if (!ok) break;
                const int qq = g * kTilesPerWork + lane;
                if (lane < 2 && qq < P.nq) {  // a tile each
                    const int b = bh / P.heads, h = bh - b * P.heads;
                    Coord cc = block_coord(P.gq, qq, b, h, P.heads, P.merge_o, P.Tq);
                    const CUtensorMap* tmo = &P.tm_o[0];
                    if (P.o_frames > 0) {  // blocks never straddle ranks: o_frames is a multiple of the block's frames
                        const int dst = cc.c3 / P.o_frames;
                        cc.c3 -= dst * P.o_frames;
                        tmo = &P.tm_o[dst];
                    }
                    const uint32_t src = sbase + kOffQ + lane * kTileBytes;
                    tma_store_5d(tmo, src, 0, cc.c1, cc.c2, cc.c3, cc.c4);
                    if (kHalves == 2) tma_store_5d(tmo, src + kHalfBytes, 64, cc.c1, cc.c2, cc.c3, cc.c4);
                    tma_store_commit();
                    tma_store_wait_read();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_q_free);
            }
            ++wk;
            }
            if (!there) break;
            bh = nx_bh;
            g = nx_g;
            my_cnt = my_n;
            n_iter = max(1, max(my_n, other_n));
            next_item(nx_bh, nx_g);
            peek(w + gridDim.x < total_work);
        }
        if (warp == 12 && lane < 2) tma_store_wait_all();
    } else if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
      if (warp == 8 || warp == 11) {
        // ================================================================== TMA producers: warp 8 Q and K, warp 11 V
        const bool is_k = warp == 8;
        // One code path for both rings: they have the same number of slots of the same size.
        const uint32_t ring = sbase + (is_k ? kOffK : kOffV), full0 = is_k ? bar_k_full(0) : bar_v_full(0), empty0 = is_k ? bar_k_empty(0) : bar_v_empty(0);
        unsigned gk = 0, wk = 0, nq_issued = 0;  // gk: blocks requested over the whole kernel
        int slot = 0;
        unsigned parity = 1;  // of the wait on an empty slot: the ring starts empty
        bool ok = true;
        // Q tiles of item (bh, g) into the Q buffer, one by lane 0 and one by lane 1
        auto request_q = [&](int bh, int g) {
            const int qt = g * kTilesPerWork + lane;
            if (lane == 0) mbar_arrive_tx(bar_q_full, min(P.nq - qt, 2) * kTileBytes);
            __syncwarp();
            if (lane < 2 && qt < P.nq) {
                const int b = bh / P.heads, h = bh - b * P.heads;
                const Coord cc = block_coord(P.gq, qt, b, h, P.heads, P.merge_q, P.Tq);
                const uint32_t dst = sbase + kOffQ + lane * kTileBytes;
                tma_load_5d(dst, &P.tm_q, bar_q_full, 0, cc.c1, cc.c2, cc.c3, cc.c4);
                if (kHalves == 2) tma_load_5d(dst + kHalfBytes, &P.tm_q, bar_q_full, 64, cc.c1, cc.c2, cc.c3, cc.c4);
            }
            ++nq_issued;
            __syncwarp();
        };
        if (is_k && blockIdx.x < total_work) request_q(first_bh, first_g);
        int bh = first_bh, g = first_g, nx_bh = first_bh, nx_g = first_g;
        int ca_n = 0, cb_n = 0;
        auto peek = [&](bool there) {  // list lengths of item nx, read one item ahead
            if (there) {
                ca_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork);
                cb_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork + 1);
            }
        };
        peek(blockIdx.x < total_work);
        // The first two windows of an item's list are read while the item before is under way: reading them at its start
        // kept the ring waiting for some 800 cycles.
        int raw0 = 0, raw1 = 0;
        auto load_ahead = [&](int bh, int g, int ca, int cb) {
            const int t = lane & 1, it = lane >> 1, c = t ? cb : ca;
            const int32_t* l = P.idx + ((long long)bh * P.nq + min(g * kTilesPerWork + t, P.nq - 1)) * P.cap;
            if (it < c) raw0 = l[it];
            if (16 + it < c) raw1 = l[16 + it];
        };
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk, bh = nx_bh, g = nx_g) {
            const int b = bh / P.heads, h = bh % P.heads;
            const int qa = g * kTilesPerWork;
            const int ca = ca_n, cb = cb_n;
            const int n_iter = max(1, max(ca, cb));
            // Block coordinates are fetched and decoded by the whole warp: lane L holds, for tile (L & 1) and
            // block win + (L >> 1), the block's first token packed as t << 20 | h << 10 | w.  `nxt` holds the window of
            // sixteen blocks behind the current one.
            const int my_t = lane & 1, my_s = lane >> 1;
            const int my_c = my_t ? cb : ca;
            const int32_t* my_l = P.idx + ((long long)bh * P.nq + min(qa + my_t, P.nq - 1)) * P.cap;
            auto decode = [&](int blk, int it) {  // list entry `it` of the lane's tile
                if (it >= my_c) return 0;
                if ((unsigned)blk >= (unsigned)P.gk.nblk) {
                    // A list entry outside [0, Nk) never becomes an address: its box is placed at w = W, wholly
                    // outside the tensor map, so TMA fills the tile with zeros; the call is flagged.
                    if (atomicCAS(P.status, 0u, kStatusBadBlockIndex) == 0u) {
                        P.status[1] = bh;
                        P.status[2] = qa + my_t;
                        P.status[3] = it;
                    }
                    return P.gk.W;
                }
                int bt, bhh, bw;
                block_coords(P.gk, blk, bt, bhh, bw);
                return ((bt * P.gk.ct) << 20) | ((bhh * P.gk.ch) << 10) | (bw * P.gk.cw);
            };
            if (wk == 0) load_ahead(bh, g, ca, cb);
            int cur = decode(raw0, my_s);
            int nxt = decode(raw1, 16 + my_s);
            next_item(nx_bh, nx_g);
            const bool more_items = w + gridDim.x < total_work;
            peek(more_items);
            const bool mrg = is_k ? P.merge_k : P.merge_v;
            const int c3 = mrg ? b * P.Tk : 0, c4 = mrg ? h : b * P.heads + h;
            // the boxes of both query blocks' tiles of list position j into ring slot `dst`
            auto request = [&](int j, const CUtensorMap* tm, uint32_t bar, uint32_t dst) {
                const int pa = __shfl_sync(0xffffffffu, cur, (j & 15) << 1), pb = __shfl_sync(0xffffffffu, cur, ((j & 15) << 1) | 1);
                mbar_arrive_tx_elect(bar, ((j < ca) + (j < cb)) * kTileBytes);
#pragma unroll 1
                for (int t = 0; t < 2; ++t, dst += kTileBytes) {
                    if (j >= (t ? cb : ca)) continue;
                    const int pt = t ? pb : pa;
                    tma_load_5d_elect(dst, tm, bar, 0, pt & 1023, (pt >> 10) & 1023, (pt >> 20) + c3, c4);
                    if (kHalves == 2) tma_load_5d_elect(dst + kHalfBytes, tm, bar, 64, pt & 1023, (pt >> 10) & 1023, (pt >> 20) + c3, c4);
                }
            };
            // ragged grids: which keys of this lane's list entry lie inside the grid (decoded here once per entry; the softmax
            // warps spent two divisions per round and thread on it)
            auto entry_mask = [&]() {
                return slot_mask64(P.gk.ct, P.gk.ch, P.gk.cw, P.gk.T - (cur >> 20), P.gk.H - ((cur >> 10) & 1023), P.gk.W - (cur & 1023));
            };
            unsigned long long my_mask = kRagged ? entry_mask() : 0ull;
            bool q_due = is_k && more_items;  // Q of the next item has not been requested yet
#pragma unroll 1
            for (int j = 0; j < n_iter; ++j) {
                // Q of the next item as soon as the buffer is free again (see the epilogue warps), which is early in this
                // item; behind the last chance for it comes the item's last K.
                if (q_due) {
                    const uint32_t bar = wk == 0 ? bar_qt_full : bar_q_free, ph = wk == 0 ? 0 : (wk - 1) & 1;
                    bool go = __all_sync(0xffffffffu, mbar_test(bar, ph));
                    if (!go && j == n_iter - 1) {
                        ok = go = mbar_wait_warp(bar, ph, ctl, 10, wk);
                        if (!ok) break;
                    }
                    if (go) {
                        request_q(nx_bh, nx_g);
                        q_due = false;
                    }
                }
                if (j == min(2, n_iter - 1) && more_items) load_ahead(nx_bh, nx_g, ca_n, cb_n);
                ok = mbar_wait_warp(empty0 + 8u * slot, parity, ctl, is_k ? 20 : 22, gk);
                if (!ok) break;
                if (kRagged && is_k) {
                    if (my_s == (j & 15)) masks[(gk % kMaskRing) * 2 + my_t] = my_mask;
                    __syncwarp();
                }
                request(j, &P.tm_kv[is_k ? 0 : 1], full0 + 8u * slot, ring + slot * kSlotBytes);
                ++gk;
                if (++slot == kKSlots) {
                    slot = 0;
                    parity ^= 1;
                }
                if ((j & 15) == 15) {
                    cur = nxt;
                    nxt = decode(j + 17 + my_s < my_c ? my_l[j + 17 + my_s] : 0, j + 17 + my_s);
                    if (kRagged) my_mask = entry_mask();
                }
            }
        }
        if (!ok && lane == 0) {
            // drain: give the copies this warp issued a bounded time to land before the CTA exits
            const long long t0 = clock64();
            for (unsigned r = gk > kKSlots ? gk - kKSlots : 0; r < gk; ++r)
                while (!mbar_try(full0 + 8u * (r % kKSlots), (r / kKSlots) & 1) && clock64() - t0 < 40000000ll) {
                }
            if (nq_issued > 0)
                while (!mbar_try(bar_q_full, (nq_issued - 1) & 1) && clock64() - t0 < 40000000ll) {
                }
        }
      } else if (warp == 9) {
        // ================================================================== S = Q K^T issuer
        const uint32_t idesc_s = instr_desc(bf16, 64, 64, 0);
        unsigned gb = 0, wk = 0, rr0 = 0, rr1 = 0;
        bool ok = true;
        int bh = first_bh, g = first_g, ca_n = 0, cb_n = 0;
        auto peek = [&](bool there) {  // list lengths of item (bh, g), which is then stepped: read one item ahead
            if (!there) return;
            ca_n = clamp_cnt(P, bh, g * kTilesPerWork);
            cb_n = clamp_cnt(P, bh, g * kTilesPerWork + 1);
            next_item(bh, g);
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk) {
            const int ca = ca_n, cb = cb_n;
            peek(w + gridDim.x < total_work);
            const int n_iter = max(1, max(ca, cb));
            ok = mbar_wait_warp(bar_qt_full, wk & 1, ctl, 30, wk);  // Q of this item is in TMEM
            bool pre = false;
            for (int i = 0; i < n_iter && ok; ++i, ++gb) {
                const int wg = i & 1;
                const unsigned rr = wg ? rr1 : rr0;
                const int slot = gb % kKSlots;
                if (!pre) {  // not already seen ready by the look-ahead of the block before
                    ok = mbar_wait_warp(bar_k_full(slot), (gb / kKSlots) & 1, ctl, 40, gb);
                    // the warpgroup has the S of its round before in registers
                    if (ok) ok = mbar_wait_warp(bar_s_free(wg), (rr & 1) ^ 1, ctl, 34 + wg, gb);
                    if (!ok) break;
                }
                // look ahead: probe the two barriers of the item's next block now, read the answer after the MMAs
                bool nk = false, np = false;
                if (i + 1 < n_iter) {
                    nk = mbar_test(bar_k_full((gb + 1) % kKSlots), ((gb + 1) / kKSlots) & 1);
                    np = mbar_test(bar_s_free(wg ^ 1), ((wg ? rr0 : rr1) & 1) ^ 1);
                }
                tc_fence_after();
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    if (!(i < (hf ? cb : ca))) continue;  // warp-uniform
                    const uint32_t qa = tmem + kTmQ + ((16u * hf) << 16);
                    const uint64_t kd = smem_desc(sbase + kOffK + slot * kSlotBytes + hf * kTileBytes, 16, 1024);
                    const uint32_t d = tmem + kTmS + 64u * wg + ((16u * hf) << 16);
#pragma unroll
                    for (int j = 0; j < kD / 16; ++j) {
                        // 32 bytes per 16-column step inside a 64-column half, halves 8 KiB apart
                        const uint64_t off = (uint64_t)(((j >> 2) * kHalfBytes + (j & 3) * 32) >> 4);
                        tc_mma_ts(d, qa + 8u * j, kd + off, idesc_s, j > 0);
                    }
                }
                tc_commit(bar_k_empty(slot));  // K is free once these MMAs have read it
                // The softmax warps read the block's key masks once s_full completes.  The masks are generic stores of the K
                // producer, which its arrival on k_full released to this warp; the commit only reports MMAs, so an arrival
                // of this warp passes them on.
                if (kRagged) mbar_arrive_elect(bar_s_full(wg));
                tc_commit(bar_s_full(wg));
                __syncwarp();
                if (i == n_iter - 1) tc_commit(bar_qt_free);  // and so are Q's TMEM columns after the last S of the item
                if (wg) ++rr1; else ++rr0;
                pre = __all_sync(0xffffffffu, nk && np);
            }
        }
      } else if (warp == 10) {
        // ================================================================== O += P V issuer
        const uint32_t idesc_pv = instr_desc(bf16, 64, kD, 1);
        unsigned gb = 0, wk = 0, rr0 = 0, rr1 = 0;
        bool ok = true;
        int bh = first_bh, g = first_g, ca_n = 0, cb_n = 0;
        auto peek = [&](bool there) {  // list lengths of item (bh, g), which is then stepped: read one item ahead
            if (!there) return;
            ca_n = clamp_cnt(P, bh, g * kTilesPerWork);
            cb_n = clamp_cnt(P, bh, g * kTilesPerWork + 1);
            next_item(bh, g);
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk) {
            const int ca = ca_n, cb = cb_n;
            peek(w + gridDim.x < total_work);
            const int n_iter = max(1, max(ca, cb));
            // the epilogue of the previous item has read both O accumulators
            ok = mbar_wait_warp(bar_o_free, (wk & 1) ^ 1, ctl, 36, wk);
            bool pre = false;
            for (int i = 0; i < n_iter && ok; ++i, ++gb) {
                const int wg = i & 1;
                const unsigned rr = wg ? rr1 : rr0;
                const int slot = gb % kVSlots;
                if (!pre) {
                    ok = mbar_wait_warp(bar_v_full(slot), (gb / kVSlots) & 1, ctl, 60, gb);
                    if (ok) ok = mbar_wait_warp(bar_p_full(wg), rr & 1, ctl, 50 + wg, gb);
                    if (!ok) break;
                }
                bool nv = false, np = false;  // look ahead to the item's next block
                if (i + 1 < n_iter) {
                    nv = mbar_test(bar_v_full((gb + 1) % kVSlots), ((gb + 1) / kVSlots) & 1);
                    np = mbar_test(bar_p_full(wg ^ 1), (wg ? rr0 : rr1) & 1);
                }
                tc_fence_after();
                // A: P in the warpgroup's 32 P columns, 8 columns per 16-key step; the second tile of
                // the pair sits 16 lanes up, like its accumulators.
                // B: V tile, MN-major: 64-column halves 8 KiB apart (LBO), 8-key groups 1 KiB apart (SBO).
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    if (!(i < (hf ? cb : ca))) continue;  // warp-uniform
                    const uint32_t pa = tmem + kTmP + 32u * wg + ((16u * hf) << 16);
                    const uint64_t vd = smem_desc(sbase + kOffV + slot * kSlotBytes + hf * kTileBytes, kHalfBytes, 1024);
                    const uint32_t d = tmem + kTmO + 128u * wg + ((16u * hf) << 16);
#pragma unroll
                    for (int j = 0; j < kBlk / 16; ++j)
                        tc_mma_ts(d, pa + 8u * j, vd + (uint64_t)((j * 2048) >> 4), idesc_pv, (i > 1 || j > 0) ? 1u : 0u);
                }
                tc_commit(bar_v_empty(slot));
                tc_commit(bar_pv_done(wg));
                __syncwarp();
                if (wg) ++rr1; else ++rr0;
                pre = __all_sync(0xffffffffu, nv && np);
            }
        }
      }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
        // ================================================================== softmax warpgroups
        const int wg = warp >> 2;         // warpgroup: takes blocks wg, wg + 2, ... of every work item
        const int wq = warp & 3;          // TMEM quadrant of this warp
        const int hf = lane >> 4;         // tile of the pair this lane serves
        const uint32_t t_lane = (uint32_t)(wq * 32) << 16;
        const uint32_t tm_s = tmem + kTmS + 64u * wg + t_lane, tm_p = tmem + kTmP + 32u * wg + t_lane;
        const uint32_t tm_o_mine = tmem + kTmO + 128u * wg + t_lane;
        const int ml_idx = wq * 32 + lane;
        unsigned wk = 0, gb = 0, rr = 0;  // rr: rounds of this warpgroup over the whole kernel
        bool ok = true;

        int bh = first_bh, g = first_g, nx_bh = first_bh, nx_g = first_g, my_n = 0, other_n = 0;
        auto peek = [&](bool there) {  // list lengths of item nx, read one item ahead
            if (there) {
                my_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork + hf);
                other_n = clamp_cnt(P, nx_bh, nx_g * kTilesPerWork + (hf ^ 1));
            }
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk, bh = nx_bh, g = nx_g) {
            const int my_cnt = my_n, other_cnt = other_n;
            next_item(nx_bh, nx_g);
            peek(w + gridDim.x < total_work);
            const int n_iter = max(1, max(my_cnt, other_cnt));

            float m_ref = -INFINITY, l_sum = 0.f;
            bool first = true;  // no block of this item seen yet by this warpgroup

            unsigned long long present = ~0ull;  // ragged grids: which keys of the round's block lie inside the grid
            // S of the warpgroup's round into registers; the buffer is then free for the S of its next round
            uint32_t sr[64];
            if (wg < n_iter) {
                ok = mbar_wait_warp(bar_s_full(wg), rr & 1, ctl, 80 + wg, rr);
                if (!ok) break;
                tc_fence_after();
                tc_ld64(tm_s, sr);
                if (kRagged) present = masks[((gb + wg) % kMaskRing) * 2 + hf];
                tc_wait_ld();
                tc_fence_before();
                mbar_arrive_elect(bar_s_free(wg));
            }
            for (int i = wg; i < n_iter && ok; i += 2, ++rr) {
                const bool active = i < my_cnt;
                float alpha = 1.f;
                bool need = false;
                uint4 pk[8];  // this row of P in the input dtype, 8 keys per 16-byte chunk
                if (active) {
                    if (kRagged) {  // keys of a partial block that lie outside the grid
                        if (present != ~0ull) {
                            const uint32_t p_lo = (uint32_t)present, p_hi = (uint32_t)(present >> 32);
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                if (!((p_lo >> j) & 1u)) sr[j] = 0xff800000u;  // -inf
                                if (!((p_hi >> j) & 1u)) sr[32 + j] = 0xff800000u;
                            }
                        }
                    }
                    // head_dim 128, one pass: the probabilities are computed against the current reference maximum while the row maximum is
                    // tracked beside them (one basic block, so that the comparisons run under the exponentials); only if the
                    // maximum has moved by more than 2^8 is the pass repeated with the new reference.  The warpgroup's first
                    // block takes its own maximum as the reference.
                    auto probs = [&](float mref, float& rsum) {
                        // two keys per instruction where the machine has packed fp32 forms (fma, add); the four partial
                        // sums take the keys j = 0, 1, 2, 3 (mod 4) in ascending order
                        const float2 sc2 = make_float2(P.scale2, P.scale2), nm2 = make_float2(-mref, -mref);
                        float2 r01 = make_float2(0.f, 0.f), r23 = make_float2(0.f, 0.f);
#pragma unroll
                        for (int cch = 0; cch < 8; ++cch) {
                            float2 e[4];
#pragma unroll
                            for (int jp = 0; jp < 4; ++jp) {
                                const float2 s2 = make_float2(__uint_as_float(sr[cch * 8 + 2 * jp]), __uint_as_float(sr[cch * 8 + 2 * jp + 1]));
                                const float2 x = __ffma2_rn(s2, sc2, nm2);
                                e[jp] = make_float2(ex2(x.x), ex2(x.y));
                            }
                            r01 = __fadd2_rn(r01, e[0]);
                            r23 = __fadd2_rn(r23, e[1]);
                            r01 = __fadd2_rn(r01, e[2]);
                            r23 = __fadd2_rn(r23, e[3]);
                            pk[cch].x = pack2(bf16, e[0].x, e[0].y);
                            pk[cch].y = pack2(bf16, e[1].x, e[1].y);
                            pk[cch].z = pack2(bf16, e[2].x, e[2].y);
                            pk[cch].w = pack2(bf16, e[3].x, e[3].y);
                        }
                        rsum = (r01.x + r01.y) + (r23.x + r23.y);
                    };
                    // the row maximum of this block, in units of log2
                    auto row_max = [&]() {
                        float mx8[8];  // eight chains of eight values, three at a time
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            auto sv = [&](int i) { return __uint_as_float(sr[8 * i + k]); };
                            mx8[k] = fmaxf(max3(max3(max3(sv(0), sv(1), sv(2)), sv(3), sv(4)), sv(5), sv(6)), sv(7));
                        }
                        return fmaxf(max3(max3(mx8[0], mx8[1], mx8[2]), mx8[3], mx8[4]), max3(mx8[5], mx8[6], mx8[7])) * P.scale2;
                    };
                    float rs = 0.f;
                    if constexpr (kD == 64) {
                        // The reference is the running maximum itself, as in the warp-level kernel that served head_dim 64 before:
                        // the largest probability of a row, which carries most of its weight, is then exactly 1 and not rounded
                        // to the input type.  With a reference that lags the error against float64 was 5 to 12 % larger.
                        const float m_new = fmaxf(m_ref, row_max());
                        if (!first && m_new > m_ref) {
                            need = true;
                            alpha = ex2(m_ref - m_new);
                        }
                        m_ref = fmaxf(m_new, kNoScore);
                        probs(m_ref, rs);
                    } else if (kRagged) {
                        // the instantiation with the masking code: a single copy of the pass in the instruction stream.  The loop
                        // body runs once in the common case (pass, then the row maximum, which confirms the reference) and twice
                        // when the reference moves; for the warpgroup's first block the first pass is skipped.
                        bool run_pass = !first, decided = false;
#pragma unroll 1
                        for (int turn = 0; turn < 2; ++turn) {
                            if (run_pass) probs(m_ref, rs);
                            if (decided) break;
                            const float m_new = fmaxf(m_ref, row_max());
                            run_pass = first || m_new - m_ref > 8.f;
                            if (!run_pass) break;
                            if (!first) {
                                need = true;
                                alpha = ex2(m_ref - m_new);
                            }
                            m_ref = fmaxf(m_new, kNoScore);
                            decided = true;
                        }
                    } else {
                        float m_new = m_ref;
                        if (LCBSA_UNLIKELY(first)) {
                            m_new = fmaxf(m_ref, row_max());
                            m_ref = fmaxf(m_new, kNoScore);
                        }
                        probs(m_ref, rs);
                        const float m_top = row_max();
                        if (LCBSA_UNLIKELY(m_top - m_ref > 8.f)) {
                            need = true;
                            alpha = ex2(m_ref - m_top);
                            m_ref = m_top;
                            probs(m_ref, rs);
                        }
                    }
                    l_sum = l_sum * alpha + rs;  // alpha is 1 unless this row's reference maximum moved
                }
                first = false;
                const bool any_need = __any_sync(0xffffffffu, need);
                // P may be overwritten, and O rescaled, once the warpgroup's PV of the round before has finished
                ok = mbar_wait_warp(bar_pv_done(wg), (rr & 1) ^ 1, ctl, 92 + wg, rr);
                if (!ok) break;
                tc_fence_after();  // orders the store of P behind the MMAs that read the columns (no other barrier does)
                {   // all 32 lanes take part in the store (a lane whose tile has run out of blocks writes don't-cares)
                    uint32_t pr[32];
#pragma unroll
                    for (int cch = 0; cch < 8; ++cch) {
                        pr[4 * cch + 0] = pk[cch].x;
                        pr[4 * cch + 1] = pk[cch].y;
                        pr[4 * cch + 2] = pk[cch].z;
                        pr[4 * cch + 3] = pk[cch].w;
                    }
                    tc_st32(tm_p, pr);
                }
                // head_dim 128: rare, only when a row maximum jumps
                if (kD == 64 ? any_need : LCBSA_UNLIKELY(any_need)) tc_scale_row<kD>(tm_o_mine, alpha);
                if (i + 2 < n_iter) {
                    // The next round's S is on its way into the registers while P is being stored: it has usually been ready
                    // for some hundred cycles, since it only waits for this round's S to be in registers.
                    ok = mbar_wait_warp(bar_s_full(wg), (rr + 1) & 1, ctl, 80 + wg, rr);
                    if (!ok) break;
                    tc_fence_after();
                    __syncwarp();
                    tc_ld64(tm_s, sr);
                    if (kRagged) present = masks[((gb + i + 2) % kMaskRing) * 2 + hf];
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive_elect(bar_p_full(wg));
                    tc_wait_ld();
                    tc_fence_before();
                    mbar_arrive_elect(bar_s_free(wg));
                } else {
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive_elect(bar_p_full(wg));
                }
            }
            if (!ok) break;
            gb += n_iter;
            // The epilogue warps merge this item's partial results; they have read the (maximum, row sum) of the item before once
            // they have arrived on o_free.
            if (wk > 0) {
                if (!__all_sync(0xffffffffu, mbar_test(bar_o_free, (wk - 1) & 1))) {
                    ok = mbar_wait_warp(bar_o_free, (wk - 1) & 1, ctl, 102 + wg, wk);
                    if (!ok) break;
                }
            }
            ml[wg * 128 + ml_idx] = make_float2(m_ref, l_sum);
            __syncwarp();
            mbar_arrive_elect(bar_ml_ready);
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

}  // namespace

namespace tc {
DeviceState* device_states() {
    static DeviceState states[kMaxDevices];
    return states;
}
}  // namespace tc

static std::atomic<int> g_sm_reserve{0};
int set_attn_sm_reserve(int n_sms) { return g_sm_reserve.exchange(n_sms); }
namespace tc {
int attn_sm_reserve() { return g_sm_reserve.load(); }
}  // namespace tc

bool attn_tc_supported(const AttnArgs& a, const char** why) {
    if (a.dtype != LCBSA_BF16 && a.dtype != LCBSA_FP16) { *why = "needs bf16 or fp16"; return false; }
    if (a.D != 128 && a.D != 64) { *why = "needs head_dim 64 or 128"; return false; }
    if (a.D == 64 && a.sm_scale < 0.f) {
        // The reference is the maximum of the raw scores times the scale, here the smallest scaled score of a block, and P grows
        // with the range of the scores.  Two partial results with references of their own let an fp16 P overflow where the one
        // of the warp-level kernel, which has always served head_dim 64 with such a scale, does not.
        *why = "head_dim 64 needs a scale that is not negative";
        return false;
    }
    if (a.gq.bs != kBlk || a.gk.bs != kBlk) { *why = "needs 64-token query and key blocks"; return false; }
    if (a.gq.ct > 256 || a.gq.ch > 256 || a.gq.cw > 256 || a.gk.ct > 256 || a.gk.ch > 256 || a.gk.cw > 256) {
        *why = "block axis above the TMA box limit";
        return false;
    }
    if (a.gk.T > 1023 || a.gk.H > 1023 || a.gk.W > 1023) {
        *why = "key grid axis above 1023 tokens (block coordinates are packed into 10-bit fields)";
        return false;
    }
    if (a.n_out_dst > 0) {
        if (a.n_out_dst > kMaxOutDst) { *why = "more than 8 output destinations"; return false; }
        if (a.B != 1) { *why = "scattered output needs batch 1"; return false; }
        if (a.gq.ragged || a.gq.T % a.n_out_dst != 0 || (a.gq.T / a.n_out_dst) % a.gq.ct != 0) {
            *why = "scattered output needs a query grid whose frames split evenly, on block boundaries, over the destinations";
            return false;
        }
    }
    const View* vs[4] = {&a.q, &a.k, &a.v, &a.o};
    const Geom* gs[4] = {&a.gq, &a.gk, &a.gk, &a.gq};
    for (int i = 0; i < (a.n_out_dst > 0 ? 3 : 4); ++i) {
        if (merge_mode(*vs[i], a.B, a.H, *gs[i]) < 0) { *why = "batch stride cannot be folded into a 5-D tensor map"; return false; }
        if (vs[i]->ss * 2 >= (1ll << 40) || vs[i]->sh * 2 >= (1ll << 40)) { *why = "stride too large for a tensor map"; return false; }
    }
    return true;
}

cudaError_t launch_attn_tc(const AttnArgs& a, cudaStream_t st, const char** why) {
    if (a.gq.nblk == 0 || a.B * a.H == 0) return cudaSuccess;
    TcParams P;
    const int mq = merge_mode(a.q, a.B, a.H, a.gq), mk = merge_mode(a.k, a.B, a.H, a.gk);
    const int mv = merge_mode(a.v, a.B, a.H, a.gk), mo = merge_mode(a.o, a.B, a.H, a.gq);
    if (!make_map(&P.tm_q, a.dtype, a.q, a.B, a.H, a.gq, mq, a.D) || !make_map(&P.tm_kv[0], a.dtype, a.k, a.B, a.H, a.gk, mk, a.D) ||
        !make_map(&P.tm_kv[1], a.dtype, a.v, a.B, a.H, a.gk, mv, a.D)) {
        *why = "cuTensorMapEncodeTiled rejected a tensor";
        return cudaErrorInvalidValue;
    }
    P.o_frames = 0;
    if (a.n_out_dst > 0) {
        // one map per destination over [D, W, H, T / n, heads]: the rank-major grid split along T
        Geom gl = a.gq;
        gl.T = a.gq.T / a.n_out_dst;
        P.o_frames = gl.T;
        for (int r = 0; r < a.n_out_dst; ++r) {
            View vo = a.o;
            vo.data = a.out_dst[r];
            if (!make_map(&P.tm_o[r], a.dtype, vo, 1, a.H, gl, 0, a.D)) {
                *why = "cuTensorMapEncodeTiled rejected a destination of the scattered output";
                return cudaErrorInvalidValue;
            }
        }
    } else if (!make_map(&P.tm_o[0], a.dtype, a.o, a.B, a.H, a.gq, mo, a.D)) {
        *why = "cuTensorMapEncodeTiled rejected a tensor";
        return cudaErrorInvalidValue;
    }
    P.idx = a.idx; P.cnt = a.cnt; P.lse = a.lse; P.status = a.status;
    P.cap = a.cap; P.nq = a.gq.nblk; P.bh_total = a.B * a.H; P.heads = a.H;
    P.merge_q = mq; P.merge_k = mk; P.merge_v = mv; P.merge_o = mo; P.Tq = a.gq.T; P.Tk = a.gk.T;
    P.gq = a.gq; P.gk = a.gk;
    P.scale2 = a.sm_scale * 1.4426950408889634f;
    P.is_bf16 = a.dtype == LCBSA_BF16;

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) { *why = "device ordinal above 63"; return cudaErrorInvalidValue; }
    DeviceState& ds = device_states()[dev];
    int sm_count = ds.sm_count.load(std::memory_order_relaxed);
    if (sm_count == 0) {
        e = cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        ds.sm_count.store(sm_count, std::memory_order_relaxed);
    }
    const bool ragged = a.gk.ragged;
    using Kern = void (*)(const TcParams);
    Kern kern;
    if (a.D == 128)
        kern = P.is_bf16 ? (ragged ? attn_tc_kernel<true, true, 128> : attn_tc_kernel<true, false, 128>)
                         : (ragged ? attn_tc_kernel<false, true, 128> : attn_tc_kernel<false, false, 128>);
    else
        kern = P.is_bf16 ? (ragged ? attn_tc_kernel<true, true, 64> : attn_tc_kernel<true, false, 64>)
                         : (ragged ? attn_tc_kernel<false, true, 64> : attn_tc_kernel<false, false, 64>);
    const int smem_bytes = a.D == 128 ? Lay<128>::smem : Lay<64>::smem;
    const int bit = (a.D == 128 ? 1 : 256) << ((P.is_bf16 ? 0 : 1) + (ragged ? 2 : 0));  // bits 0-3 and 8-11 of attr_set
    if (!(ds.attr_set.load(std::memory_order_relaxed) & bit)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        if (e != cudaSuccess) return e;
        ds.attr_set.fetch_or(bit, std::memory_order_relaxed);
    }
    const long long groups = (a.gq.nblk + kTilesPerWork - 1) / kTilesPerWork;
    const long long work = groups * a.B * a.H;
    const int usable = sm_count - g_sm_reserve.load() > 0 ? sm_count - g_sm_reserve.load() : 1;
    const int grid = (int)(work < usable ? work : usable);
    kern<<<grid, kThreads, smem_bytes, st>>>(P);
    return cudaGetLastError();
}

}  // namespace lcbsa
