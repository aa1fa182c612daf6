// Block-sparse flash-attention forward for sm_100a, 128-token blocks: TMA + tcgen05 + TMEM.
//
// The block shape that flash_attn_bsa_3d takes by default (chunk_3d_shape = [4, 4, 8], bsa_interface.py:619-622),
// for which the reference launches _attn_fwd_bsa_varlen_align with BLOCK_M = BLOCK_N_LG = 128
// (flash_attn_bsa_varlen_mask.py:172-285, launcher bsa_interface.py:290-341).  Same contract as attn_tc.cu (the
// 64-token kernel): q, k, v are read and the output is written straight from / to T,H,W order by 5-D TMA boxes.
//
// Shape handled: head_dim 128, query blocks of 128 tokens, key blocks of 128, 256 or 512 tokens (for which the
// reference switches to _attn_fwd_bsa_varlen, flash_attn_bsa_varlen_mask.py:37-153, bsa_interface.py:309-315), bf16 or fp16.
//
// One persistent CTA per SM.  A work item is ONE query block of one head: a 128-row tile, i.e. M=128 tcgen05 MMAs
// that run the tensor pipe at its full rate (the 64-row tiles of the other kernel occupy it like 128-row ones).  A
// selected key block is processed as 2, 4 or 8 units of 64 keys (sub-boxes of the block, cut along its outermost even
// axes), which keeps the S tile at 64 TMEM columns, so that S, P and O of both warpgroups and Q fit, exactly as in the
// 64-token kernel:
//
//   warps 0-3, 4-7 : softmax warpgroups 0 and 1 (units of even / odd number; thread = one query row)
//   warp 8 : TMA producer of Q and K   warp 9 : S = Q K^T issuer   warp 10 : O += P V issuer   warp 11: TMA producer of V
//   warps 12-15 : Q to TMEM, merge and store of O (epilogue warps)
//
// Per unit i (warpgroup g = i & 1):  S = Q K^T (M128 N64 K128, A = Q from TMEM) -> tcgen05.ld, exp2 online softmax in registers, P in the input dtype into TMEM columns of its own ->
// O_g += P V (M128 N128 K64, A from TMEM).  The two warpgroups keep separate maxima, row sums and accumulators and
// are merged once per work item by the epilogue warps, while the softmax warps go on with the next item.  K and V rings: six slots of one
// 64-key tile (16 KiB) each.  The finished O (128 rows x 256 B) is staged in the Q buffer and leaves by TMA store.
//
// Q in TMEM: an S with both operands in shared memory reads 48 KB of them per unit, which takes longer than its MMAs
// (M128 N64 K128: 256 cycles); with A from TMEM it reads 16 KB.
// What bounds it: the softmax warps.  A unit's MMAs take 512 cycles, its exponentials 512 cycles of the transcendental
// unit, and a warpgroup needs about 1900 cycles per round (two rounds per pair of units at the same time): the two
// warpgroups run in step, so nobody uses the transcendental unit while both store P and fetch S.  720p grid, 90 of 720
// blocks, 8 heads, attention launch: 5.08 ms with one producer warp, Q in shared memory and P over S; 4.0 ms without; with 32
// heads (16.5 ms) the launch runs into the power cap of the GPU.  Turns for the transcendental unit (a warp waits until the one
// that shares its scheduler is through with its exponentials) make it 5 % slower: alone, a warp needs 1000 cycles for them.
// Epilogue warps and code that fits the instruction caches (55 KB, 144 KB before): 720p, 32 heads, whole call 17277 -> 17047 us, timed
// in turn (at the power cap either way); forward attention of 8 heads of an 8x32x48 grid, 12 of 96 blocks, 93 -> 87 us.
//
// Every wait on an mbarrier is bounded, as in attn_tc.cu.
#include "tc_common.cuh"


namespace lcbsa {

namespace {

using namespace tc;

constexpr int kD = 128;
constexpr int kQRows = 128;                        // tokens per query block: one M=128 tile
constexpr int kBlk = 64;                           // keys per unit: a key block is 2, 4 or 8 units
constexpr int kQTileBytes = kQRows * kD * 2;       // 32 KiB: the Q tile, and the staged O tile
constexpr int kQHalfBytes = kQTileBytes / 2;       // one 64-column half of it: 128 rows x 128 B, 128B-swizzled
constexpr int kTileBytes = kBlk * kD * 2;          // 16 KiB: one K or V tile of 64 keys
constexpr int kHalfBytes = kTileBytes / 2;         // one 64-column half: 64 rows x 128 B
constexpr int kSlotBytes = kTileBytes;             // a ring slot holds one unit's tile
constexpr int kMaxUnits = 8;                       // units of 64 keys per key block: blocks of up to 512 tokens
constexpr int kKSlots = 6, kVSlots = 6;            // the same number: one code path serves both producers
constexpr int kThreads = 512;
// setmaxnreg per warpgroup: (176 + 176 + 48 + 112) * 128 threads = the 64 K registers of the SM, 128 per thread at launch
constexpr int kRegsSoftmax = 176, kRegsOther = 48, kRegsEpilogue = 112;

// TMEM columns: O accumulator of warpgroup g at 128 * g, its S at 256 + 64 * g, its P (16-bit pairs) at 384 + 32 * g; Q (16-bit pairs)
constexpr uint32_t kTmO = 0, kTmS = 256, kTmP = 384, kTmQ = 448;

// shared memory map (offsets from the 1024-byte aligned base of dynamic shared memory)
constexpr int kOffQ = 0;
constexpr int kOffK = kOffQ + kQTileBytes;
constexpr int kOffV = kOffK + kKSlots * kSlotBytes;
constexpr int kOffBar = kOffV + kVSlots * kSlotBytes;
// barriers: k_full[6] k_empty[6] v_full[6] v_empty[6] q_full q_free s_full[2] s_free[2] p_full[2] pv_done[2]
//           ml_ready o_free o_staged qt_full qt_free
constexpr int kNumBars = 2 * kKSlots + 2 * kVSlots + 2 + 8 + 5;
constexpr int kOffMisc = kOffBar + kNumBars * 8;      // abort flag, TMEM base
constexpr int kOffMl = kOffMisc + 64;                 // [2 warpgroups][128 lanes] (maximum, row sum)
constexpr int kSmemBytes = kOffMl + 2 * 128 * 8;

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
    // A key block of 128, 256 or 512 tokens is cut into 2, 4 or 8 units of 64 keys: unit u of a block starts
    // (sub_t[u], sub_h[u], sub_w[u]) tokens into it.  lg_units = log2 of the units per block.
    int lg_units;
    int sub_t[kMaxUnits], sub_h[kMaxUnits], sub_w[kMaxUnits];
    Geom gu;                // the key geometry with the block shape replaced by the unit's: slot order inside a unit
};

// ------------------------------------------------------------------------------------------ kernel

__device__ __forceinline__ int clamp_cnt(const TcParams& P, int bh, int qt) {
    return qt < P.nq ? min(max(P.cnt[(long long)bh * P.nq + qt], 0), P.cap) : 0;
}

// kRagged: the key grid has partial blocks.  The masking code exists only in that instantiation, which keeps the
// instruction stream of the softmax loop of whole grids short (the loop is sensitive to instruction fetch).
template <bool kBf16, bool kRagged>
__global__ void __launch_bounds__(kThreads, 1) attn_tc128_kernel(const __grid_constant__ TcParams P) {
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
            mbar_init(bar_s_full(b), 1);
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

    const int groups = P.nq;  // one work item per query block
    const int total_work = start_ok ? P.bh_total * groups : 0;  // q alone has 32 KB per item, so this is far below 2^31
    // The CTA's items are blockIdx.x, blockIdx.x + gridDim.x, ...; every role steps through them as (head, query block) pairs, since a
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

    // All roles walk the same list of work items and units.  Unit number gb (counted over the whole kernel)
    // uses K slot gb % 6 and V slot gb % 6.  Within an item unit i belongs to warpgroup i & 1.
    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
        // ================================================================== epilogue warps (as in attn_tc.cu)
        // Between two items: Q of the next one from shared memory to TMEM as soon as the last S of the current one has read
        // the columns, then the merge of the two partial results, staged in the Q buffer that has just become free (a thread
        // writes the row that it read Q from) and sent off by TMA store.  The softmax warps meanwhile go on with the next item.
        const int wq = warp & 3;          // TMEM quadrant of this warp
        const int row = wq * 32 + lane;   // row of the query block = TMEM lane
        const uint32_t t_lane = (uint32_t)(wq * 32) << 16;
        unsigned char* const buf = smem + kOffQ + row * 128;  // this thread's row: chunk c at 16 * (c ^ (row & 7)), halves kQHalfBytes apart
        unsigned wk = 0, rr = 0;  // rr: rounds of either softmax warpgroup over the whole kernel
        bool ok = true;
        auto q_to_tmem = [&](unsigned item) -> bool {  // Q of the CTA's work item number `item`
            // the last S of the item before has read the columns
            if (item > 0 && !mbar_wait_warp(bar_qt_free, (item - 1) & 1, ctl, 106, item)) return false;
            if (!mbar_wait_warp(bar_q_full, item & 1, ctl, 108, item)) return false;
            tc_fence_after();
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                uint32_t qr[32];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(buf + half * kQHalfBytes + ((c ^ (row & 7)) << 4));
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

        int bh = 0, qt = 0, nx_bh = first_bh, nx_g = first_g, cnt_n = 0, n_act = 0;
        auto peek = [&](bool there) {  // list length of item nx, read one item ahead
            if (there) cnt_n = clamp_cnt(P, nx_bh, nx_g);
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x;; w += gridDim.x) {  // item w gets its Q, the one before (number wk) is finished
            const bool there = w < total_work;
            const bool start = w == blockIdx.x;
            if (there && !q_to_tmem(start ? 0 : wk + 1)) break;
            // Behind the last item comes no Q, whose arrival would mean that the store of the item before has left the buffer.
            if (!there && wk > 0 && !mbar_wait_warp(bar_q_free, (wk - 1) & 1, ctl, 112, wk)) break;
            if (!start) {
                rr += max(2, n_act) >> 1;  // the units of an item are even in number and at least two
                // Both warpgroups have stored their last P, hence seen every PV but their last finish; no PV of the next item
                // starts before o_free, so the waits below are for exactly the item's last PVs.
                ok = mbar_wait_warp(bar_ml_ready, wk & 1, ctl, 104, wk);
                if (!ok) break;
                const float2 ml0 = ml[row], ml1 = ml[128 + row];
                // merged scale of both partial sums: everything relative to the larger reference maximum.  A row with a NaN or an
                // infinite score has a NaN sum and comes out as NaN, like on the warp-level kernel; a side that saw no key has the
                // maximum -inf, hence the weight 0.
                const float m_all = fmaxf(ml0.x, ml1.x), m_base = m_all == -INFINITY ? 0.f : m_all;
                const float w0 = ex2(ml0.x - m_base), w1 = ex2(ml1.x - m_base);
                const float l_all = ml0.y * w0 + ml1.y * w1;
                const float inv = l_all == 0.f ? 0.f : 1.f / l_all;
                const float f0 = w0 * inv, f1 = w1 * inv;
                const float2 f0_2 = make_float2(f0, f0), f1_2 = make_float2(f1, f1);
                const bool saw = n_act > 0;  // an empty list: the accumulators hold garbage and are not used
                ok = mbar_wait_warp(bar_pv_done(0), (rr - 1) & 1, ctl, 100, wk);
                if (ok) ok = mbar_wait_warp(bar_pv_done(1), (rr - 1) & 1, ctl, 101, wk);
                if (!ok) break;
                tc_fence_after();
                const uint32_t tm_o = tmem + kTmO + t_lane;
#pragma unroll 1
                for (int cch = 0; cch < kD / 32; ++cch) {
                    uint32_t oa[32], ob[32];
                    if (saw) {
                        tc_ld32(tm_o + 32 * cch, oa);
                        tc_ld32(tm_o + 128 + 32 * cch, ob);
                    }
                    tc_wait_ld();
                    if (cch == kD / 32 - 1) {  // both O accumulators may be overwritten by the next item's first PVs
                        tc_fence_before();
                        __syncwarp();
                        mbar_arrive_elect(bar_o_free);
                    }
                    if (LCBSA_UNLIKELY(!saw)) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) oa[j] = ob[j] = 0u;
                    }
                    unsigned char* const half = buf + (cch >> 1) * kQHalfBytes;
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
                if (P.lse != nullptr) {
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
                    if (lane == 0) {
                        const int b = bh / P.heads, h = bh - b * P.heads;
                        Coord cc = block_coord(P.gq, qt, b, h, P.heads, P.merge_o, P.Tq);
                        const CUtensorMap* tmo = &P.tm_o[0];
                        if (P.o_frames > 0) {  // blocks never straddle ranks: o_frames is a multiple of the block's frames
                            const int dst = cc.c3 / P.o_frames;
                            cc.c3 -= dst * P.o_frames;
                            tmo = &P.tm_o[dst];
                        }
                        tma_store_5d(tmo, sbase + kOffQ, 0, cc.c1, cc.c2, cc.c3, cc.c4);
                        tma_store_5d(tmo, sbase + kOffQ + kQHalfBytes, 64, cc.c1, cc.c2, cc.c3, cc.c4);
                        tma_store_commit();
                        tma_store_wait_read();
                        mbar_arrive(bar_q_free);
                    }
                    __syncwarp();
                }
                ++wk;
            }
            if (!there) break;
            bh = nx_bh;
            qt = nx_g;
            n_act = cnt_n << P.lg_units;
            next_item(nx_bh, nx_g);
            peek(w + gridDim.x < total_work);
        }
        if (warp == 12 && lane == 0) tma_store_wait_all();
    } else if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
      if (warp == 8 || warp == 11) {
        // ================================================================== TMA producers: warp 8 Q and K, warp 11 V
        const bool is_k = warp == 8;
        // One code path for both rings: they have the same number of slots of the same size.
        const uint32_t ring = sbase + (is_k ? kOffK : kOffV), full0 = is_k ? bar_k_full(0) : bar_v_full(0), empty0 = is_k ? bar_k_empty(0) : bar_v_empty(0);
        unsigned gk = 0, wk = 0, nq_issued = 0;  // gk: units requested over the whole kernel
        int slot = 0;
        unsigned parity = 1;  // of the wait on an empty slot: the ring starts empty
        bool ok = true;
        auto request_q = [&](int bh, int qb) {  // Q tile of item (bh, qb) into the Q buffer
            if (lane == 0) {
                mbar_arrive_tx(bar_q_full, kQTileBytes);
                const int b = bh / P.heads, h = bh - b * P.heads;
                const Coord cc = block_coord(P.gq, qb, b, h, P.heads, P.merge_q, P.Tq);
                tma_load_5d(sbase + kOffQ, &P.tm_q, bar_q_full, 0, cc.c1, cc.c2, cc.c3, cc.c4);
                tma_load_5d(sbase + kOffQ + kQHalfBytes, &P.tm_q, bar_q_full, 64, cc.c1, cc.c2, cc.c3, cc.c4);
            }
            ++nq_issued;
            __syncwarp();
        };
        if (is_k && blockIdx.x < total_work) request_q(first_bh, first_g);
        int bh = first_bh, qb = first_g, nx_bh = first_bh, nx_g = first_g;
        int cnt_n = 0;
        auto peek = [&](bool there) {  // list length of item nx, read one item ahead
            if (there) cnt_n = clamp_cnt(P, nx_bh, nx_g);
        };
        peek(blockIdx.x < total_work);
        // The first two windows of an item's list are read while the item before is under way.
        int raw0 = 0, raw1 = 0;
        auto load_ahead = [&](int bh, int qb, int cnt) {
            const int32_t* l = P.idx + ((long long)bh * P.nq + qb) * P.cap;
            if (lane < cnt) raw0 = l[lane];
            if (32 + lane < cnt) raw1 = l[32 + lane];
        };
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk, bh = nx_bh, qb = nx_g) {
            const int b = bh / P.heads, h = bh % P.heads;
            const int cnt = cnt_n;
            const int n_act = cnt << P.lg_units;  // units that exist: 2, 4 or 8 per listed key block
            const int n_iter = max(2, n_act);     // an empty list still goes through one (masked) pair of units
            // Block coordinates are fetched and decoded by the whole warp: lane L holds list entry 32 n + L as the
            // block's first token packed t << 20 | h << 10 | w.  `nxt` holds the thirty-two entries behind the current ones.
            const int32_t* my_l = P.idx + ((long long)bh * P.nq + qb) * P.cap;
            auto decode = [&](int blk, int e) {  // list entry e
                if (e >= cnt) return 0;
                if ((unsigned)blk >= (unsigned)P.gk.nblk) {
                    // A list entry outside [0, Nk) never becomes an address: its box is placed at w = W, wholly
                    // outside the tensor map, so TMA fills the tile with zeros; the call is flagged.
                    if (atomicCAS(P.status, 0u, kStatusBadBlockIndex) == 0u) {
                        P.status[1] = bh;
                        P.status[2] = qb;
                        P.status[3] = e;
                    }
                    return P.gk.W;
                }
                int bt, bhh, bw;
                block_coords(P.gk, blk, bt, bhh, bw);
                return ((bt * P.gk.ct) << 20) | ((bhh * P.gk.ch) << 10) | (bw * P.gk.cw);
            };
            if (wk == 0) load_ahead(bh, qb, cnt);
            int cur = decode(raw0, lane);
            int nxt = decode(raw1, 32 + lane);
            next_item(nx_bh, nx_g);
            const bool more_items = w + gridDim.x < total_work;
            peek(more_items);
            const bool mrg = is_k ? P.merge_k : P.merge_v;
            const int c3 = mrg ? b * P.Tk : 0, c4 = mrg ? h : b * P.heads + h;
            // the boxes of unit j: its block's first token plus the offset of the unit inside the block
            auto request = [&](int j, const CUtensorMap* tm, uint32_t bar, uint32_t dst) {
                const int e = j >> P.lg_units, u = j & ((1 << P.lg_units) - 1);
                const int pk = __shfl_sync(0xffffffffu, cur, e & 31);
                mbar_arrive_tx_elect(bar, j < n_act ? kTileBytes : 0);
                if (j < n_act) {
                    const int cw = (pk & 1023) + P.sub_w[u], chh = ((pk >> 10) & 1023) + P.sub_h[u], ctt = (pk >> 20) + P.sub_t[u] + c3;
                    tma_load_5d_elect(dst, tm, bar, 0, cw, chh, ctt, c4);
                    tma_load_5d_elect(dst + kHalfBytes, tm, bar, 64, cw, chh, ctt, c4);
                }
                if ((e & 31) == 31 && u == (1 << P.lg_units) - 1) {
                    cur = nxt;
                    nxt = decode(e + 33 + lane < cnt ? my_l[e + 33 + lane] : 0, e + 33 + lane);
                }
            };
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
                if (j == min(2, n_iter - 1) && more_items) load_ahead(nx_bh, nx_g, cnt_n);
                ok = mbar_wait_warp(empty0 + 8u * slot, parity, ctl, is_k ? 20 : 22, gk);
                if (!ok) break;
                request(j, &P.tm_kv[is_k ? 0 : 1], full0 + 8u * slot, ring + slot * kSlotBytes);
                ++gk;
                if (++slot == kKSlots) {
                    slot = 0;
                    parity ^= 1;
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
        const uint32_t idesc_s = instr_desc(bf16, kQRows, kBlk, 0);
        unsigned gb = 0, wk = 0, rr0 = 0, rr1 = 0;
        bool ok = true;
        int bh = first_bh, g = first_g, cnt_n = 0;
        auto peek = [&](bool there) {  // list length of item (bh, g), which is then stepped: read one item ahead
            if (!there) return;
            cnt_n = clamp_cnt(P, bh, g);
            next_item(bh, g);
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk) {
            const int n_act = cnt_n << P.lg_units;
            peek(w + gridDim.x < total_work);
            const int n_iter = max(2, n_act);
            ok = mbar_wait_warp(bar_qt_full, wk & 1, ctl, 30, wk);  // Q of this item is in TMEM
            bool pre = false;
            for (int i = 0; i < n_iter && ok; ++i, ++gb) {
                const int wg = i & 1;
                const unsigned rr = wg ? rr1 : rr0;
                const int slot = gb % kKSlots;
                if (!pre) {  // not already seen ready by the look-ahead of the unit before
                    ok = mbar_wait_warp(bar_k_full(slot), (gb / kKSlots) & 1, ctl, 40, gb);
                    // the warpgroup has the S of its round before in registers
                    if (ok) ok = mbar_wait_warp(bar_s_free(wg), (rr & 1) ^ 1, ctl, 34 + wg, gb);
                    if (!ok) break;
                }
                // look ahead: probe the two barriers of the item's next unit now, read the answer after the MMAs
                bool nk = false, np = false;
                if (i + 1 < n_iter) {
                    nk = mbar_test(bar_k_full((gb + 1) % kKSlots), ((gb + 1) / kKSlots) & 1);
                    np = mbar_test(bar_s_free(wg ^ 1), ((wg ? rr0 : rr1) & 1) ^ 1);
                }
                tc_fence_after();
                if (i < n_act) {
                    const uint64_t kd = smem_desc(sbase + kOffK + slot * kSlotBytes, 16, 1024);
                    const uint32_t d = tmem + kTmS + 64u * wg;
#pragma unroll
                    for (int j = 0; j < kD / 16; ++j) {
                        // 32 bytes per 16-column step inside a 64-column half, halves 8 KiB apart
                        const uint64_t koff = (uint64_t)(((j >> 2) * kHalfBytes + (j & 3) * 32) >> 4);
                        tc_mma_ts(d, tmem + kTmQ + 8u * j, kd + koff, idesc_s, j > 0);
                    }
                }
                tc_commit(bar_k_empty(slot));  // K is free once these MMAs have read it
                tc_commit(bar_s_full(wg));
                __syncwarp();
                if (i == n_iter - 1) tc_commit(bar_qt_free);  // and so are Q's TMEM columns after the last S of the item
                if (wg) ++rr1; else ++rr0;
                pre = __all_sync(0xffffffffu, nk && np);
            }
        }
      } else if (warp == 10) {
        // ================================================================== O += P V issuer
        const uint32_t idesc_pv = instr_desc(bf16, kQRows, kD, 1);
        unsigned gb = 0, wk = 0, rr0 = 0, rr1 = 0;
        bool ok = true;
        int bh = first_bh, g = first_g, cnt_n = 0;
        auto peek = [&](bool there) {  // list length of item (bh, g), which is then stepped: read one item ahead
            if (!there) return;
            cnt_n = clamp_cnt(P, bh, g);
            next_item(bh, g);
        };
        peek(blockIdx.x < total_work);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk) {
            const int n_act = cnt_n << P.lg_units;
            peek(w + gridDim.x < total_work);
            const int n_iter = max(2, n_act);
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
                bool nv = false, np = false;  // look ahead to the item's next unit
                if (i + 1 < n_iter) {
                    nv = mbar_test(bar_v_full((gb + 1) % kVSlots), ((gb + 1) / kVSlots) & 1);
                    np = mbar_test(bar_p_full(wg ^ 1), (wg ? rr0 : rr1) & 1);
                }
                tc_fence_after();
                // A: P in the warpgroup's 32 P columns, 8 columns per 16-key step.
                // B: V tile, MN-major: 64-column halves 8 KiB apart (LBO), 8-key groups 1 KiB apart (SBO).
                if (i < n_act) {
                    const uint32_t pa = tmem + kTmP + 32u * wg;
                    const uint64_t vd = smem_desc(sbase + kOffV + slot * kSlotBytes, kHalfBytes, 1024);
                    const uint32_t d = tmem + kTmO + 128u * wg;
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
        const int wg = warp >> 2;         // warpgroup: takes units wg, wg + 2, ... of every work item
        const int wq = warp & 3;          // TMEM quadrant of this warp
        const int row = wq * 32 + lane;   // row of the query block = TMEM lane
        const uint32_t t_lane = (uint32_t)(wq * 32) << 16;
        const uint32_t tm_s = tmem + kTmS + 64u * wg + t_lane, tm_p = tmem + kTmP + 32u * wg + t_lane;
        const uint32_t tm_o_mine = tmem + kTmO + 128u * wg + t_lane;
        unsigned wk = 0, rr = 0;  // rr: rounds of this warpgroup over the whole kernel
        bool ok = true;

        int bh = first_bh, qt = first_g, nx_bh = first_bh, nx_g = first_g, cnt_n = 0;
        if (blockIdx.x < total_work) cnt_n = clamp_cnt(P, bh, qt);
        for (int w = blockIdx.x; w < total_work && ok; w += gridDim.x, ++wk, bh = nx_bh, qt = nx_g) {
            const int n_act = cnt_n << P.lg_units;
            next_item(nx_bh, nx_g);
            if (w + gridDim.x < total_work) cnt_n = clamp_cnt(P, nx_bh, nx_g);  // read one item ahead
            const int n_iter = max(2, n_act);
            const int32_t* my_list = P.idx + ((long long)bh * P.nq + qt) * P.cap;

            float m_ref = -INFINITY, l_sum = 0.f;
            bool first = true;  // no block of this item seen yet by this warpgroup

            // ragged grids: the block index of a round is fetched a round ahead, so that the global load never sits
            // between S and the softmax (unit i belongs to list entry i >> lg_units)
            int blk_ahead = (kRagged && wg < n_act) ? my_list[0] : 0;
            // S of the warpgroup's round into registers; the buffer is then free for the S of its next round
            uint32_t sr[64];
            if (wg < n_iter) {
                ok = mbar_wait_warp(bar_s_full(wg), rr & 1, ctl, 80 + wg, rr);
                if (!ok) break;
                tc_fence_after();
                tc_ld64(tm_s, sr);
                tc_wait_ld();
                tc_fence_before();
                mbar_arrive_elect(bar_s_free(wg));
            }
            for (int i = wg; i < n_iter && ok; i += 2, ++rr) {
                const bool active = i < n_act;
                const int blk_now = blk_ahead;
                if (kRagged && i + 2 < n_act) blk_ahead = my_list[(i + 2) >> P.lg_units];
                float alpha = 1.f;
                bool need = false;
                uint4 pk[8];  // this row of P in the input dtype, 8 keys per 16-byte chunk
                if (active) {
                    if (kRagged) {  // keys of a partial block that lie outside the grid
                        const int blk = blk_now;
                        int bt, bhh, bw;
                        block_coords(P.gk, blk, bt, bhh, bw);
                        // tokens left along each axis from the first token of this unit
                        int vt = P.gk.T - bt * P.gk.ct, vh = P.gk.H - bhh * P.gk.ch, vw = P.gk.W - bw * P.gk.cw;
                        const int sub = i & ((1 << P.lg_units) - 1);
                        vt -= P.sub_t[sub];
                        vh -= P.sub_h[sub];
                        vw -= P.sub_w[sub];
                        if (vt < P.gu.ct || vh < P.gu.ch || vw < P.gu.cw) {
                            const uint64_t present = slot_mask64(P.gu.ct, P.gu.ch, P.gu.cw, vt, vh, vw);
                            const uint32_t p_lo = (uint32_t)present, p_hi = (uint32_t)(present >> 32);
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                if (!((p_lo >> j) & 1u)) sr[j] = 0xff800000u;  // -inf
                                if (!((p_hi >> j) & 1u)) sr[32 + j] = 0xff800000u;
                            }
                        }
                    }
                    // One pass: the probabilities are computed against the current reference maximum while the row maximum is
                    // tracked beside them (one basic block, so that the comparisons run under the exponentials); only if the
                    // maximum has moved by more than 2^8 is the pass repeated with the new reference.  The warpgroup's first
                    // unit takes its own maximum as the reference.
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
                    // the row maximum of this unit, in units of log2
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
                    float m_new = m_ref;
                    if (LCBSA_UNLIKELY(first)) {
                        m_new = row_max();
                        m_ref = (m_new == -INFINITY) ? 0.f : m_new;
                    }
                    first = first && m_new == -INFINITY;  // a unit wholly outside a ragged grid leaves no reference behind
                    probs(m_ref, rs);
                    const float m_top = row_max();
                    if (LCBSA_UNLIKELY(m_top - m_ref > 8.f)) {
                        need = true;
                        alpha = ex2(m_ref - m_top);
                        m_ref = m_top;
                        probs(m_ref, rs);
                    }
                    l_sum = l_sum * alpha + rs;  // alpha is 1 unless this row's reference maximum moved
                } else {
                    first = false;
                }
                const bool any_need = __any_sync(0xffffffffu, need);
                // P may be overwritten, and O rescaled, once the warpgroup's PV of the round before has finished.  The next S
                // only waits for this one to be in registers, so it is usually there too: both barriers are probed at once
                // (a wait costs its warp 200 cycles even on a completed phase) and the next S is fetched under the store of P.
                const bool more = i + 2 < n_iter;
                const bool pv_ok = mbar_test(bar_pv_done(wg), (rr & 1) ^ 1), s_ok = !more || mbar_test(bar_s_full(wg), (rr + 1) & 1);
                const bool ready = __all_sync(0xffffffffu, pv_ok && s_ok);
                if (!ready) {
                    ok = mbar_wait_warp(bar_pv_done(wg), (rr & 1) ^ 1, ctl, 92 + wg, rr);
                    if (!ok) break;
                }
                tc_fence_after();  // orders the store of P behind the MMAs that read the columns (no other barrier does)
                uint32_t pr[32];  // all 32 lanes take part in the store (don't-cares for a unit that does not exist)
#pragma unroll
                for (int cch = 0; cch < 8; ++cch) {
                    pr[4 * cch + 0] = pk[cch].x;
                    pr[4 * cch + 1] = pk[cch].y;
                    pr[4 * cch + 2] = pk[cch].z;
                    pr[4 * cch + 3] = pk[cch].w;
                }
                if (LCBSA_UNLIKELY(any_need)) tc_scale_row<kD>(tm_o_mine, alpha);  // rare: only when a row maximum jumps
                if (ready && more) {
                    tc_st32(tm_p, pr);
                    tc_ld64(tm_s, sr);
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive_elect(bar_p_full(wg));
                    tc_wait_ld();
                    tc_fence_before();
                    mbar_arrive_elect(bar_s_free(wg));
                } else {
                    tc_st32(tm_p, pr);
                    tc_wait_st();
                    tc_fence_before();
                    mbar_arrive_elect(bar_p_full(wg));
                    if (more) {
                        ok = mbar_wait_warp(bar_s_full(wg), (rr + 1) & 1, ctl, 80 + wg, rr);
                        if (!ok) break;
                        tc_fence_after();
                        tc_ld64(tm_s, sr);
                        tc_wait_ld();
                        tc_fence_before();
                        mbar_arrive_elect(bar_s_free(wg));
                    }
                }
            }
            if (!ok) break;
            // The epilogue warps merge this item's partial results; they have read the (maximum, row sum) of the item before once
            // they have arrived on o_free.
            if (wk > 0) {
                if (!__all_sync(0xffffffffu, mbar_test(bar_o_free, (wk - 1) & 1))) {
                    ok = mbar_wait_warp(bar_o_free, (wk - 1) & 1, ctl, 102 + wg, wk);
                    if (!ok) break;
                }
            }
            ml[wg * 128 + row] = make_float2(first ? -INFINITY : m_ref, l_sum);  // no key seen: m_ref is a placeholder
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

// Cuts a key block of 64 * 2^k tokens into units of 64 keys: the outermost even axis is halved until 64 tokens are
// left, so that a unit is one TMA box and the units are as close to contiguous runs of the block's slot order as the
// shape allows.  (ut, uh, uw): the unit's extents; units are numbered t-major, then h, then w.
struct UnitSplit {
    int ut, uh, uw, lg_units;
};
static UnitSplit split_into_units(const Geom& g) {
    UnitSplit u{g.ct, g.ch, g.cw, 0};
    while (u.ut * u.uh * u.uw > kBlk) {
        if (u.ut % 2 == 0) u.ut /= 2;
        else if (u.uh % 2 == 0) u.uh /= 2;
        else u.uw /= 2;  // the token count is a power of two, so some axis is even
        ++u.lg_units;
    }
    return u;
}

bool attn_tc128_supported(const AttnArgs& a, const char** why) {
    if (a.dtype != LCBSA_BF16 && a.dtype != LCBSA_FP16) { *why = "needs bf16 or fp16"; return false; }
    if (a.D != kD) { *why = "needs head_dim 128"; return false; }
    if (a.gq.bs != kQRows || (a.gk.bs != 128 && a.gk.bs != 256 && a.gk.bs != 512)) {
        *why = "needs 128-token query blocks and key blocks of 128, 256 or 512 tokens";
        return false;
    }
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

cudaError_t launch_attn_tc128(const AttnArgs& a, cudaStream_t st, const char** why) {
    if (a.gq.nblk == 0 || a.B * a.H == 0) return cudaSuccess;
    TcParams P;
    // geometry of one unit of 64 keys, and where every unit starts inside its block
    const UnitSplit us = split_into_units(a.gk);
    Geom gu = a.gk;
    gu.ct = us.ut; gu.ch = us.uh; gu.cw = us.uw;
    gu.bs = kBlk;
    P.lg_units = us.lg_units;
    {
        const int ph = a.gk.ch / us.uh, pw = a.gk.cw / us.uw;
        for (int u = 0; u < (1 << us.lg_units); ++u) {
            P.sub_w[u] = (u % pw) * us.uw;
            P.sub_h[u] = ((u / pw) % ph) * us.uh;
            P.sub_t[u] = (u / (pw * ph)) * us.ut;
        }
        for (int u = 1 << us.lg_units; u < kMaxUnits; ++u) P.sub_t[u] = P.sub_h[u] = P.sub_w[u] = 0;
    }
    P.gu = gu;
    const int mq = merge_mode(a.q, a.B, a.H, a.gq), mk = merge_mode(a.k, a.B, a.H, a.gk);
    const int mv = merge_mode(a.v, a.B, a.H, a.gk), mo = merge_mode(a.o, a.B, a.H, a.gq);
    if (!make_map(&P.tm_q, a.dtype, a.q, a.B, a.H, a.gq, mq) || !make_map(&P.tm_kv[0], a.dtype, a.k, a.B, a.H, gu, mk) ||
        !make_map(&P.tm_kv[1], a.dtype, a.v, a.B, a.H, gu, mv)) {
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
            if (!make_map(&P.tm_o[r], a.dtype, vo, 1, a.H, gl, 0)) {
                *why = "cuTensorMapEncodeTiled rejected a destination of the scattered output";
                return cudaErrorInvalidValue;
            }
        }
    } else if (!make_map(&P.tm_o[0], a.dtype, a.o, a.B, a.H, a.gq, mo)) {
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
    auto kern = P.is_bf16 ? (ragged ? attn_tc128_kernel<true, true> : attn_tc128_kernel<true, false>)
                          : (ragged ? attn_tc128_kernel<false, true> : attn_tc128_kernel<false, false>);
    const int bit = 16 << ((P.is_bf16 ? 0 : 1) + (ragged ? 2 : 0));  // bits 4-7 of attr_set
    if (!(ds.attr_set.load(std::memory_order_relaxed) & bit)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return e;
        ds.attr_set.fetch_or(bit, std::memory_order_relaxed);
    }
    const long long work = (long long)a.gq.nblk * a.B * a.H;
    const int reserve = attn_sm_reserve();
    const int usable = sm_count - reserve > 0 ? sm_count - reserve : 1;
    const int grid = (int)(work < usable ? work : usable);
    kern<<<grid, kThreads, kSmemBytes, st>>>(P);
    return cudaGetLastError();
}

}  // namespace lcbsa
