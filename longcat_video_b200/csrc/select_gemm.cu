// Block-select stage, parts 2 and 3, two-kernel form: block scores as a register-tiled fp32 GEMM, then per-row top-k.
//
// Replaces cal_score + get_select_indices_topk_from_score
// (longcat_video/block_sparse_attention/bsa_interface.py:180-184, 212-224) like select.cu does, with the same
// arithmetic:  score(i,j) = fp32 FMA chain over d = 0..D-1 (ascending), rounded to the input dtype.  The FMA pipe
// can only be kept busy if every operand word read from shared memory feeds several FMAs (shared memory hands a
// warp 32 words per cycle, the FMA pipes take 128 lanes per cycle), and that needs a two-dimensional register
// tile: here 8 x 8 scores per thread, 128 x 128 per CTA, 16 FMAs per 128-bit operand read (4 x 4 or 2 x 2 on small calls).  A tile of that shape
// cannot keep whole rows of scores on chip, so the rounded scores go to a workspace as order-preserving 16-bit keys
// (2 bytes per score, written once and read once: 0.27 GB of traffic at 720p with 32 heads) and a second kernel
// selects per row, one warp per row with the row in registers.  Used by lcbsa_block_select when the caller's
// workspace has room for the keys; otherwise the fused kernel of select.cu runs.
#include "select_common.cuh"

namespace lcbsa {

namespace {

using namespace sel;

constexpr int kGemmThreads = 256;   // 16 x 16 threads, R x R scores each

// q: [BH, Nq, D], k: [BH, Nk, D] pooled rows in the input dtype; keys: [BH, Nq, nk_pad].  R: scores per thread and direction, 8, 4
// or 2 (tiles of 128, 64 or 32 scores; see launch_gemm)
template <typename T, int D, int R>
__global__ void __launch_bounds__(kGemmThreads, 2) score_gemm_kernel(const T* __restrict__ qc, const T* __restrict__ kc, int Nq, int Nk,
                                                                    int nk_pad, uint16_t* __restrict__ keys) {
    constexpr int kTile = 16 * R;              // scores per CTA: kTile x kTile
    constexpr int kBK = 2048 / kTile;          // head-dimension elements per shared-memory slab: a 128-bit load per thread and operand
    constexpr int kPitch = kTile + 4;          // slab row pitch in floats
    constexpr int kG = R == 8 ? 2 : 1;         // groups of neighbouring rows (columns) of a thread, 64 apart
    constexpr int kW = R / kG;                 // rows (columns) per group: 4, 4 or 2
    static_assert(sizeof(T) == 2 && D % kBK == 0, "16-bit inputs, head_dim a multiple of the slab");
    __shared__ __align__(16) float qs[2][kBK][kPitch];  // [slab][d][row]: transposed, so that a thread's rows are contiguous
    __shared__ __align__(16) float ks[2][kBK][kPitch];

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int bh = blockIdx.z;
    const int i0 = blockIdx.y * kTile, j0 = blockIdx.x * kTile;
    const T* qbase = qc + (long long)bh * Nq * D;
    const T* kbase = kc + (long long)bh * Nk * D;

    // global -> registers: a thread brings 8 consecutive d of one row of the Q tile and of the K tile
    constexpr int kPer = kBK / 8;  // threads per row
    const int lrow = tid / kPer, ldh = (tid % kPer) * 8;
    const bool q_ok = i0 + lrow < Nq, k_ok = j0 + lrow < Nk;
    const T* qsrc = qbase + (long long)(q_ok ? i0 + lrow : 0) * D + ldh;
    const T* ksrc = kbase + (long long)(k_ok ? j0 + lrow : 0) * D + ldh;
    uint4 qpre, kpre;
    auto fetch = [&](int slab) {
        qpre = q_ok ? __ldg(reinterpret_cast<const uint4*>(qsrc + slab * kBK)) : make_uint4(0u, 0u, 0u, 0u);
        kpre = k_ok ? __ldg(reinterpret_cast<const uint4*>(ksrc + slab * kBK)) : make_uint4(0u, 0u, 0u, 0u);
    };
    auto stash = [&](int buf) {
        const T* qe = reinterpret_cast<const T*>(&qpre);
        const T* ke = reinterpret_cast<const T*>(&kpre);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            qs[buf][ldh + i][lrow] = DType<T>::to_f32(qe[i]);
            ks[buf][ldh + i][lrow] = DType<T>::to_f32(ke[i]);
        }
    };

    // this thread's scores: rows kW ty .. (and 64 + 4 ty ..), columns kW tx .. (and 64 + 4 tx ..)
    // column pairs: two fused multiply-adds per instruction, each rounded like a scalar one (32 x 1440 x 1440 scores: 476 us with
    // scalar ones, 443 us; 236 us is what the FMA pipes need)
    float2 acc[R][R / 2];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);

    fetch(0);
    stash(0);
    __syncthreads();
    constexpr int kSlabs = D / kBK;
#pragma unroll 1
    for (int slab = 0; slab < kSlabs; ++slab) {
        const int buf = slab & 1;
        if (slab + 1 < kSlabs) fetch(slab + 1);
        // unrolled whole, the loop of the large tile is 36 KB of code and waits for instructions (32 x 1440 x 1440 scores: 26 us of
        // 400; a 16 x 8 tile per thread, with fewer operand reads but half the warps, is 5 to 8 % slower than 8 x 8)
#pragma unroll (32 / R)
        for (int d = 0; d < kBK; ++d) {  // ascending d: every score is one chain acc = fmaf(q[d], k[d], acc)
            float qv[R];
            float2 kv[R / 2];
#pragma unroll
            for (int g = 0; g < kG; ++g) {
                if constexpr (kW == 4) {
                    const float4 q4 = *reinterpret_cast<const float4*>(&qs[buf][d][64 * g + 4 * ty]);
                    const float4 k4 = *reinterpret_cast<const float4*>(&ks[buf][d][64 * g + 4 * tx]);
                    qv[4 * g] = q4.x; qv[4 * g + 1] = q4.y; qv[4 * g + 2] = q4.z; qv[4 * g + 3] = q4.w;
                    kv[2 * g] = make_float2(k4.x, k4.y);
                    kv[2 * g + 1] = make_float2(k4.z, k4.w);
                } else {
                    const float2 q2 = *reinterpret_cast<const float2*>(&qs[buf][d][2 * ty]);
                    qv[0] = q2.x; qv[1] = q2.y;
                    kv[0] = *reinterpret_cast<const float2*>(&ks[buf][d][2 * tx]);
                }
            }
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int j = 0; j < R / 2; ++j) acc[i][j] = __ffma2_rn(make_float2(qv[i], qv[i]), kv[j], acc[i][j]);
        }
        if (slab + 1 < kSlabs) stash(buf ^ 1);
        __syncthreads();
    }

    // rounded scores -> keys; columns past Nk get the smallest key, columns past nk_pad do not exist
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = i0 + 64 * (i / kW) + kW * ty + i % kW;
        if (row >= Nq) continue;
        uint16_t* out = keys + ((long long)bh * Nq + row) * nk_pad;
#pragma unroll
        for (int g = 0; g < kG; ++g) {
            const int col = j0 + 64 * g + kW * tx;
            if (col >= nk_pad) continue;  // nk_pad is a multiple of 64, so a group of columns is all in or all out
            uint32_t kk[kW];
#pragma unroll
            for (int j = 0; j < kW; ++j) {
                const float2 a2 = acc[i][(kW * g + j) >> 1];
                kk[j] = (col + j < Nk) ? (uint32_t)make_key(DType<T>::from_f32((j & 1) ? a2.y : a2.x)) : 0u;
            }
            if constexpr (kW == 4) *reinterpret_cast<uint2*>(out + col) = make_uint2(kk[0] | (kk[1] << 16), kk[2] | (kk[3] << 16));
            else *reinterpret_cast<uint32_t*>(out + col) = kk[0] | (kk[1] << 16);
        }
    }
}

// one warp per row of keys; NW: words a lane keeps (rows of up to 64 * NW keys), 0: a row of any length, counted where it lies
template <int NW>
__global__ void __launch_bounds__(256) topk_rows_kernel(const uint16_t* __restrict__ keys, long long rows, int Nk, int nk_pad, int nsel,
                                                       int cap, uint32_t first_step, int32_t* __restrict__ idx, int32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    if constexpr (NW > 0)
        select_row_regs<NW>(keys + row * nk_pad, Nk, nk_pad, nsel, cap, first_step, idx + row * cap, cnt + row, lane);
    else
        select_row<uint16_t>(keys + row * nk_pad, Nk, nk_pad, nsel, cap, idx + row * cap, cnt + row, lane);
}

// The same for a grid with a "first part" (the conditioning frames of video continuation): query blocks of the first
// part take nsel_first blocks among the key blocks of the first part, all other query blocks nsel blocks among all.
template <int NW>
__global__ void __launch_bounds__(256) topk_rows_split_kernel(const uint16_t* __restrict__ keys, long long rows, int Nq, int Nk, int nk_pad,
                                                             SelectSplit sp, int nsel, int cap, uint32_t first_step,
                                                             int32_t* __restrict__ idx, int32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int qblk = (int)(row % Nq);
    const bool first = ((qblk / sp.hw_q) % sp.period_q) < sp.split_q;
    const KeyMask mask{sp.hw_k, first ? sp.period_k : 0, sp.split_k};
    const int n_keys = first ? Nk / sp.hw_k / sp.period_k * sp.split_k * sp.hw_k : Nk;
    select_row_regs<NW>(keys + row * nk_pad, n_keys, nk_pad, first ? sp.nsel_first : nsel, cap, first_step, idx + row * cap, cnt + row, lane, mask);
}

template <int NW>
cudaError_t launch_topk(const uint16_t* keys, long long rows, int Nq, int Nk, int nk_pad, const SelectSplit* split, int nsel, int cap,
                        uint32_t first_step, int32_t* idx, int32_t* cnt, cudaStream_t st) {
    const unsigned grid = (unsigned)((rows + 7) / 8);
    if constexpr (NW > 0) {
        if (split != nullptr) {
            topk_rows_split_kernel<NW><<<grid, 256, 0, st>>>(keys, rows, Nq, Nk, nk_pad, *split, nsel, cap, first_step, idx, cnt);
            return cudaGetLastError();
        }
    }
    topk_rows_kernel<NW><<<grid, 256, 0, st>>>(keys, rows, Nk, nk_pad, nsel, cap, first_step, idx, cnt);
    return cudaGetLastError();
}

// The narrowest register row that holds nk_pad keys, in steps of 128 keys: the work of a count is proportional to the words a
// lane keeps, and with two words a step no row counts more than one word of padding.  Rows above 64 * kRegWords keys are
// counted where they lie.
template <int NW>
cudaError_t launch_topk_for(const uint16_t* keys, long long rows, int Nq, int Nk, int nk_pad, const SelectSplit* split, int nsel, int cap,
                            uint32_t first_step, int32_t* idx, int32_t* cnt, cudaStream_t st) {
    if constexpr (NW <= kRegWords) {
        if (nk_pad <= 64 * NW) return launch_topk<NW>(keys, rows, Nq, Nk, nk_pad, split, nsel, cap, first_step, idx, cnt, st);
        return launch_topk_for<NW + 2>(keys, rows, Nq, Nk, nk_pad, split, nsel, cap, first_step, idx, cnt, st);
    } else {
        return launch_topk<0>(keys, rows, Nq, Nk, nk_pad, nullptr, nsel, cap, first_step, idx, cnt, st);
    }
}

template <typename T, int D>
cudaError_t launch_gemm(const void* qc, const void* kc, int BH, int Nq, int Nk, int nk_pad, uint16_t* keys, cudaStream_t st) {
    auto tiles = [&](int t) { return (long long)((nk_pad + t - 1) / t) * ((Nq + t - 1) / t) * BH; };
    auto run = [&](auto kern, int t) {
        const dim3 grid((nk_pad + t - 1) / t, (Nq + t - 1) / t, BH);
        kern<<<grid, kGemmThreads, 0, st>>>(reinterpret_cast<const T*>(qc), reinterpret_cast<const T*>(kc), Nq, Nk, nk_pad, keys);
        return cudaGetLastError();
    };
    // A tile of 128 takes 9 us whatever is in it, so small calls take small tiles as long as those fit the chip in two (32) or three
    // (64) waves of one per SM; operand reads per multiply-add double from one size to the next.  Scores and selection, us, tiles of
    // 128 / 64 / 32:  2 x 12 x 12 scores 15.9 / 8.7 / 5.8;  1 x 312 x 312 (100 tiles of 32) 21.3 / 11.0 / 7.6;  1 x 624 x 624
    // (400 tiles of 32) 23.0 / 12.4 / 14.9;  4 x 624 x 624 (400 tiles of 64) 25.2 / 24.2 / 38.8;  1 x 1440 x 1440 (529) 28.8 / 32.6 / 50.8.
    constexpr long long kSms = 148;
    if (tiles(32) <= 2 * kSms) return run(score_gemm_kernel<T, D, 2>, 32);
    if (tiles(64) <= 3 * kSms) return run(score_gemm_kernel<T, D, 4>, 64);
    return run(score_gemm_kernel<T, D, 8>, 128);
}

}  // namespace

size_t score_keys_bytes(int dtype, int BH, int Nq, int Nk, int D) {
    if (dtype == LCBSA_FP32 || (D != 64 && D != 128) || BH > 65535) return 0;  // this form does not apply
    const size_t nk_pad = ((size_t)Nk + 63) / 64 * 64;
    return (size_t)BH * Nq * nk_pad * sizeof(uint16_t);
}

// scores only: the 16-bit keys of all [BH, Nq, Nk] scores into keys_ws (score_keys_bytes(...) bytes)
cudaError_t launch_score_keys(int dtype, const void* qc, const void* kc, int BH, int Nq, int Nk, int D, void* keys_ws, cudaStream_t st,
                              const char** why) {
    if (BH == 0 || Nq == 0) return cudaSuccess;
    if (score_keys_bytes(dtype, BH, Nq, Nk, D) == 0) {
        *why = "the score kernel takes bf16 or fp16 with head_dim 64 or 128";
        return cudaErrorInvalidValue;
    }
    const int nk_pad = (Nk + 63) / 64 * 64;
    uint16_t* keys = static_cast<uint16_t*>(keys_ws);
    if (dtype == LCBSA_BF16)
        return D == 128 ? launch_gemm<__nv_bfloat16, 128>(qc, kc, BH, Nq, Nk, nk_pad, keys, st)
                        : launch_gemm<__nv_bfloat16, 64>(qc, kc, BH, Nq, Nk, nk_pad, keys, st);
    return D == 128 ? launch_gemm<__half, 128>(qc, kc, BH, Nq, Nk, nk_pad, keys, st) : launch_gemm<__half, 64>(qc, kc, BH, Nq, Nk, nk_pad, keys, st);
}

cudaError_t launch_score_gemm_topk(int dtype, const void* qc, const void* kc, int BH, int Nq, int Nk, int D, int nsel, int cap,
                                   int32_t* idx, int32_t* cnt, void* keys_ws, cudaStream_t st, const char** why, const SelectSplit* split) {
    if (BH == 0 || Nq == 0) return cudaSuccess;
    if (score_keys_bytes(dtype, BH, Nq, Nk, D) == 0) {
        *why = "the two-kernel form takes bf16 or fp16 with head_dim 64 or 128";
        return cudaErrorInvalidValue;
    }
    const int nk_pad = (Nk + 63) / 64 * 64;
    uint16_t* keys = static_cast<uint16_t*>(keys_ws);
    cudaError_t e;
    if (dtype == LCBSA_BF16)
        e = D == 128 ? launch_gemm<__nv_bfloat16, 128>(qc, kc, BH, Nq, Nk, nk_pad, keys, st)
                     : launch_gemm<__nv_bfloat16, 64>(qc, kc, BH, Nq, Nk, nk_pad, keys, st);
    else
        e = D == 128 ? launch_gemm<__half, 128>(qc, kc, BH, Nq, Nk, nk_pad, keys, st) : launch_gemm<__half, 64>(qc, kc, BH, Nq, Nk, nk_pad, keys, st);
    if (e != cudaSuccess) return e;
    const long long rows = (long long)BH * Nq;
    if (split != nullptr && nk_pad > 64 * kRegWords) {
        *why = "the split selection handles up to 1536 key blocks";
        return cudaErrorInvalidValue;
    }
    const uint32_t first_step = dtype == LCBSA_BF16 ? FirstStep<__nv_bfloat16>::value : FirstStep<__half>::value;
    return launch_topk_for<2>(keys, rows, Nq, Nk, nk_pad, split, nsel, cap, first_step, idx, cnt, st);
}

}  // namespace lcbsa
