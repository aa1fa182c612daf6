// The step immediately before the BSA path: RMSNorm (fp32) of q and k over the head dimension, times the learned
// weight, then the 3-D rotary embedding, written straight into the [B, H, S, D] layout the attention (or the Ulysses
// exchange) reads.
//
// Replaces, for q and k each (longcat_video/modules/attention.py:113-121):
//   RMSNorm_FP32.forward   (longcat_video/modules/blocks.py:42-53)
//   RotaryPositionalEmbedding.forward   (longcat_video/modules/rope_3d.py:99-120)
// which in the reference are six elementwise passes over q and k with fp32 temporaries.  Here it is one pass:
// every input element is read once from the strided view of the fused qkv projection and every output element
// written once.  HBM-bound: 2 bytes in + 2 bytes out per element.
//
// Eight lanes per token: a lane owns D/8 consecutive elements (whole rotation pairs, two 16-byte loads at
// head_dim 128), a warp works on four neighbouring tokens and walks over a group of heads, so that the position
// arithmetic, the angles and the weights are set up once and stay in registers, and every warp instruction of the
// row arithmetic serves four rows (the kernel is bound by instruction issue as much as by HBM: at the HBM rate an
// SM has about 90 issue slots per 256-byte row).
// Arithmetic, in the order the CPU oracle fixes it: per-lane sum of squares with fmaf in ascending order, butterfly
// over the 8 lanes (xor 4, 2, 1), mean = sum / D, 1 / sqrtf(mean + eps) correctly rounded, y = T(x * r),
// z = T(y * w) (one packed multiply in the storage type: the product of two 8- or 11-bit significands is exact in
// fp32, so rounding it once is the same thing), out = T(z * cos + rot(z) * sin) with the two products rounded
// separately.
//
// The rotary angles depend on t for the first D - 4*(D/6) elements of the head dimension, on h for the next
// 2*(D/6) and on w for the last 2*(D/6) (rope_3d.py:62-84), so the [S, D] cos/sin tables of the reference factor
// into three small ones, [T, dt], [H, dh], [W, dw]; both elements of a pair have the same angle (rope_3d.py:113-115).
//
// A launch works on up to kMaxRowJobs tensors at once: all that a layer does to its q, k, v rows before the attention
// (normalise, embed, also keep the normalised k, copy v into or behind the cache).  The copies ran as library copies of
// strided views, two bytes per thread and step: 480p grid, 32 heads, bf16, the clone of v took 361 us and v behind its cache
// 376 us; as jobs they take 118 and 105 us, at the rate of the other rows.
#include "common.cuh"

namespace lcbsa {

namespace {

constexpr int kWarps = 8;         // warps per CTA, four tokens each
constexpr int kTokens = 4;        // tokens per warp: eight lanes each
constexpr int kHeadsPerCta = 16;  // heads one warp walks over, at most

// Two values of the storage type in one 32-bit word: rounding two floats costs one packed conversion.
template <typename T>
struct Pair;
template <>
struct Pair<__nv_bfloat16> {
    __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&t);
    }
    __device__ static __forceinline__ void unpack(uint32_t u, float& lo, float& hi) {
        lo = __uint_as_float(u << 16);
        hi = __uint_as_float(u & 0xffff0000u);
    }
    __device__ static __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {  // round(a * b) per half, one rounding
        const __nv_bfloat162 t = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&t);
    }
};
template <>
struct Pair<__half> {
    __device__ static __forceinline__ uint32_t pack(float lo, float hi) {
        const __half2 t = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&t);
    }
    __device__ static __forceinline__ void unpack(uint32_t u, float& lo, float& hi) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u));
        lo = f.x;
        hi = f.y;
    }
    __device__ static __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
        const __half2 t = __hmul2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const uint32_t*>(&t);
    }
};

// NORM: RMSNorm times weight (off: the input is already normalised, e.g. cached keys); ROPE: the rotary embedding
// (off: normalised q / k as they are cached before the embedding, attention.py:118-119).  The token at grid position
// (t, h, w) takes the angles of frame t + t_off; tab_t is the number of frames the table holds (>= T + t_off).
// Neither: the rows are copied.  KEEP: the normalised row also goes to out2.
template <typename T, int D, bool NORM, bool ROPE, bool KEEP>
__device__ __forceinline__ void do_rows(const RowJob& j, unsigned s_blk, int b, int h0, int h1, float eps) {
    const View& x = j.x;
    const int S = j.S, tab_t = j.tab_t, Hg = j.Hg, Wg = j.Wg;
    const T* __restrict__ weight = static_cast<const T*>(j.weight);
    const float* __restrict__ tab = j.tab;
    constexpr int PER = D / 8;   // elements per lane: 16 or 8
    constexpr int NV = PER / 8;  // 16-byte vectors per lane
    constexpr int NP = PER / 2;  // rotation pairs per lane
    static_assert(PER == 8 || PER == 16, "a lane owns one or two 16-byte vectors");
    constexpr int DH = 2 * (D / 6), DW = DH, DT = D - DH - DW;
    const int lane = threadIdx.x & 31, sub = lane & 7, tok = lane >> 3;
    const long long first = ((long long)s_blk * kWarps + (threadIdx.x >> 5)) * kTokens;  // the warp's first token
    if (first >= S) return;
    const bool live = first + tok < S;  // the last warp may have fewer than four tokens
    const int s = live ? (int)(first + tok) : S - 1;
    const int w_pos = s % Wg, h_pos = (s / Wg) % Hg, t_pos = s / (Wg * Hg) + j.t_off;

    // table layout: cos_t [T, DT] sin_t [T, DT] cos_h [H, DH] sin_h [H, DH] cos_w [W, DW] sin_w [W, DW]
    const float* cos_t = tab;
    const float* sin_t = cos_t + (long long)tab_t * DT;
    const float* cos_h = sin_t + (long long)tab_t * DT;
    const float* sin_h = cos_h + (long long)Hg * DH;
    const float* cos_w = sin_h + (long long)Hg * DH;
    const float* sin_w = cos_w + (long long)Wg * DW;
    float cs[NP], sn[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int d = sub * PER + 2 * p;  // even: d and d + 1 are one rotation pair and lie in the same part
        const float *c, *n;
        if (d < DT) {
            c = cos_t + t_pos * DT + d; n = sin_t + t_pos * DT + d;
        } else if (d < DT + DH) {
            c = cos_h + h_pos * DH + (d - DT); n = sin_h + h_pos * DH + (d - DT);
        } else {
            c = cos_w + w_pos * DW + (d - DT - DH); n = sin_w + w_pos * DW + (d - DT - DH);
        }
        cs[p] = ROPE ? __ldg(c) : 1.0f;
        sn[p] = ROPE ? __ldg(n) : 0.0f;
    }
    uint4 wv[NV];  // the lane's weights, packed as they are stored
#pragma unroll
    for (int i = 0; i < NV; ++i) wv[i] = NORM ? __ldg(reinterpret_cast<const uint4*>(weight + sub * PER) + i) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t* wp = reinterpret_cast<const uint32_t*>(wv);

    const T* sp = reinterpret_cast<const T*>(x.data) + (long long)b * x.sb + (long long)s * x.ss + (long long)h0 * x.sh + sub * PER;
    T* dp = static_cast<T*>(j.out) + (long long)b * j.osb + (long long)s * j.oss + (long long)h0 * j.osh + sub * PER;
    T* dp2 = KEEP ? static_cast<T*>(j.out2) + (long long)b * j.o2sb + (long long)s * j.o2ss + (long long)h0 * j.o2sh + sub * PER : nullptr;
    uint4 cur[NV], nxt[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) cur[i] = reinterpret_cast<const uint4*>(sp)[i];
#pragma unroll 1
    for (int h = h0; h < h1; ++h) {
        sp += x.sh;
        if (h + 1 < h1) {  // the next head's row is in flight during the arithmetic
#pragma unroll
            for (int i = 0; i < NV; ++i) nxt[i] = reinterpret_cast<const uint4*>(sp)[i];
        }
        const uint32_t* cw = reinterpret_cast<const uint32_t*>(cur);
        float rinv = 1.0f;
        if (NORM) {
            float v[PER];
#pragma unroll
            for (int p = 0; p < NP; ++p) Pair<T>::unpack(cw[p], v[2 * p], v[2 * p + 1]);
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < PER; ++i) ss = fmaf(v[i], v[i], ss);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
            const float mean = __fmul_rn(ss, 1.0f / (float)D);
            rinv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
        }
        uint4 res[NV];
        uint32_t* rw = reinterpret_cast<uint32_t*>(res);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            uint32_t rn[4];
#pragma unroll
            for (int p4 = 0; p4 < 4; ++p4) {
                const int p = 4 * i + p4;
                uint32_t z = cw[p];
                if (NORM) {
                    float v0, v1;
                    Pair<T>::unpack(cw[p], v0, v1);
                    z = Pair<T>::mul(Pair<T>::pack(__fmul_rn(v0, rinv), __fmul_rn(v1, rinv)), wp[p]);
                }
                rn[p4] = z;
                if (ROPE) {
                    float z0, z1;
                    Pair<T>::unpack(z, z0, z1);
                    z = Pair<T>::pack(__fadd_rn(__fmul_rn(z0, cs[p]), __fmul_rn(-z1, sn[p])),
                                      __fadd_rn(__fmul_rn(z1, cs[p]), __fmul_rn(z0, sn[p])));
                }
                rw[p] = z;
            }
            if (KEEP && live) reinterpret_cast<uint4*>(dp2)[i] = make_uint4(rn[0], rn[1], rn[2], rn[3]);
        }
        if (live) {
#pragma unroll
            for (int i = 0; i < NV; ++i) reinterpret_cast<uint4*>(dp)[i] = res[i];
        }
        if (KEEP) dp2 += j.o2sh;
        dp += j.osh;
#pragma unroll
        for (int i = 0; i < NV; ++i) cur[i] = nxt[i];
    }
}

// One CTA: 32 tokens and up to `hpc` heads of one batch entry of one job.  The jobs' CTAs follow each other in the grid.
// kKind: what the only job of the launch does (kCopy ..), or kMixed: any number of jobs of any kind.
enum { kCopy, kRope, kNorm, kNormRope, kNormRopeKeep, kMixed };

__host__ __device__ __forceinline__ int kind_of(const RowJob& j) {
    if (j.weight != nullptr && j.tab != nullptr) return j.out2 != nullptr ? kNormRopeKeep : kNormRope;
    return j.weight != nullptr ? kNorm : j.tab != nullptr ? kRope : kCopy;
}

// CTAs per SM that a kernel's registers have to allow: memory bound, so as many as fit without spilling in the loop.  A uniform 4, with the
// CTA's place worked out from a one-dimensional grid in every kind: 24x48x80 grid, 32 heads, bf16, RMSNorm and embedding 262 us,
// RMSNorm alone 248, embedding alone 252 (head_dim 64: 154); as here 258, 242, 244 (141).
constexpr int min_ctas(int D, int kind) {
    return kind == kCopy ? 8 : kind == kRope ? (D == 128 ? 5 : 8) : kind == kNorm ? (D == 128 ? 5 : 6) : (D == 128 ? 4 : 5);
}

template <typename T, int D, int kKind>
__global__ void __launch_bounds__(kWarps * 32, min_ctas(D, kKind)) norm_rope_kernel(const __grid_constant__ RowJobs P) {
    int i = 0;
    unsigned s_blk = blockIdx.x, hg = blockIdx.y, b = blockIdx.z;
    if (kKind == kMixed) {
        while (i + 1 < P.n && blockIdx.x >= P.job[i + 1].first) ++i;
        const unsigned r = blockIdx.x - P.job[i].first, s_blks = (unsigned)(P.job[i].S + kTokens * kWarps - 1) / (kTokens * kWarps);
        s_blk = r % s_blks;
        hg = r / s_blks % P.head_groups;
        b = r / s_blks / P.head_groups;
    }
    const RowJob& j = P.job[kKind == kMixed ? i : 0];
    const int h0 = (int)hg * P.hpc, h1 = min(P.H, h0 + P.hpc);
    const int kind = kKind == kMixed ? kind_of(j) : kKind;
    if (kind == kNormRopeKeep) do_rows<T, D, true, true, true>(j, s_blk, (int)b, h0, h1, P.eps);
    else if (kind == kNormRope) do_rows<T, D, true, true, false>(j, s_blk, (int)b, h0, h1, P.eps);
    else if (kind == kNorm) do_rows<T, D, true, false, false>(j, s_blk, (int)b, h0, h1, P.eps);
    else if (kind == kRope) do_rows<T, D, false, true, false>(j, s_blk, (int)b, h0, h1, P.eps);
    else do_rows<T, D, false, false, false>(j, s_blk, (int)b, h0, h1, P.eps);
}

template <typename T, int D>
cudaError_t launch(RowJobs& P, int kind, int B, cudaStream_t st) {
    long long total = 0;
    P.head_groups = (unsigned)((P.H + P.hpc - 1) / P.hpc);
    for (int i = 0; i < P.n; ++i) {
        P.job[i].first = (unsigned)total;
        total += (long long)((P.job[i].S + kTokens * kWarps - 1) / (kTokens * kWarps)) * P.head_groups * B;
    }
    if (total == 0) return cudaSuccess;
    if (kind == kMixed ? total > 0x7fffffffll : P.head_groups > 65535u) return cudaErrorInvalidConfiguration;
    const dim3 grid = kind == kMixed ? dim3((unsigned)total) : dim3((unsigned)(total / P.head_groups / B), P.head_groups, (unsigned)B);
    switch (kind) {
        case kCopy: norm_rope_kernel<T, D, kCopy><<<grid, kWarps * 32, 0, st>>>(P); break;
        case kRope: norm_rope_kernel<T, D, kRope><<<grid, kWarps * 32, 0, st>>>(P); break;
        case kNorm: norm_rope_kernel<T, D, kNorm><<<grid, kWarps * 32, 0, st>>>(P); break;
        case kNormRope: norm_rope_kernel<T, D, kNormRope><<<grid, kWarps * 32, 0, st>>>(P); break;
        case kNormRopeKeep: norm_rope_kernel<T, D, kNormRopeKeep><<<grid, kWarps * 32, 0, st>>>(P); break;
        default: norm_rope_kernel<T, D, kMixed><<<grid, kWarps * 32, 0, st>>>(P); break;
    }
    return cudaGetLastError();
}

template <typename T, int D>
cudaError_t run(RowJobs& P, int B, cudaStream_t st) {
    // A warp takes up to 16 heads, which spreads its set-up (position, angles, weights) over that many rows; small calls take
    // fewer, so that there are some eight CTAs per SM: the heads of a warp are a serial chain of loads.
    long long tokens = 0;
    for (int i = 0; i < P.n; ++i) tokens += (P.job[i].S + kTokens * kWarps - 1) / (kTokens * kWarps);
    P.hpc = kHeadsPerCta;
    while (P.hpc > 2 && tokens * B * ((P.H + P.hpc - 1) / P.hpc) < 148 * 8) P.hpc /= 2;
    // Calls that do not fill the chip are bound by their launches: all jobs in one.  Larger ones take a launch per job, whose
    // kernel has the registers and the code of its kind alone: q and k of a 24x48x80 grid, 32 heads: 509 us in two launches, 582 us
    // through the kernel that serves all kinds.
    if (P.n > 1 && tokens * B * ((P.H + P.hpc - 1) / P.hpc) < 148 * 16) return launch<T, D>(P, kMixed, B, st);
    for (int i = 0; i < P.n; ++i) {
        RowJobs one = P;
        one.job[0] = P.job[i];
        one.n = 1;
        cudaError_t e = launch<T, D>(one, kind_of(one.job[0]), B, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

size_t rope_table_floats(int Tg, int Hg, int Wg, int D) {
    const int dh = 2 * (D / 6), dt = D - 2 * dh;
    return 2 * ((size_t)Tg * dt + (size_t)Hg * dh + (size_t)Wg * dh);
}

cudaError_t launch_norm_rope(int dtype, RowJobs& jobs, int B, int D, cudaStream_t st, const char** why) {
    if (dtype == LCBSA_FP32 || (D != 64 && D != 128)) {
        *why = "norm_rope takes bf16 or fp16 with head_dim 64 or 128";
        return cudaErrorInvalidValue;
    }
    if (B > 65535) {
        *why = "norm_rope: batch above 65535";
        return cudaErrorInvalidValue;
    }
    if (B == 0 || jobs.H == 0) return cudaSuccess;
    if (dtype == LCBSA_BF16) return D == 128 ? run<__nv_bfloat16, 128>(jobs, B, st) : run<__nv_bfloat16, 64>(jobs, B, st);
    return D == 128 ? run<__half, 128>(jobs, B, st) : run<__half, 64>(jobs, B, st);
}

}  // namespace lcbsa
