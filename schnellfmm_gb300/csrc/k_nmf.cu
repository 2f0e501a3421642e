// NMF imputation (src/nmf.rs:80-455, src/parallel.rs:219-321,
// src/testing.rs:423-487) on the resident genotypes.
//
// The dense products of the multiplicative updates and of the imputed passes
// run through the ordinary contractions with missing calls as 0; the values
// NMF puts at the missing calls, f_ir = W_i . H_r, enter as sparse
// corrections over the missing-call lists (CSR by SNP, CSC by sample), so no
// imputed copy of the matrix is ever formed.  W (n x k) and H (p x k, one row
// per SNP) are FP32 row-major here; k <= kMaxNmfK (kernels are built for
// rank bounds 16 and 32).
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "chacha8.cuh"
#include "slfmm_internal.h"
#include "stats_common.cuh"

namespace slfmm {
namespace {

constexpr uint64_t kGamma = 0x9E3779B97F4A7C15ull;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Draw `ctr` of the counter stream keyed by mix64(seed + gamma) is the
// uniform (m >> 11) 2^-53; it is below `rate` iff (m >> 11) < ceil(rate 2^53)
// -- compared as integers, without forming the FP64 uniform
__device__ __forceinline__ bool draw_below(uint64_t key, uint64_t ctr, uint64_t thresh) {
    return (mix64(key + (ctr + 1) * kGamma) >> 11) < thresh;
}

// The reference's mask stream (src/nmf.rs:433-434, src/testing.rs:437-438) is
// ChaCha8Draws (chacha8.cuh) sampled by Uniform(0, 1): the uniform of an output
// is (u64 >> 12) 2^-52, below `rate` iff (u64 >> 12) < ceil(rate 2^52).

__device__ __forceinline__ uint32_t code_at(const uint8_t* row, uint64_t s) {
    return (row[s >> 2] >> ((s & 3) * 2)) & 3u;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// f = W_i . h (h in shared memory, k <= KM)
template <int KM>
__device__ __forceinline__ float fill_dot(const float* __restrict__ Wi, const float* h, int k) {
    float f = 0.f;
#pragma unroll
    for (int c = 0; c < KM; ++c)
        if (c < k) f = fmaf(Wi[c], h[c], f);
    return f;
}

// Per-SNP statistics with the NMF values at the missing calls: every call is
// valid, mu = (S1 + F1) / n, s = scale(mu), TSS = s^2 (S2 + F2 - (S1+F1)^2/n)
// (decode_single_snp with a fill, src/bed.rs:300-379).  One warp per SNP.
template <int KM>
__global__ void __launch_bounds__(256) k_fill_stats(uint64_t p, uint64_t n, int norm, const int32_t* __restrict__ counts,
                                                    const uint64_t* __restrict__ ptr, const uint32_t* __restrict__ idx,
                                                    const float* __restrict__ W, const float* __restrict__ H, int k,
                                                    double* __restrict__ mean, double* __restrict__ scale,
                                                    double* __restrict__ tss, uint8_t* __restrict__ zero_var) {
    dependent_wait();
    __shared__ float hs[8][KM];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * 8;
    for (uint64_t r = (uint64_t)blockIdx.x * 8 + wl; r < p; r += nw) {
        __syncwarp();
        if (lane < k) hs[wl][lane] = H[r * k + lane];
        __syncwarp();
        double f1 = 0.0, f2 = 0.0;
        for (uint64_t e = ptr[r] + lane; e < ptr[r + 1]; e += 32) {
            const float f = fill_dot<KM>(W + (uint64_t)idx[e] * k, hs[wl], k);
            f1 += (double)f;
            f2 += (double)f * (double)f;
        }
        f1 = warp_sum_d(f1);
        f2 = warp_sum_d(f2);
        if (lane == 0) {
            const int64_t c1 = counts[r * 4 + 1], c2 = counts[r * 4 + 2];
            const double s1 = (double)(c1 + 2 * c2) + f1, s2 = (double)(c1 + 4 * c2) + f2;
            const double mu = n > 0 ? s1 / (double)n : 0.0;
            const double sc = scale_from_mean(mu, norm);
            const double css = n > 0 ? fmax(s2 - s1 * s1 / (double)n, 0.0) : 0.0;
            mean[r] = mu;
            scale[r] = sc;
            tss[r] = sc * sc * css;
            zero_var[r] = (sc == 0.0 || !(css > 0.0)) ? 1 : 0;
        }
    }
}

// One round of a correction: add d_t * op[row_t, c] over the round's `cnt`
// (row, d) pairs held by lanes 0..cnt-1.  For operands of width w <= CG
// (CG = 8, 16, 32) the warp splits into 32/CG groups that take different
// entries (lane = group * CG + column); CG = 0 is the wide form (one entry per
// step, columns lane + 32 q, w <= 128).  Steps are unrolled so several
// gathers are in flight.
template <int CG>
__device__ __forceinline__ void round_accum(float (&acc)[4], uint32_t my, float dm, int cnt, const float* __restrict__ op,
                                            int ldop, int w, int lane) {
    if constexpr (CG == 0) {
#pragma unroll 4
        for (int t = 0; t < 32; ++t) {
            if (t >= cnt) break;
            const uint64_t r = __shfl_sync(0xffffffffu, my, t);
            const float d = __shfl_sync(0xffffffffu, dm, t);
            const float* row = op + r * ldop;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (lane + 32 * q < w) acc[q] = fmaf(d, row[lane + 32 * q], acc[q]);
        }
    } else {
        constexpr int EPI = 32 / CG;
        const int e = lane / CG, c = lane % CG;
#pragma unroll 4
        for (int t = 0; t < 32; t += EPI) {
            if (t >= cnt) break;
            const int te = t + e;
            const uint64_t r = __shfl_sync(0xffffffffu, my, te & 31);
            const float d = __shfl_sync(0xffffffffu, dm, te & 31);
            if (te < cnt && c < w) acc[0] = fmaf(d, op[r * ldop + c], acc[0]);
        }
    }
}

// after the rounds: column c's total in lane c (narrow form) / lane + 32 q (wide)
template <int CG>
__device__ __forceinline__ void round_finish(float (&acc)[4]) {
    if constexpr (CG != 0) {
#pragma unroll
        for (int off = CG; off < 32; off <<= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    }
}

// f = row . h (h in shared memory) as fill_dot, the row read in vectors of VW
// floats (k % VW == 0, rows aligned to them).  The gathers are bound by the L1's
// look-ups, one per vector: 32 bytes at a time, the most a load takes, a rank of 8
// costs one instead of two (317 -> 265 us a column pass of 8 columns over 21 million
// calls, 207 -> 192 us a row pass).
template <int VW, int KM>
__device__ __forceinline__ float fill_dot_vec(const float* __restrict__ row, const float* h, int k) {
    if constexpr (VW == 1) {
        return fill_dot<KM>(row, h, k);
    } else {
        float f = 0.f;
#pragma unroll
        for (int c = 0; c < KM; c += VW) {
            if (c < k) {
                float v[VW];
                if constexpr (VW == 8)
                    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                        : "l"(row + c));
                else
                    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(row + c);
#pragma unroll
                for (int i = 0; i < VW; ++i) f = fmaf(v[i], h[c + i], f);
            }
        }
        return f;
    }
}

// Row pass correction: out[r, c] += s_r * sum_{i in miss(r)} (f_ir - mu_r) Wop[i, c]
// (the base pass counted the missing calls at the mean).  One warp per SNP;
// 32 missing indices and their fills are formed per round and broadcast.
template <int CG, int VW, int KM>
__global__ void __launch_bounds__(256) k_fill_row_correct(float* __restrict__ out, int ldo, uint64_t p, int w,
                                                          const uint64_t* __restrict__ ptr,
                                                          const uint32_t* __restrict__ idx, const float* __restrict__ Wop,
                                                          int ldw, const float* __restrict__ Wn,
                                                          const float* __restrict__ H, int k,
                                                          const double* __restrict__ mean,
                                                          const double* __restrict__ scale) {
    dependent_wait();
    __shared__ float hs[8][KM];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * 8;
    for (uint64_t r = (uint64_t)blockIdx.x * 8 + wl; r < p; r += nw) {
        __syncwarp();
        if (lane < k) hs[wl][lane] = H[r * k + lane];
        __syncwarp();
        const uint64_t e0 = ptr[r], e1 = ptr[r + 1];
        if (e0 == e1) continue;
        const float mu = (float)mean[r], sc = (float)scale[r];
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (uint64_t b = e0; b < e1; b += 32) {
            uint32_t my = 0;
            float dm = 0.f;
            if (b + lane < e1) {
                my = idx[b + lane];
                const float f = fill_dot_vec<VW, KM>(Wn + (uint64_t)my * k, hs[wl], k);
                dm = f - mu;
            }
            round_accum<CG>(acc, my, dm, (int)(e1 - b < 32 ? e1 - b : 32), Wop, ldw, w, lane);
        }
        round_finish<CG>(acc);
        float* o = out + r * ldo;
        if constexpr (CG == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (lane + 32 * q < w) o[lane + 32 * q] += sc * acc[q];
        } else {
            if (lane < w) o[lane] += sc * acc[0];
        }
    }
}

// Column pass correction: S[i, c] += sum_{r in miss(i)} s_r (f_ir - mu_r) Qop[r, c].
// Per-sample lists can be long (thousands of calls), so each list is cut into
// segments of kColSeg calls, one warp per (sample, segment), and the segment
// sums are added into S with FP64 atomics.
constexpr uint64_t kColSeg = 1024;
// sm[r] = (s_r, mu_r) in FP32 (the values the correction uses), one 8-byte
// gather per call.
template <int CG, int VW, int KM>
__global__ void __launch_bounds__(256) k_fill_col_correct(double* __restrict__ S, int lds, uint64_t n, int w,
                                                          uint64_t nseg, const uint64_t* __restrict__ cptr,
                                                          const uint32_t* __restrict__ cidx,
                                                          const float* __restrict__ Qop, int ldq,
                                                          const float* __restrict__ Wn, const float* __restrict__ H,
                                                          int k, const float2* __restrict__ sm) {
    dependent_wait();
    __shared__ float ws[8][KM];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * 8;
    for (uint64_t gw = (uint64_t)blockIdx.x * 8 + wl; gw < n * nseg; gw += nw) {
        const uint64_t i = gw / nseg, sg = gw - i * nseg;
        const uint64_t e0 = cptr[i] + sg * kColSeg, e1 = min(cptr[i + 1], e0 + kColSeg);
        if (e0 >= e1) continue;
        __syncwarp();
        if (lane < k) ws[wl][lane] = Wn[i * k + lane];
        __syncwarp();
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (uint64_t b = e0; b < e1; b += 32) {
            uint32_t my = 0;
            float dm = 0.f;
            if (b + lane < e1) {
                my = cidx[b + lane];
                const float f = fill_dot_vec<VW, KM>(H + (uint64_t)my * k, ws[wl], k);
                const float2 smv = sm[my];
                dm = smv.x * (f - smv.y);
            }
            round_accum<CG>(acc, my, dm, (int)(e1 - b < 32 ? e1 - b : 32), Qop, ldq, w, lane);
        }
        round_finish<CG>(acc);
        double* o = S + i * lds;
        if constexpr (CG == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (lane + 32 * q < w) atomicAdd(o + lane + 32 * q, (double)acc[q]);
        } else {
            if (lane < w) atomicAdd(o + lane, (double)acc[0]);
        }
    }
}

// out[r, c] += mu_r cs_c: a centred pass (missing at the mean) turned into the
// raw mean-filled product (MeanRaw, src/parallel.rs:53-71)
__global__ void k_add_mean_colsum(float* __restrict__ out, int ldo, uint64_t p, int w,
                                  const double* __restrict__ mean, const double* __restrict__ cs) {
    dependent_start();
    const uint64_t total = p * (uint64_t)w;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = e / w;
        const int c = (int)(e - r * w);
        out[r * ldo + c] = (float)((double)out[r * ldo + c] + mean[r] * cs[c]);
    }
}

// Multiplicative update (src/nmf.rs:150-230): X <- X num / denom where
// denom > eps, then X <- max(X, eps).  X, denom: m x k (FP64); num: ld ldn.
template <typename TN>
__global__ void k_nmf_update(double* __restrict__ X, uint64_t m, int k, const TN* __restrict__ num, int ldn,
                             const double* __restrict__ denom, double eps) {
    dependent_start();
    const uint64_t total = m * (uint64_t)k;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = e / k;
        const int c = (int)(e - r * k);
        double x = X[e];
        const double dn = denom[e];
        if (dn > eps) x = x * ((double)num[r * ldn + c] / dn);
        X[e] = fmax(x, eps);
    }
}

// normalize_w (src/nmf.rs:259-271): W[:, j] /= ||W[:, j]||_1 and
// H[:, j] *= ||W[:, j]||_1 for columns whose L1 norm (W >= 0) exceeds eps
__global__ void k_nmf_normalize(double* __restrict__ W, uint64_t n, double* __restrict__ H, uint64_t p, int k,
                                const double* __restrict__ colsum, double eps) {
    dependent_start();
    const uint64_t total = (n + p) * (uint64_t)k;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const int c = (int)(e % k);
        const double cs = colsum[c];
        if (!(cs > eps)) continue;
        if (e < n * (uint64_t)k) W[e] *= 1.0 / cs;
        else H[e - n * (uint64_t)k] *= cs;
    }
}

// X <- |X| (mode 0) or max(X, 0) (mode 1), FP64, with an optional FP32
// source (ld ldsrc) copied into the m x k destination first
template <typename TS>
__global__ void k_nmf_sign(const TS* __restrict__ src, int ldsrc, double* __restrict__ X, uint64_t m, int k,
                           int mode) {
    dependent_start();
    const uint64_t total = m * (uint64_t)k;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = e / k;
        const int c = (int)(e - r * k);
        const double v = (double)src[r * ldsrc + c];
        X[e] = mode == 0 ? fabs(v) : fmax(v, 0.0);
    }
}

// Hold-out draws, eight consecutive counters of a stream at a time: bit j of
// mask8(blk) is set iff draw 8 blk + j is below the rate.  The counter stream
// (draw_below), or with kChaCha one ChaCha8 block, its comparison
// (u64 >> 12) < thresh made on the whole u64.
template <bool kChaCha>
struct HoldDraws {
    ChaCha8Draws cc;
    uint64_t key, thresh;
    bool all;
    __device__ HoldDraws(uint64_t seed, uint64_t t)
        : cc(seed), key(mix64(seed + kGamma)), thresh(kChaCha ? t << 12 : t), all(kChaCha && (t >> 52) != 0) {}
    __device__ __forceinline__ uint32_t mask8(uint64_t blk) {
        uint32_t m = 0;
        if constexpr (kChaCha) {
            cc.blk = blk;
            cc.refill();
#pragma unroll
            for (int j = 0; j < 8; ++j) m |= cc.word(j) < thresh ? 1u << j : 0u;
            if (all) m = 0xffu;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) m |= draw_below(key, 8 * blk + j, thresh) ? 1u << j : 0u;
        }
        return m;
    }
};

// the even bits 0, 2 .. 14 of x as bits 0 .. 7
__device__ __forceinline__ uint32_t even_bits8(uint32_t x) {
    x &= 0x5555u;
    x = (x | (x >> 1)) & 0x3333u;
    x = (x | (x >> 2)) & 0x0f0fu;
    return (x | (x >> 4)) & 0xffu;
}
// bit b: code b of the eight is 01, a missing call
__device__ __forceinline__ uint32_t missing8(uint32_t codes) { return even_bits8(codes & ~(codes >> 1)); }

// Held-out calls are few (1 % by default) and uneven over the lanes, and their
// absolute errors are FP64: warps queue them and take 32 at a time.
struct HeldCounts {
    uint32_t g0 = 0, g1 = 0, g2 = 0;  // held-out calls by genotype
    __device__ __forceinline__ void add(uint32_t code, bool on) {
        g0 += __popc(__ballot_sync(0xffffffffu, on && code == 0u));
        g1 += __popc(__ballot_sync(0xffffffffu, on && code == 2u));
        g2 += __popc(__ballot_sync(0xffffffffu, on && code == 3u));
    }
    __device__ __forceinline__ uint32_t total() const { return g0 + g1 + g2; }
};

// Estimation-phase CV (compute_cv_error_masked, src/nmf.rs:379-455).  Chunk
// `seq` of `chunk` SNPs uses the stream of mask_seed + seq (the counter
// stream, or ChaCha8 with kChaCha); entry (i, r) draws counter
// (r - chunk start) n + i (column-major, missing calls included) and is held
// out iff the draw is below `rate` and the call is observed.  Sums of
// |g - W_i.H_r|, |g - mean_r| and the count, one row of `part` per warp.
//
// Bound by the integer pipe: a ChaCha8 block is 384 additions, exclusive-ors
// and rotations for eight calls.  A lane takes one whole block, whatever the
// alignment of the SNP's first counter to the blocks.  100 000 SNPs x 3 000
// samples, rate 1 %: 1.10 ms with the calls laid out by code words, 0.71 ms so.
template <bool kChaCha, int KM>
__global__ void __launch_bounds__(256) k_nmf_cv(const uint8_t* __restrict__ packed, uint64_t stride, uint64_t n,
                                                uint64_t p, uint64_t chunk, uint64_t mask_seed, uint64_t thresh,
                                                const float* __restrict__ W, const float* __restrict__ H, int k,
                                                const int32_t* __restrict__ counts, double* __restrict__ part) {
    dependent_wait();
    __shared__ float hs[8][KM];
    __shared__ uint32_t queue[8][64];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * 8, first = (uint64_t)blockIdx.x * 8 + wl;
    uint32_t* q = queue[wl];
    const uint64_t nwords = (n + 15) / 16;
    double e1 = 0.0, e2 = 0.0;
    unsigned long long cnt = 0;
    // SNP number j of the warp leaves its held-out counts with lane j mod 32;
    // the means they are compared with are divided out 32 SNPs at a time
    HeldCounts mine;
    uint64_t mine_r = 0;
    auto mean_errors = [&]() {
        if (mine.total()) {
            const int4 cs = *reinterpret_cast<const int4*>(counts + mine_r * 4);
            const int64_t nobs = (int64_t)cs.x + cs.y + cs.z;
            const double cm = (double)((int64_t)cs.y + 2 * (int64_t)cs.z) / (double)nobs;
            e2 += (double)mine.g0 * fabs(0.0 - cm) + (double)mine.g1 * fabs(1.0 - cm) + (double)mine.g2 * fabs(2.0 - cm);
        }
        mine = HeldCounts();
    };
    int turn = 0;
    for (uint64_t r = first; r < p; r += nw, turn = (turn + 1) & 31) {
        __syncwarp();
        if (lane < k) hs[wl][lane] = H[r * k + lane];
        __syncwarp();
        const uint64_t seq = r / chunk, e0 = (r - seq * chunk) * n;
        HoldDraws<kChaCha> draws(mask_seed + seq, thresh);
        const uint8_t* rowb = packed + r * stride;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(rowb);
        HeldCounts held_here;
        int queued = 0;
        auto take = [&](int m) {
            uint32_t code = 0;
            if (lane < m) {
                const uint64_t i = q[lane];
                code = code_at(rowb, i);
                const double g = code == 0 ? 0.0 : (double)(code - 1);
                e1 += fabs(g - (double)fill_dot<KM>(W + i * k, hs[wl], k));
            }
            held_here.add(code, lane < m);
        };
        const uint64_t b1 = (e0 + n + 7) >> 3;
        for (uint64_t bb = e0 >> 3; bb < b1; bb += 32) {
            // the block's calls i0 .. i0 + 7 of the SNP (i0 may be below 0)
            const int64_t i0 = (int64_t)(8 * (bb + lane)) - (int64_t)e0;
            const int64_t wd = i0 >> 4;
            uint32_t w0 = 0, w1 = 0;
            if (wd >= 0 && wd < (int64_t)nwords) w0 = row[wd];
            if (wd + 1 < (int64_t)nwords) w1 = row[wd + 1];
            const uint32_t codes = __funnelshift_r(w0, w1, 2 * (uint32_t)(i0 & 15));
            const int lo = i0 < 0 ? (int)-i0 : 0;
            const int hi = i0 + 8 <= (int64_t)n ? 8 : i0 < (int64_t)n ? (int)((int64_t)n - i0) : 0;
            uint32_t held = draws.mask8(bb + lane) & ~missing8(codes);
            held &= hi > lo ? (1u << hi) - (1u << lo) : 0u;
            while (const uint32_t any = __ballot_sync(0xffffffffu, held != 0)) {
                if (held) {
                    q[queued + __popc(any & ((1u << lane) - 1))] = (uint32_t)(i0 + __ffs(held) - 1);
                    held &= held - 1;
                }
                queued += __popc(any);
                __syncwarp();
                if (queued >= 32) {
                    take(32);
                    queued -= 32;
                    const uint32_t v = q[32 + lane];
                    __syncwarp();
                    q[lane] = v;
                    __syncwarp();
                }
            }
        }
        take(queued);
        if (lane == turn) {
            mine = held_here;
            mine_r = r;
        }
        cnt += held_here.total();
        if (turn == 31) mean_errors();
    }
    mean_errors();
    e1 = warp_sum_d(e1);
    e2 = warp_sum_d(e2);
    if (lane == 0) {
        part[first * 3] = e1;
        part[first * 3 + 1] = e2;
        part[first * 3 + 2] = (double)cnt;
    }
}

// Observed calls before each SNP within its chunk (the GWAS-phase CV numbers
// its draws by the rank of the observed call in column-major order).  A block
// per chunk, 1 024 SNPs at a time; a thread walking each chunk of 10 000 took
// 1.2 ms.
__global__ void __launch_bounds__(1024) k_obs_base(const int32_t* __restrict__ counts, uint64_t p, uint64_t chunk,
                                                   uint64_t* __restrict__ base) {
    dependent_start();
    __shared__ uint64_t wsum[32];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nchunks = (p + chunk - 1) / chunk;
    for (uint64_t b = blockIdx.x; b < nchunks; b += gridDim.x) {
        uint64_t carry = 0;
        const uint64_t r0 = b * chunk, r1 = chunk < p - r0 ? r0 + chunk : p;
        for (uint64_t s = r0; s < r1; s += 1024) {
            const uint64_t r = s + threadIdx.x;
            uint64_t v = 0;
            if (r < r1) v = (uint64_t)(counts[r * 4] + counts[r * 4 + 1] + counts[r * 4 + 2]);
            uint64_t incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) wsum[wl] = incl;
            __syncthreads();
            uint64_t before = carry;
            for (int w = 0; w < 32; ++w) {
                if (w < wl) before += wsum[w];
                carry += wsum[w];
            }
            if (r < r1) base[r] = before + incl - v;
            __syncthreads();
        }
    }
}

// The hold-out draws of consecutive counters from `before` on, for a warp that
// takes them up to 256 at a time: two runs of 32 blocks, a block per lane, so
// that every block is computed once.
template <bool kChaCha>
struct HeldStream {
    HoldDraws<kChaCha> draws;
    uint64_t before, base;  // next counter; first block of `cur`
    uint32_t cur = 0, nxt = 0;
    int filled = 0;
    __device__ HeldStream(uint64_t seed, uint64_t thresh, uint64_t c0)
        : draws(seed, thresh), before(c0), base(c0 >> 3) {}
    // Bits of the lane's eight calls that are held out: `obs` marks those that
    // draw, lane 0's first, each lane's in order; `before` moves past them.
    __device__ __forceinline__ uint32_t held8(uint32_t obs) {
        const int lane = threadIdx.x & 31;
        const int cnt = __popc(obs);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t rel = (uint32_t)(before - 8 * base);  // below 256
        const uint32_t total = (uint32_t)__shfl_sync(0xffffffffu, incl, 31);
        const int need = rel + total > 256u ? 2 : 1;
        for (; filled < need; ++filled) {
            const uint32_t m = draws.mask8(base + 32 * (uint64_t)filled + lane);
            if (filled == 0) cur = m;
            else nxt = m;
        }
        const uint32_t both = cur | nxt << 8;
        const uint32_t c = rel + (uint32_t)(incl - cnt), o = c >> 3;
        const uint32_t v0 = __shfl_sync(0xffffffffu, both, o & 31), v1 = __shfl_sync(0xffffffffu, both, (o + 1) & 31);
        const uint32_t lo8 = o < 32 ? v0 & 0xffu : v0 >> 8, hi8 = o + 1 < 32 ? v1 & 0xffu : v1 >> 8;
        uint32_t bits = (lo8 | hi8 << 8) >> (c & 7), held = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b)
            if ((obs >> b) & 1u) {
                held |= (bits & 1u) << b;
                bits >>= 1;
            }
        before += total;
        if (rel + total >= 256u) {
            cur = nxt;
            base += 32;
            --filled;
        }
        return held;
    }
};

// acc[c] += row[c] * g, or += row[c], for c < k
template <bool W4, int KM>
__device__ __forceinline__ void load_row(const float* __restrict__ wp, int k, float (&w)[KM]) {
    if constexpr (W4) {
#pragma unroll
        for (int c = 0; c < KM; c += 4)
            if (c < k) {
                const float4 v = *reinterpret_cast<const float4*>(wp + c);
                w[c] = v.x, w[c + 1] = v.y, w[c + 2] = v.z, w[c + 3] = v.w;
            }
    } else {
#pragma unroll
        for (int c = 0; c < KM; ++c)
            if (c < k) w[c] = wp[c];
    }
}

constexpr int kHeldList = 512;

// GWAS-phase CV (src/testing.rs:423-487): per chunk the stream seed + seq,
// one draw per OBSERVED call (counter = its column-major rank in the chunk),
// held out iff the draw is below `rate`; the held-out column is refilled with
// its leave-out mean mu', H = max(0, W+ y~) and the MAE of W_i.H and of mu'
// over the held-out calls accumulate, one row of `part` per warp.  W+ y~ = A +
// mu' B with A = sum over kept observed calls of W+_i g, B = sum over missing
// and held-out calls of W+_i.  One warp per SNP: lane l draws for samples
// i0 + 8 l .. i0 + 8 l + 7 of each 256, and takes i0 + l, i0 + l + 32 .. of
// A and B, so that its W+ rows are read in order.  The held-out calls are
// listed for the errors (kHeldList of them; a SNP with more goes over its
// codes and draws a second time).
//
// Bound by the draws, as k_nmf_cv.  100 000 SNPs x 3 000 samples, rate 1 %:
// 6.96 ms with each block computed four times (for two lanes, in two
// passes) and FP64 counts, 1.97 ms so.
template <bool kChaCha, bool W4, int KM>
__global__ void __launch_bounds__(256) k_nmf_gwas_cv(const uint8_t* __restrict__ packed, uint64_t stride, uint64_t n,
                                                     uint64_t p, uint64_t chunk, uint64_t seed, uint64_t thresh,
                                                     const float* __restrict__ W, const float* __restrict__ Wpt, int k,
                                                     const int32_t* __restrict__ counts,
                                                     const uint64_t* __restrict__ base, double* __restrict__ part) {
    dependent_wait();
    __shared__ float hh[8][KM];
    __shared__ uint32_t list[8][kHeldList];
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const uint64_t nw = (uint64_t)gridDim.x * 8, first = (uint64_t)blockIdx.x * 8 + wl;
    uint32_t* q = list[wl];
    double e1 = 0.0, e2 = 0.0;
    unsigned long long cnt = 0;
    for (uint64_t r = first; r < p; r += nw) {
        const uint64_t seq = r / chunk;
        const uint8_t* row = packed + r * stride;
        float A[KM], B[KM];
#pragma unroll
        for (int c = 0; c < KM; ++c) A[c] = B[c] = 0.f;
        HeldCounts held_here;
        // pass 0 fills A, B and the list; pass 1, only when the list did not
        // hold every held-out call, takes their errors from the draws again
        for (int pass = 0; pass < 2; ++pass) {
            HeldStream<kChaCha> draws(seed + seq, thresh, base[r]);
            uint32_t listed = 0;
            for (uint64_t i0 = 0; i0 < n; i0 += 256) {
                const uint64_t ib = i0 + 8 * (uint64_t)lane;
                uint32_t codes = 0x5555u, obs = 0;  // past n: neither observed nor drawn
                if (ib < n) {
                    codes = *reinterpret_cast<const uint16_t*>(row + ib / 4);
                    obs = 0xffu & ~missing8(codes);
                    if (n - ib < 8) obs &= (1u << (n - ib)) - 1;
                }
                uint32_t held = draws.held8(obs);
                if (pass == 0) {
                    const uint32_t both = codes | held << 16;
#pragma unroll 2
                    for (int j = 0; j < 8; ++j) {
                        const uint64_t i = i0 + 32 * (uint64_t)j + lane;
                        const uint32_t v = __shfl_sync(0xffffffffu, both, 4 * j + (lane >> 3));
                        if (i >= n) continue;
                        const uint32_t code = (v >> (2 * (lane & 7))) & 3u;
                        const bool kept = code != 1u && !((v >> (16 + (lane & 7))) & 1u);
                        float w[KM];
                        load_row<W4, KM>(Wpt + i * k, k, w);
                        const float g = code == 0 ? 0.f : (float)(code - 1);
                        if (kept) {
#pragma unroll
                            for (int c = 0; c < KM; ++c)
                                if (c < k) A[c] = fmaf(w[c], g, A[c]);
                        } else {
#pragma unroll
                            for (int c = 0; c < KM; ++c)
                                if (c < k) B[c] += w[c];
                        }
                    }
                }
                while (const uint32_t any = __ballot_sync(0xffffffffu, held != 0)) {
                    const int b = held ? __ffs(held) - 1 : 0;
                    const uint32_t code = (codes >> (2 * b)) & 3u;
                    const uint32_t at = listed + __popc(any & ((1u << lane) - 1));
                    if (pass == 0) {
                        if (held && at < kHeldList) q[at] = (uint32_t)(ib + b);
                        held_here.add(code, held != 0);
                    } else if (held) {
                        const double g = code == 0 ? 0.0 : (double)(code - 1);
                        e1 += fabs(g - (double)fill_dot<KM>(W + (ib + b) * k, hh[wl], k));
                    }
                    held &= held - 1;
                    listed += __popc(any);
                }
            }
            if (pass == 1 || listed == 0) break;
            const int4 cs = *reinterpret_cast<const int4*>(counts + r * 4);
            const int64_t s1 = (int64_t)cs.y + 2 * (int64_t)cs.z - held_here.g1 - 2 * (int64_t)held_here.g2;
            const int64_t nk = (int64_t)cs.x + cs.y + cs.z - held_here.total();
            const double mu = nk > 0 ? (double)s1 / (double)nk : 0.0;
            __syncwarp();  // the last SNP's errors are done with hh
#pragma unroll
            for (int c = 0; c < KM; ++c) {
                if (c < k) {
                    const float a = warp_sum_f(A[c]), b = warp_sum_f(B[c]);
                    if (lane == 0) hh[wl][c] = fmaxf(a + (float)mu * b, 0.f);
                }
            }
            __syncwarp();
            if (lane < 3)
                e2 += (double)(lane == 0 ? held_here.g0 : lane == 1 ? held_here.g1 : held_here.g2) *
                      fabs((double)lane - mu);
            cnt += listed;
            if (listed > kHeldList) continue;
            for (uint32_t t = lane; t < listed; t += 32) {
                const uint64_t i = q[t];
                const uint32_t code = code_at(row, i);
                const double g = code == 0 ? 0.0 : (double)(code - 1);
                e1 += fabs(g - (double)fill_dot<KM>(W + i * k, hh[wl], k));
            }
            break;
        }
        __syncwarp();
    }
    e1 = warp_sum_d(e1);
    e2 = warp_sum_d(e2);
    if (lane == 0) {
        part[first * 3] = e1;
        part[first * 3 + 1] = e2;
        part[first * 3 + 2] = (double)cnt;
    }
}

}  // namespace

// ceil(rate 2^bits): u < rate for u = m 2^-bits iff m < this (bits = 53 for
// the counter stream's uniforms, 52 for the ChaCha8 stream's)
static uint64_t rate_threshold(double rate, int bits = 53) {
    if (!(rate > 0.0)) return 0;
    if (rate >= 1.0) return 1ull << bits;
    return (uint64_t)std::ceil(std::ldexp(rate, bits));
}

void launch_fill_stats(Ctx& c, const Geno& g, int norm, const float* W, const float* H, int k, double* mean,
                       double* scale, double* tss, uint8_t* zero_var) {
    if (!g.p) return;
    SLFMM_REQUIRE(k >= 1 && k <= kMaxNmfK, SLFMM_ERR_BAD_ARG, "NMF rank must be in 1.." + std::to_string(kMaxNmfK));
    if (k <= 16)
        launch_next(c, k_fill_stats<16>, grid_for(c, g.p, 8), 256, 0, g.p, g.n, norm, g.counts.get(), g.miss_ptr.get(),
                                                                     g.miss_idx.get(), W, H, k, mean, scale, tss,
                                                                     zero_var);
    else
        launch_next(c, k_fill_stats<32>, grid_for(c, g.p, 8), 256, 0, g.p, g.n, norm, g.counts.get(), g.miss_ptr.get(),
                                                                     g.miss_idx.get(), W, H, k, mean, scale, tss,
                                                                     zero_var);
    SLFMM_LAUNCHED(c, "k_fill_stats");
}

// narrow operand group size: the smallest of 8, 16, 32 that holds w, else 0
static int narrow_group(int w) { return w <= 8 ? 8 : w <= 16 ? 16 : w <= 32 ? 32 : 0; }

// fn(vector width, rank bound) for rows of rank k at `rows`: the widest loads up to
// `widest` that k and the rows' alignment allow
template <class F>
static void with_rows(const float* rows, int k, int widest, F&& fn) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(rows);
    auto ranks = [&](auto vw) {
        if (k <= 16) fn(vw, std::integral_constant<int, 16>{});
        else fn(vw, std::integral_constant<int, 32>{});
    };
    if (widest >= 8 && k % 8 == 0 && at % 32 == 0) ranks(std::integral_constant<int, 8>{});
    else if (k % 4 == 0 && at % 16 == 0) ranks(std::integral_constant<int, 4>{});
    else ranks(std::integral_constant<int, 1>{});
}

template <int VW, int KM>
static void fill_row_correct_launch(Ctx& c, const Geno& g, unsigned grid, float* out, int ldo, int w,
                                    const float* Wop, int ldw, const float* Wn, const float* H, int k,
                                    const double* mean, const double* scale) {
    const uint64_t* mp = g.miss_ptr.get();
    const uint32_t* mi = g.miss_idx.get();
    switch (narrow_group(w)) {
        case 8:
            launch_next(c, k_fill_row_correct<8, VW, KM>, grid, 256, 0, out, ldo, g.p, w, mp, mi, Wop, ldw, Wn, H, k,
                        mean,
                                                                  scale);
            break;
        case 16:
            launch_next(c, k_fill_row_correct<16, VW, KM>, grid, 256, 0, out, ldo, g.p, w, mp, mi, Wop, ldw, Wn, H, k,
                        mean,
                                                                   scale);
            break;
        case 32:
            launch_next(c, k_fill_row_correct<32, VW, KM>, grid, 256, 0, out, ldo, g.p, w, mp, mi, Wop, ldw, Wn, H, k,
                        mean,
                                                                   scale);
            break;
        default:
            launch_next(c, k_fill_row_correct<0, VW, KM>, grid, 256, 0, out, ldo, g.p, w, mp, mi, Wop, ldw, Wn, H, k,
                        mean,
                                                                  scale);
    }
}

void launch_fill_row_correct(Ctx& c, const Geno& g, float* out, int ldo, int w, const float* Wop, int ldw,
                             const float* Wn, const float* H, int k, const double* mean, const double* scale) {
    if (!g.p || !w) return;
    SLFMM_REQUIRE(w <= 128 && k >= 1 && k <= kMaxNmfK, SLFMM_ERR_BAD_ARG, "NMF correction shape");
    const unsigned grid = (unsigned)grid_for(c, g.p, 8);
    with_rows(Wn, k, 8, [&](auto vw, auto km) {
        fill_row_correct_launch<decltype(vw)::value, decltype(km)::value>(c, g, grid, out, ldo, w, Wop, ldw, Wn, H, k,
                                                                          mean, scale);
    });
    SLFMM_LAUNCHED(c, "k_fill_row_correct");
}

__global__ void k_scale_mean_f32(const double* __restrict__ mean, const double* __restrict__ scale, uint64_t p,
                                 float2* __restrict__ out) {
    dependent_start();
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < p; r += (uint64_t)gridDim.x * blockDim.x)
        out[r] = make_float2((float)scale[r], (float)mean[r]);
}

template <int VW, int KM>
static void fill_col_correct_launch(Ctx& c, const Geno& g, unsigned grid, uint64_t nseg, double* S, int lds, int w,
                                    const float* Qop, int ldq, const float* Wn, const float* H, int k,
                                    const float2* sm) {
    const uint64_t* cp = g.missT_ptr.get();
    const uint32_t* ci = g.missT_idx.get();
    switch (narrow_group(w)) {
        case 8:
            launch_next(c, k_fill_col_correct<8, VW, KM>, grid, 256, 0, S, lds, g.n, w, nseg, cp, ci, Qop, ldq, Wn, H,
                        k, sm);
            break;
        case 16:
            launch_next(c, k_fill_col_correct<16, VW, KM>, grid, 256, 0, S, lds, g.n, w, nseg, cp, ci, Qop, ldq, Wn,
                        H, k, sm);
            break;
        case 32:
            launch_next(c, k_fill_col_correct<32, VW, KM>, grid, 256, 0, S, lds, g.n, w, nseg, cp, ci, Qop, ldq, Wn,
                        H, k, sm);
            break;
        default:
            launch_next(c, k_fill_col_correct<0, VW, KM>, grid, 256, 0, S, lds, g.n, w, nseg, cp, ci, Qop, ldq, Wn, H,
                        k, sm);
    }
}

void launch_fill_col_correct(Ctx& c, const Geno& g, double* S, int lds, int w, const float* Qop, int ldq,
                             const float* Wn, const float* H, int k, const double* mean, const double* scale) {
    if (!g.n || !w) return;
    SLFMM_REQUIRE(w <= 128 && k >= 1 && k <= kMaxNmfK, SLFMM_ERR_BAD_ARG, "NMF correction shape");
    const uint64_t nseg = std::max<uint64_t>(1, ceil_div(g.missT_max, kColSeg));
    const unsigned grid = (unsigned)grid_for(c, g.n * nseg, 8);
    DBuf<float2> sm(std::max<uint64_t>(g.p, 1), c.stream);
    launch_next(c, k_scale_mean_f32, grid_for(c, g.p, 256), 256, 0, mean, scale, g.p, sm.get());
    SLFMM_LAUNCHED(c, "k_scale_mean_f32");
    // 3 000 samples x 7 000 missing calls, rank 8, with 16 and 32 bytes at a time: 8
    // columns 317 and 265 us, 18 (a lane each) 588 and 720
    with_rows(H, k, w <= 16 ? 8 : 4, [&](auto vw, auto km) {
        fill_col_correct_launch<decltype(vw)::value, decltype(km)::value>(c, g, grid, nseg, S, lds, w, Qop, ldq, Wn, H,
                                                                          k, sm.get());
    });
    SLFMM_LAUNCHED(c, "k_fill_col_correct");
}

void launch_add_mean_colsum(Ctx& c, float* out, int ldo, uint64_t p, int w, const double* mean, const double* cs) {
    if (!p || !w) return;
    launch_next(c, k_add_mean_colsum, grid_for(c, p * w, 256), 256, 0, out, ldo, p, w, mean, cs);
    SLFMM_LAUNCHED(c, "k_add_mean_colsum");
}

void launch_nmf_update_f64(Ctx& c, double* X, uint64_t m, int k, const double* num, int ldn, const double* denom,
                           double eps) {
    if (!m) return;
    launch_next(c, k_nmf_update<double>, grid_for(c, m * k, 256), 256, 0, X, m, k, num, ldn, denom, eps);
    SLFMM_LAUNCHED(c, "k_nmf_update");
}

void launch_nmf_update_f32(Ctx& c, double* X, uint64_t m, int k, const float* num, int ldn, const double* denom,
                           double eps) {
    if (!m) return;
    launch_next(c, k_nmf_update<float>, grid_for(c, m * k, 256), 256, 0, X, m, k, num, ldn, denom, eps);
    SLFMM_LAUNCHED(c, "k_nmf_update");
}

void launch_nmf_normalize(Ctx& c, double* W, uint64_t n, double* H, uint64_t p, int k, const double* colsum,
                          double eps) {
    launch_next(c, k_nmf_normalize, grid_for(c, (n + p) * k, 256), 256, 0, W, n, H, p, k, colsum, eps);
    SLFMM_LAUNCHED(c, "k_nmf_normalize");
}

void launch_nmf_abs_f64(Ctx& c, const double* src, int ld, double* X, uint64_t m, int k) {
    if (!m) return;
    launch_next(c, k_nmf_sign<double>, grid_for(c, m * k, 256), 256, 0, src, ld, X, m, k, 0);
    SLFMM_LAUNCHED(c, "k_nmf_sign");
}

void launch_nmf_clamp0_f32(Ctx& c, const float* src, int ld, double* X, uint64_t m, int k) {
    if (!m) return;
    launch_next(c, k_nmf_sign<float>, grid_for(c, m * k, 256), 256, 0, src, ld, X, m, k, 1);
    SLFMM_LAUNCHED(c, "k_nmf_sign");
}

// a warp per SNP at a time, as many as are resident
static unsigned cv_grid(const Ctx& c, uint64_t p) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(p, 8), (uint64_t)c.sm_count * 8));
}

uint64_t launch_nmf_cv(Ctx& c, const Geno& g, uint64_t chunk, uint64_t mask_seed, double rate, const float* W,
                       const float* H, int k, DBuf<double>& part) {
    const bool cc = c.rng == SLFMM_RNG_CHACHA8;
    const uint64_t th = cc ? rate_threshold(rate, 52) : rate_threshold(rate);
    const unsigned grid = cv_grid(c, g.p);
    const uint64_t rows = (uint64_t)grid * 8;
    if (part.n < rows * 3) part.alloc(rows * 3, c.stream);
    auto go = [&](auto kern) {
        launch_next(c, kern, grid, 256, 0, packed_rows(g), g.stride, g.n, g.p, chunk, mask_seed, th, W, H, k,
                                         g.counts.get(), part.get());
    };
    if (k <= 16) {
        if (cc) go(k_nmf_cv<true, 16>);
        else go(k_nmf_cv<false, 16>);
    } else {
        if (cc) go(k_nmf_cv<true, 32>);
        else go(k_nmf_cv<false, 32>);
    }
    SLFMM_LAUNCHED(c, "k_nmf_cv");
    return rows;
}

uint64_t launch_nmf_gwas_cv(Ctx& c, const Geno& g, uint64_t chunk, uint64_t seed, double rate, const float* W,
                            const float* Wpt, int k, DBuf<double>& part) {
    DBuf<uint64_t> base(std::max<uint64_t>(g.p, 1), c.stream);
    const uint64_t nchunks = ceil_div(g.p, chunk);
    launch_next(c, k_obs_base, grid_for(c, nchunks, 1), 1024, 0, g.counts.get(), g.p, chunk, base.get());
    SLFMM_LAUNCHED(c, "k_obs_base");
    const bool cc = c.rng == SLFMM_RNG_CHACHA8;
    const uint64_t th = cc ? rate_threshold(rate, 52) : rate_threshold(rate);
    const unsigned grid = cv_grid(c, g.p);
    const uint64_t rows = (uint64_t)grid * 8;
    if (part.n < rows * 3) part.alloc(rows * 3, c.stream);
    // rows of W+ as 16-byte vectors
    const bool w4 = k % 4 == 0 && reinterpret_cast<uintptr_t>(Wpt) % 16 == 0;
    auto go = [&](auto kern) {
        launch_next(c, kern, grid, 256, 0, packed_rows(g), g.stride, g.n, g.p, chunk, seed, th, W, Wpt, k,
                                         g.counts.get(), base.get(), part.get());
    };
    if (k <= 16) {
        if (cc) w4 ? go(k_nmf_gwas_cv<true, true, 16>) : go(k_nmf_gwas_cv<true, false, 16>);
        else w4 ? go(k_nmf_gwas_cv<false, true, 16>) : go(k_nmf_gwas_cv<false, false, 16>);
    } else {
        if (cc) w4 ? go(k_nmf_gwas_cv<true, true, 32>) : go(k_nmf_gwas_cv<true, false, 32>);
        else w4 ? go(k_nmf_gwas_cv<false, true, 32>) : go(k_nmf_gwas_cv<false, false, 32>);
    }
    SLFMM_LAUNCHED(c, "k_nmf_gwas_cv");
    return rows;
}

}  // namespace slfmm
