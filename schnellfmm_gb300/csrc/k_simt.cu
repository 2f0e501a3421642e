// Plain FP32 SIMT contractions over the packed genotype matrix.
//
// This is the straightforward GPU formulation of the reference's per-chunk
// dgemms (src/rsvd.rs:61-69, :88-97, :117-125, :144-153 and
// src/testing.rs:355-374): every 2-bit code is mapped through a per-SNP
// 4-entry lookup table (the standardised value of that genotype, 0 for a
// missing call under mean imputation) and multiplied in FP32.  It serves as
// the "plain FP32 GPU path" the tensor-core path is measured against and as
// an independent second implementation for parity checks.
#include "fp_convert.cuh"
#include "slfmm_internal.h"

namespace slfmm {
namespace {

// Both contractions give a thread whole rows of 16 outputs, two of them (SNPs or
// samples): a genotype's value is looked up once (a table in shared memory, two
// integer operations for its address) for 16 multiply-adds, whose operand row is
// four 16-byte loads of one address for the warp.  With 16 threads to a SNP, each
// looking the value up for a column of its own, the loads bound both passes:
// 2 504 x 60 000 x 16 took 671 us by rows and 344 us by columns, now 161 and 175
// (65 us at the FP32 rate; the shared-memory return, 18 cycles per K step and warp
// for 32 x 32 products, is 80 % busy).  Tiles of 4 x 16 (too few warps: 210 and
// 215), of 4 x 8 (215 and 185) and two products to an instruction (176 and 182)
// were slower.
constexpr int kLutThreads = 64;
constexpr int kLutCols = 16;
constexpr int kRowSamples = 128; // samples per smem stage (32 bytes per SNP row)

__device__ __forceinline__ void copy16(void* dst, const void* src, bool in) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_issued() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest group have landed
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// acc[c] += v w[c] for a row of 16 in shared memory
__device__ __forceinline__ void fma_row(float v, const float4 (&w)[4], float (&acc)[kLutCols]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        acc[4 * q] = fmaf(v, w[q].x, acc[4 * q]);
        acc[4 * q + 1] = fmaf(v, w[q].y, acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(v, w[q].z, acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(v, w[q].w, acc[4 * q + 3]);
    }
}

// out[j, c] = sum_i lut_j[code_ij] * W[i, c]; W is (n_pad x wp) row-major
// with zero rows beyond n.  R SNPs and 16 columns (blockIdx.y) per thread.
template <int R>
__global__ void __launch_bounds__(kLutThreads) k_row_lut(const uint8_t* __restrict__ packed, uint64_t stride,
                                                         uint64_t p, uint64_t n, const float4* __restrict__ lut,
                                                         const float* __restrict__ W, int wp,
                                                         float* __restrict__ out) {
    dependent_wait();
    __shared__ __align__(16) float ws[2][kRowSamples][kLutCols];
    __shared__ float luts[R][4][kLutThreads];
    const int tid = threadIdx.x;
    const uint64_t j0 = (uint64_t)blockIdx.x * (kLutThreads * R) + tid;
    const float* Wc = W + blockIdx.y * kLutCols;
    const uint64_t nblk = (n + kRowSamples - 1) / kRowSamples;
    auto stage = [&](uint64_t blk) {
        if (blk < nblk)
            for (int e = tid; e < kRowSamples * 4; e += kLutThreads)
                copy16(&ws[blk & 1][e >> 2][4 * (e & 3)], Wc + (blk * kRowSamples + (e >> 2)) * wp + 4 * (e & 3), true);
        copies_issued();
    };
    stage(0);
    const uint32_t* row[R];
    float acc[R][kLutCols];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint64_t j = j0 + r * kLutThreads;
        const float4 v = j < p ? lut[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        luts[r][0][tid] = v.x, luts[r][1][tid] = v.y, luts[r][2][tid] = v.z, luts[r][3][tid] = v.w;
        row[r] = reinterpret_cast<const uint32_t*>(packed + (j < p ? j : 0) * stride);
#pragma unroll
        for (int c = 0; c < kLutCols; ++c) acc[r][c] = 0.f;
    }
    uint32_t next[R];
#pragma unroll
    for (int r = 0; r < R; ++r) next[r] = nblk ? row[r][0] : 0u;
    for (uint64_t blk = 0; blk < nblk; ++blk) {
        stage(blk + 1);
        copies_landed();
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < 8; ++w) {
            uint32_t cw[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                cw[r] = next[r];
                if (w < 7 || blk + 1 < nblk) next[r] = row[r][blk * 8 + w + 1];
            }
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float4* ws4 = reinterpret_cast<const float4*>(ws[blk & 1][w * 16 + k]);
                const float4 wv[4] = {ws4[0], ws4[1], ws4[2], ws4[3]};
#pragma unroll
                for (int r = 0; r < R; ++r) fma_row(luts[r][(cw[r] >> (2 * k)) & 3u][tid], wv, acc[r]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint64_t j = j0 + r * kLutThreads;
        if (j >= p) continue;
        float4* o = reinterpret_cast<float4*>(out + j * wp + blockIdx.y * kLutCols);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            o[q] = make_float4(acc[r][4 * q], acc[r][4 * q + 1], acc[r][4 * q + 2], acc[r][4 * q + 3]);
    }
}

constexpr int kColSamples = 2 * kLutThreads; // samples per CTA (32 bytes per SNP row)
constexpr int kColSnps = 32;                 // a split is a whole number of these
constexpr int kColStage = 64;                // SNPs per smem stage

// part[split, i, c] = sum_{j in split} lut_j[code_ij] * Q[j, c]; Q is p x wp.
// Two samples and 16 columns (blockIdx.z) per thread.
__global__ void __launch_bounds__(kLutThreads) k_col_lut(const uint8_t* __restrict__ packed, uint64_t stride,
                                                         uint64_t p, uint64_t n_pad, const float4* __restrict__ lut,
                                                         const float* __restrict__ Q, int wp, uint64_t per_split,
                                                         float* __restrict__ part) {
    dependent_wait();
    __shared__ __align__(16) float qs[2][kColStage][kLutCols];
    __shared__ __align__(16) float luts[2][kColStage][4];
    __shared__ __align__(16) uint8_t codes[2][kColStage][kColSamples / 4];
    const int tid = threadIdx.x;
    const uint64_t tile = blockIdx.x;
    const uint64_t s0 = (uint64_t)blockIdx.y * per_split;
    const uint64_t s1 = min(p, s0 + per_split);
    const float* Qc = Q + blockIdx.z * kLutCols;
    float acc[2][kLutCols];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int c = 0; c < kLutCols; ++c) acc[s][c] = 0.f;
    // SNPs past the split: value 0 of every code (and row 0's address, unread)
    auto stage = [&](uint64_t j0, int b) {
        if (j0 < s1) {
            for (int e = tid; e < kColStage * 4; e += kLutThreads) {
                const uint64_t j = j0 + (e >> 2);
                copy16(&qs[b][e >> 2][4 * (e & 3)], Qc + (j < s1 ? j : s0) * wp + 4 * (e & 3), j < s1);
            }
            for (int e = tid; e < kColStage * 2; e += kLutThreads) {
                const uint64_t j = j0 + (e >> 1);
                copy16(&codes[b][e >> 1][16 * (e & 1)], packed + (j < s1 ? j : s0) * stride + tile * 32 + 16 * (e & 1),
                       j < s1);
            }
            for (int e = tid; e < kColStage; e += kLutThreads)
                copy16(&luts[b][e][0], lut + (j0 + e < s1 ? j0 + e : s0), j0 + e < s1);
        }
        copies_issued();
    };
    stage(s0, 0);
    int b = 0;
    for (uint64_t j0 = s0; j0 < s1; j0 += kColStage, b ^= 1) {
        stage(j0 + kColStage, b ^ 1);
        copies_landed();
        __syncthreads();
#pragma unroll 8
        for (int jj = 0; jj < kColStage; ++jj) {
            const uint32_t two = codes[b][jj][tid >> 1] >> (4 * (tid & 1));
            const float4* q4 = reinterpret_cast<const float4*>(qs[b][jj]);
            const float4 qv[4] = {q4[0], q4[1], q4[2], q4[3]};
            fma_row(luts[b][jj][two & 3u], qv, acc[0]);
            fma_row(luts[b][jj][(two >> 2) & 3u], qv, acc[1]);
        }
        __syncthreads();
    }
    float* dst = part + ((uint64_t)blockIdx.y * n_pad + tile * kColSamples + 2 * tid) * wp + blockIdx.z * kLutCols;
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            reinterpret_cast<float4*>(dst + s * wp)[q] =
                make_float4(acc[s][4 * q], acc[s][4 * q + 1], acc[s][4 * q + 2], acc[s][4 * q + 3]);
}

// S (n x wp) = the sum of the K splits' FP32 partials, in their order in FP64;
// columns w .. wp - 1 are padding and stay zero.  A thread per real element (FP64
// additions hold a scheduler for 64 cycles however many lanes take part), eight
// partials in flight: 37 splits of 8 500 x 20 of 32 took 43 us over all 32 columns
// with a load per addition, 30 us so.
__global__ void __launch_bounds__(256) k_reduce_splits(const float* __restrict__ part, int splits, uint64_t n, int w,
                                                       int wp, uint64_t n_pad, double* __restrict__ S) {
    dependent_start();
    const uint64_t total = n * (uint64_t)w, stride = n_pad * wp;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / (unsigned)w;
        const int c = (int)(t - i * w);
        const float* p = part + i * wp + c;
        double acc = 0.0;
        for (int s = 0; s < splits; s += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = s + u < splits ? p[(uint64_t)(s + u) * stride] : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (s + u < splits) acc += f64_of_f32(v[u]);
        }
        S[i * wp + c] = acc;
        for (int z = w + c; z < wp; z += w) S[i * wp + z] = 0.0;
    }
}

}  // namespace

void launch_reduce_splits(Ctx& c, const float* part, int splits, uint64_t n, int w, int wp, uint64_t n_pad,
                          double* S) {
    if (!n) return;
    launch_next(c, k_reduce_splits, grid_for(c, n * w, 256), 256, 0, part, splits, n, w, wp, n_pad, S);
    SLFMM_LAUNCHED(c, "k_reduce_splits");
}

void launch_row_lut(Ctx& c, const Geno& g, const float* lut, const float* W, int wp, float* out) {
    if (g.p == 0) return;
    SLFMM_REQUIRE(wp >= kLutCols && wp <= 128 && wp % kLutCols == 0, SLFMM_ERR_BAD_ARG,
                  "row contraction width must be a multiple of 16 <= 128");
    // two SNPs to a thread share its operand loads, but halve the warps: from more
    // than a block per SM on (2 504 samples x 16, one and two to a thread: 18 000 SNPs
    // 74 and 101 us, 25 000 107 and 109, 32 000 126 and 110, 60 000 222 and 165)
    auto go = [&](auto kern, int r) {
        // not launch_next: under a kernel that still runs the three blocks per SM
        // would take unequal places, and the pass lasts as long as the fullest SM
        kern<<<dim3((unsigned)ceil_div(g.p, (uint64_t)kLutThreads * r), (unsigned)(wp / kLutCols)), kLutThreads, 0,
               c.stream>>>(packed_rows(g), g.stride, g.p, g.n, reinterpret_cast<const float4*>(lut), W, wp, out);
    };
    const uint64_t pairs = ceil_div(g.p, 2 * kLutThreads) * (uint64_t)(wp / kLutCols);
    if (pairs > (uint64_t)std::max(c.sm_count, 1)) go(k_row_lut<2>, 2);
    else go(k_row_lut<1>, 1);
    SLFMM_LAUNCHED(c, "k_row_lut");
}

void launch_col_lut(Ctx& c, const Geno& g, const float* lut, const float* Q, int wp, double* S) {
    if (g.n == 0) return;
    if (g.p == 0) { SLFMM_CUDA(cudaMemsetAsync(S, 0, g.n * wp * sizeof(double), c.stream)); return; }
    SLFMM_REQUIRE(wp >= kLutCols && wp <= 128 && wp % kLutCols == 0, SLFMM_ERR_BAD_ARG,
                  "column contraction width must be a multiple of 16 <= 128");
    const uint64_t tiles = ceil_div(g.n, kColSamples);
    const uint64_t n_pad = tiles * kColSamples;
    // split the SNP range so each thread accumulates at most ~16k SNPs in
    // FP32 and the grid fills the device
    uint64_t splits = std::max<uint64_t>(ceil_div(g.p, 16384), ceil_div((uint64_t)c.sm_count * 4, tiles));
    splits = std::max<uint64_t>(1, std::min<uint64_t>(splits, std::max<uint64_t>(1, ceil_div(g.p, kColSnps))));
    const uint64_t per_split = round_up(ceil_div(g.p, splits), kColSnps);
    splits = ceil_div(g.p, per_split);
    DBuf<float> part(splits * n_pad * wp, c.stream);
    k_col_lut<<<dim3((unsigned)tiles, (unsigned)splits, (unsigned)(wp / kLutCols)), kLutThreads, 0, c.stream>>>(
        packed_rows(g), g.stride, g.p, n_pad, reinterpret_cast<const float4*>(lut), Q, wp, per_split, part.get());
    SLFMM_LAUNCHED(c, "k_col_lut");
    launch_reduce_splits(c, part.get(), (int)splits, g.n, wp, wp, n_pad, S);
}

}  // namespace slfmm
