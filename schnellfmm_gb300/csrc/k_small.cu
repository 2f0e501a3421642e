// FP64 dense helpers for the small / tall-skinny linear algebra of the path:
// covariate centring (src/lib.rs:102-117), Step 0 (src/precompute.rs:30-88),
// Cholesky-QR2 of the sketches (replacing the LAPACK QR of
// src/rsvd.rs:75,105,131), the small SVD (src/rsvd.rs:162, src/nmf.rs:321)
// and safe_inv (src/testing.rs:996-1024).  GB300's FP64 rate is low, so
// these only ever touch n x w, w x w or p x w objects with tiny w.
#include <cooperative_groups.h>

#include "fp_convert.cuh"
#include "slfmm_internal.h"

namespace slfmm {
namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// block-wide sum with a fixed reduction order (deterministic)
__device__ double block_sum(double v, double* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    double t = 0.0;
    if (wid == 0) {
        t = lane < nw ? red[lane] : 0.0;
        t = warp_sum(t);
    }
    __syncthreads();
    if (threadIdx.x == 0) red[0] = t;
    __syncthreads();
    const double r = red[0];
    __syncthreads();
    return r;
}

__global__ void k_colmeans(const double* __restrict__ A, uint64_t m, int lda, double* __restrict__ out,
                           int divide) {
    dependent_start();
    __shared__ double red[32];
    const int col = blockIdx.x;
    double s = 0.0;
    for (uint64_t i = threadIdx.x; i < m; i += blockDim.x) s += A[i * lda + col];
    s = block_sum(s, red);
    if (threadIdx.x == 0) out[col] = divide ? (m ? s / (double)m : 0.0) : s;
}

__global__ void k_center_cols(double* __restrict__ A, uint64_t m, int a, int lda,
                              const double* __restrict__ means) {
    dependent_start();
    const uint64_t total = m * a;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / a;
        const int c = (int)(t - i * a);
        A[i * lda + c] -= means[c];
    }
}

// divide a column by its sample sd (n-1 denominator) unless sd <= 1e-14
__global__ void k_scale_cols_sd(double* __restrict__ A, uint64_t m, int lda) {
    dependent_start();
    __shared__ double red[32];
    const int col = blockIdx.x;
    double s = 0.0;
    for (uint64_t i = threadIdx.x; i < m; i += blockDim.x) {
        const double v = A[i * lda + col];
        s += v * v;
    }
    s = block_sum(s, red);
    const double sd = sqrt(s / ((double)m - 1.0));
    if (sd > 1e-14)
        for (uint64_t i = threadIdx.x; i < m; i += blockDim.x) A[i * lda + col] /= sd;
}

// Tiled A^T B over a row range: 32x32 output tile per CTA, 16x16 threads,
// FP64 accumulation; partial[split] written, reduced by k_sum_partials.
template <typename T>
__global__ void __launch_bounds__(256) k_atb(const T* __restrict__ A, int lda, const T* __restrict__ B,
                                             int ldb, uint64_t m, int a, int b, uint64_t rows_per_split,
                                             double* __restrict__ part) {
    dependent_start();
    __shared__ double As[32][33];
    __shared__ double Bs[32][33];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const uint64_t i0 = (uint64_t)blockIdx.z * rows_per_split;
    const uint64_t i1 = min(m, i0 + rows_per_split);
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (uint64_t ib = i0; ib < i1; ib += 32) {
        __syncthreads();
        for (int e = threadIdx.x; e < 32 * 32; e += 256) {
            const int ii = e >> 5, cc = e & 31;
            const uint64_t i = ib + ii;
            As[ii][cc] = (i < i1 && r0 + cc < a) ? (double)A[i * lda + r0 + cc] : 0.0;
            Bs[ii][cc] = (i < i1 && c0 + cc < b) ? (double)B[i * ldb + c0 + cc] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int ii = 0; ii < 32; ++ii) {
            const double a0 = As[ii][ty], a1 = As[ii][ty + 16];
            const double b0 = Bs[ii][tx], b1 = Bs[ii][tx + 16];
            acc[0][0] = fma(a0, b0, acc[0][0]);
            acc[0][1] = fma(a0, b1, acc[0][1]);
            acc[1][0] = fma(a1, b0, acc[1][0]);
            acc[1][1] = fma(a1, b1, acc[1][1]);
        }
    }
    double* dst = part + (uint64_t)blockIdx.z * a * b;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int r = r0 + ty + 16 * u, cc = c0 + tx + 16 * v;
            if (r < a && cc < b) dst[r * b + cc] = acc[u][v];
        }
}

// A^T B over a row range with the a x b outputs laid flat: thread t of the
// CTA owns outputs o0 + t + 256 k (k < R), rows of A and B are staged 32 at
// a time in shared memory, and every FMA issued is one of the a x b (the
// 32 x 32 output tiles of k_atb spend 39-61 % of their FP64 FMAs on padding
// at the widths used here: 20, 50, 71).  FP64 accumulation in row order
// within the range; partial[split] written, reduced by k_sum_partials.
template <typename T, int R>
__global__ void __launch_bounds__(256) k_atb_flat(const T* __restrict__ A, int lda, const T* __restrict__ B,
                                                  int ldb, uint64_t m, int a, int b, uint64_t rows_per_split,
                                                  double* __restrict__ part) {
    dependent_start();
    extern __shared__ double stage[];
    double* As = stage;             // [32][a]
    double* Bs = stage + 32 * a;    // [32][b]
    const int tid = threadIdx.x;
    const int ab = a * b;
    const int o0 = blockIdx.x * 256 * R;
    const uint64_t i0 = (uint64_t)blockIdx.y * rows_per_split;
    const uint64_t i1 = min(m, i0 + rows_per_split);
    int ra[R], cb[R];
    double acc[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int o = o0 + tid + 256 * k;
        ra[k] = o < ab ? o / b : 0;
        cb[k] = o < ab ? o % b : 0;
        acc[k] = 0.0;
    }
    // warp-uniform: the last k with an output in this warp
    const int wfirst = o0 + (tid & ~31);
    for (uint64_t ib = i0; ib < i1; ib += 32) {
        __syncthreads();
        for (int e = tid; e < 32 * a; e += 256) {
            const int ii = e / a, cc = e % a;
            const uint64_t i = ib + ii;
            As[e] = i < i1 ? (double)A[i * lda + cc] : 0.0;
        }
        for (int e = tid; e < 32 * b; e += 256) {
            const int ii = e / b, cc = e % b;
            const uint64_t i = ib + ii;
            Bs[e] = i < i1 ? (double)B[i * ldb + cc] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (wfirst + 256 * k >= ab) break;
#pragma unroll 8
            for (int ii = 0; ii < 32; ++ii) acc[k] = fma(As[ii * a + ra[k]], Bs[ii * b + cb[k]], acc[k]);
        }
    }
    double* dst = part + (uint64_t)blockIdx.y * ab;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int o = o0 + tid + 256 * k;
        if (o < ab) dst[o] = acc[k];
    }
}

// FP32 Gram with FP32 products summed over 32-row tiles and FP64 across
// tiles (used for the p x l sketches, whose FP64 Gram would dominate).
__global__ void __launch_bounds__(256) k_gram_f32(const float* __restrict__ A, int lda, uint64_t m, int a,
                                                  uint64_t rows_per_split, double* __restrict__ part) {
    dependent_start();
    __shared__ float As[32][33];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const uint64_t i0 = (uint64_t)blockIdx.z * rows_per_split;
    const uint64_t i1 = min(m, i0 + rows_per_split);
    __shared__ float Bs[32][33];
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (uint64_t ib = i0; ib < i1; ib += 32) {
        __syncthreads();
        for (int e = threadIdx.x; e < 32 * 32; e += 256) {
            const int ii = e >> 5, cc = e & 31;
            const uint64_t i = ib + ii;
            As[ii][cc] = (i < i1 && r0 + cc < a) ? A[i * lda + r0 + cc] : 0.f;
            Bs[ii][cc] = (i < i1 && c0 + cc < a) ? A[i * lda + c0 + cc] : 0.f;
        }
        __syncthreads();
        float t[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 8
        for (int ii = 0; ii < 32; ++ii) {
            const float a0 = As[ii][ty], a1 = As[ii][ty + 16];
            const float b0 = Bs[ii][tx], b1 = Bs[ii][tx + 16];
            t[0][0] = fmaf(a0, b0, t[0][0]);
            t[0][1] = fmaf(a0, b1, t[0][1]);
            t[1][0] = fmaf(a1, b0, t[1][0]);
            t[1][1] = fmaf(a1, b1, t[1][1]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) acc[u][v] += (double)t[u][v];
    }
    double* dst = part + (uint64_t)blockIdx.z * a * a;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int r = r0 + ty + 16 * u, cc = c0 + tx + 16 * v;
            if (r < a && cc < a) dst[r * a + cc] = acc[u][v];
        }
}

// Elements 4 q .. 4 q + 3 of a row (16-byte aligned, 4 q < lda), the ones at
// or past column a zero (no load when the whole quad is past a).
__device__ __forceinline__ float4 row_quad(const float* row, int q, int a) {
    if (4 * q >= a) return make_float4(0.f, 0.f, 0.f, 0.f);
    float4 b = reinterpret_cast<const float4*>(row)[q];
    if (4 * q + 4 > a) {
        b.y = 4 * q + 1 < a ? b.y : 0.f;
        b.z = 4 * q + 2 < a ? b.z : 0.f;
        b.w = 4 * q + 3 < a ? b.w : 0.f;
    }
    return b;
}

// Narrow (a <= 32) FP32 Gram, one warp per run of rows: lane c holds row
// element c and takes row[k] by shuffle.  FP32 sums over runs of 256 rows,
// FP64 across runs; the block's warps reduce through shared memory into one
// partial.  (Rows of any stride; the tiled kernel below covers 16-byte
// aligned rows of at most 32 floats.)
constexpr int kGramRun = 256;
constexpr size_t kGramNarrowSmem = 8 * 32 * 33 * sizeof(double);
__global__ void __launch_bounds__(256, 2) k_gram_narrow(const float* __restrict__ A, int lda, uint64_t m, int a,
                                                        double* __restrict__ part) {
    dependent_start();
    extern __shared__ double gsm[];  // [8 warps][32][33] FP64 sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* mine = gsm + warp * 32 * 33;
#pragma unroll
    for (int k = 0; k < 32; ++k) mine[k * 33 + lane] = 0.0;
    const uint64_t nruns = (m + kGramRun - 1) / kGramRun;
    for (uint64_t run = (uint64_t)blockIdx.x * 8 + warp; run < nruns; run += (uint64_t)gridDim.x * 8) {
        float acc[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = 0.f;
        const uint64_t i0 = run * kGramRun, i1 = min(m, i0 + kGramRun);
        for (uint64_t i = i0; i < i1; i += 8) {
            float v[8];  // eight rows in flight per warp
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = (lane < a && i + u < i1) ? A[(i + u) * lda + lane] : 0.f;
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int k = 0; k < 32; ++k) acc[k] = fmaf(__shfl_sync(0xffffffffu, v[u], k), v[u], acc[k]);
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) mine[k * 33 + lane] += (double)acc[k];
    }
    __syncthreads();
    // warps summed in a fixed order (deterministic)
    double* dst = part + (uint64_t)blockIdx.x * a * a;
    for (int e = threadIdx.x; e < a * a; e += blockDim.x) {
        const int k = e / a, cc = e % a;
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += gsm[w * 32 * 33 + k * 33 + cc];
        dst[e] = t;
    }
}

// A (m x a, a <= 32) <- A Linv^T in place, one warp per row: lane c holds
// column c of Linv^T (FP32) and accumulates out[c] = sum_k row[k] Linv[c][k]
// from the broadcast row elements; loads and stores are whole rows.
__global__ void __launch_bounds__(256) k_trmul_narrow(float* __restrict__ A, int lda, uint64_t m, int a,
                                                      const double* __restrict__ Linv) {
    dependent_start();
    const int lane = threadIdx.x & 31;
    float R[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) R[k] = (k < a && lane < a) ? (float)Linv[lane * a + k] : 0.f;
    // each warp takes runs of 4 consecutive rows (four loads in flight)
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t i = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 4; i < m; i += warps * 4) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = (lane < a && i + u < m) ? A[(i + u) * lda + lane] : 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float out = 0.f;
#pragma unroll
            for (int k = 0; k < 32; ++k) out = fmaf(__shfl_sync(0xffffffffu, v[u], k), R[k], out);
            if (lane < a && i + u < m) A[(i + u) * lda + lane] = out;
        }
    }
}

// Tiles of 128 rows of a narrow matrix (a <= lda <= 32, lda % 4 == 0, rows
// 16-byte aligned) stream through a ring of kPipe shared-memory stages with
// asynchronous 16-byte copies (cp.async, completion awaited by wait_group):
// tile i + kPipe - 1 is in flight while tile i is used.  One persistent block
// of 512 threads per SM takes tiles blockIdx.x, + gridDim.x, ...; each of its
// 16 warps uses 8 rows of a tile.  Rows past m are neither copied nor used.
__device__ __forceinline__ uint32_t smem_addr32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

constexpr int kNarrowTile = 128;
constexpr int kPipe = 4;
constexpr int kPipeThreads = 512;
constexpr size_t kPipeRing = (size_t)kPipe * kNarrowTile * 32 * sizeof(float);

__device__ __forceinline__ void pipe_issue(const float* A, int lda, uint64_t m, uint64_t t, float* stage) {
    const int q = lda >> 2, nf4 = kNarrowTile * q;
    const float4* src = reinterpret_cast<const float4*>(A) + t * kNarrowTile * q;
    const uint64_t rows = min((uint64_t)kNarrowTile, m - t * kNarrowTile);
#pragma unroll
    for (int r = 0; r < 1024 / kPipeThreads; ++r) {
        const int e = threadIdx.x + kPipeThreads * r;
        if (e < nf4 && (uint64_t)(e / q) < rows)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr32(stage + 4 * e)), "l"(src + e)
                         : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__device__ __forceinline__ void pipe_commit_empty() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// wait for tile i (its copy group) and make every thread's copies visible
__device__ __forceinline__ void pipe_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPipe - 2) : "memory");
    __syncthreads();
}

// Gram over tiles: lane = 8 ky + cx of each warp owns the block
// G[8 ky + i][4 cx + j] (i < 8, j < 4) and reads its 12 row elements as three
// 16-byte shared-memory loads per row.  Elements past column a (padding, or
// the next row when lda < 32) only reach entries that are never written out.
// FP32 sums over up to 32 tiles (256 rows of a warp), then into per-warp FP64
// sums in shared memory; the warps are added in a fixed order into one partial
// per block.
__global__ void __launch_bounds__(kPipeThreads, 1) k_gram_tile(const float* __restrict__ A, int lda, uint64_t m, int a,
                                                            double* __restrict__ part) {
    dependent_start();
    extern __shared__ __align__(16) float ring[];  // [kPipe][128 rows][lda], then [16 warps][32][32] FP64
    double* dsum = reinterpret_cast<double*>(reinterpret_cast<uint8_t*>(ring) + kPipeRing);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ky = lane >> 3, cx = lane & 7;
    double* mine = dsum + warp * 32 * 32;  // [entry][lane]
    float acc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k] = 0.f;
    bool first = true;
    // The first sums are only widened, by integer operations: 32 conversions and 32
    // additions to zero by every warp held the FP64 pipe for half of a small Gram.
    auto flush = [&]() {
        if (first) {
#pragma unroll
            for (int k = 0; k < 32; ++k) mine[k * 32 + lane] = f64_of_f32(acc[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) mine[k * 32 + lane] += (double)acc[k];
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = 0.f;
        first = false;
    };
    const uint64_t ntiles = (m + kNarrowTile - 1) / kNarrowTile;
    const int tsz = kNarrowTile * lda;
    for (int k = 0; k < kPipe - 1; ++k) {
        const uint64_t t = blockIdx.x + (uint64_t)k * gridDim.x;
        if (t < ntiles) pipe_issue(A, lda, m, t, ring + k * tsz);
        else pipe_commit_empty();
    }
    int since = 0;
    for (uint64_t i = 0;; ++i) {
        const uint64_t t = blockIdx.x + i * gridDim.x;
        if (t >= ntiles) break;
        pipe_wait();
        const uint64_t tn = t + (uint64_t)(kPipe - 1) * gridDim.x;
        if (tn < ntiles) pipe_issue(A, lda, m, tn, ring + ((i + kPipe - 1) % kPipe) * tsz);
        else pipe_commit_empty();
        const int r0 = warp * 8;
        const uint64_t gr = t * kNarrowTile + r0;
        const int nrows = gr >= m ? 0 : (m - gr >= 8 ? 8 : (int)(m - gr));
        const float* base = ring + (i % kPipe) * tsz + r0 * lda;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (u < nrows) {
                const float4* row = reinterpret_cast<const float4*>(base + u * lda);
                const float4 ka = row[2 * ky], kb = row[2 * ky + 1], cv = row[cx];
                const float kk[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
                const float cc[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                for (int ii = 0; ii < 8; ++ii)
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj) acc[ii * 4 + jj] = fmaf(kk[ii], cc[jj], acc[ii * 4 + jj]);
            }
        }
        if (++since == 32) {
            flush();
            since = 0;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    flush();
    __syncthreads();
    // entry (k, c) of the block partial: lane 8 (k / 8) + c / 4, slot (k % 8) 4 + c % 4
    for (int e = threadIdx.x; e < a * a; e += kPipeThreads) {
        const int k = e / a, c = e % a;
        const int ln = 8 * (k >> 3) + (c >> 2), slot = (k & 7) * 4 + (c & 3);
        double tsum = 0.0;
        for (int w = 0; w < kPipeThreads / 32; ++w) tsum += dsum[w * 32 * 32 + slot * 32 + ln];
        part[(uint64_t)blockIdx.x * a * a + e] = tsum;
    }
}

// A (m x a, a <= 32, lda % 4 == 0, rows 16-byte aligned) <- A Linv^T in
// place for a lower-triangular Linv, two rows per thread: a row is read as
// 16-byte loads, out[c] = sum_{k <= c} row[k] Linv[c][k] in the order of k, and
// written back.  Linv sits in shared memory in FP32, transposed, so that the
// factors of four outputs are one broadcast 16-byte load for both rows (144
// loads per 1056 products).  Taken from device memory: as a kernel parameter it
// cost a copy to the host and a synchronisation per call, six per fit.
constexpr int kTrmulRows = 2;
__global__ void __launch_bounds__(256) k_trmul_rows(float* __restrict__ A, int lda, uint64_t m, int a,
                                                    const double* __restrict__ Linv) {
    dependent_start();
    __shared__ __align__(16) float Rt[32][32];  // Rt[k][c] = Linv[c][k], zero padded
    for (int e = threadIdx.x; e < 32 * 32; e += 256) {
        const int k = e >> 5, c = e & 31;
        Rt[k][c] = (k <= c && c < a) ? (float)Linv[c * a + k] : 0.f;
    }
    __syncthreads();
    const uint64_t step = (uint64_t)gridDim.x * 256;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < m; i += kTrmulRows * step) {
        float o[kTrmulRows][32];
#pragma unroll
        for (int r = 0; r < kTrmulRows; ++r)
#pragma unroll
            for (int c = 0; c < 32; ++c) o[r][c] = 0.f;
#pragma unroll
        for (int kq = 0; kq < 8; ++kq) {
            if (4 * kq >= a) break;
            float x[kTrmulRows][4];
#pragma unroll
            for (int r = 0; r < kTrmulRows; ++r) {
                const uint64_t row = i + r * step;
                const float4 v = row < m ? row_quad(A + row * lda, kq, a) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[r][0] = v.x;
                x[r][1] = v.y;
                x[r][2] = v.z;
                x[r][3] = v.w;
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const int k = 4 * kq + kk;
#pragma unroll
                for (int cq = kq; cq < 8; ++cq) {
                    const float4 f = reinterpret_cast<const float4*>(Rt[k])[cq];
                    const float ff[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (4 * cq + j >= k)
#pragma unroll
                            for (int r = 0; r < kTrmulRows; ++r)
                                o[r][4 * cq + j] = fmaf(x[r][kk], ff[j], o[r][4 * cq + j]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kTrmulRows; ++r) {
            const uint64_t row = i + r * step;
            if (row >= m) break;
            float* dst = A + row * lda;
#pragma unroll
            for (int cq = 0; cq < 8; ++cq) {
                if (4 * cq + 4 <= a) {
                    reinterpret_cast<float4*>(dst)[cq] =
                        make_float4(o[r][4 * cq], o[r][4 * cq + 1], o[r][4 * cq + 2], o[r][4 * cq + 3]);
                } else if (4 * cq < a) {
#pragma unroll
                    for (int jj = 0; jj < 4; ++jj)
                        if (4 * cq + jj < a) dst[4 * cq + jj] = o[r][4 * cq + jj];
                }
            }
        }
    }
}

// one block per entry: thread t sums partials t, t + 128, ... in order, then
// a fixed-shape tree (warp shuffles, then the four warps in order)
__global__ void __launch_bounds__(128) k_sum_partials_wide(const double* __restrict__ part, int splits,
                                                           uint64_t count, double* __restrict__ out) {
    dependent_start();
    __shared__ double ws[4];
    for (uint64_t e = blockIdx.x; e < count; e += gridDim.x) {
        double s = 0.0;
        for (int k = threadIdx.x; k < splits; k += 128) s += part[(uint64_t)k * count + e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x == 0) out[e] = (ws[0] + ws[1]) + (ws[2] + ws[3]);
        __syncthreads();
    }
}

__global__ void k_sum_partials(const double* __restrict__ part, int splits, uint64_t count,
                               double* __restrict__ out) {
    dependent_start();
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < count;
         t += (uint64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int k = 0; k < splits; ++k) s += part[(uint64_t)k * count + t];
        out[t] = s;
    }
}

// C = alpha * A B + beta * C with A (m x a), B (a x b) small; one thread per output.
template <typename TO>
__global__ void k_gemm_small(const double* __restrict__ A, int lda, uint64_t m, int a,
                             const double* __restrict__ B, int ldb, int b, double alpha, double beta,
                             TO* __restrict__ C, int ldc) {
    dependent_start();
    extern __shared__ double Bsm[];  // a x b
    for (int e = threadIdx.x; e < a * b; e += blockDim.x) Bsm[e] = B[(e / b) * ldb + (e % b)];
    __syncthreads();
    const uint64_t total = m * b;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / b;
        const int cc = (int)(t - i * b);
        double s = 0.0;
        const double* ar = A + i * lda;
        for (int k = 0; k < a; ++k) s = fma(ar[k], Bsm[k * b + cc], s);
        const double prev = beta != 0.0 ? (double)C[i * ldc + cc] : 0.0;
        C[i * ldc + cc] = (TO)(alpha * s + beta * prev);
    }
}

// A (m x a, FP32) <- A * Linv^T with Linv lower-triangular (a x a, FP64),
// i.e. A <- A R^-1 for the Cholesky factor R = L^T of A^T A.  The row lives
// in registers (fully unrolled up to AMAX columns).
template <int AMAX>
__global__ void __launch_bounds__(128) k_trmul_f32(float* __restrict__ A, int lda, uint64_t m, int a,
                                                   const double* __restrict__ Linv) {
    dependent_start();
    __shared__ float R[AMAX * AMAX];  // R[k][c] = Linv[c][k], zero padded
    for (int e = threadIdx.x; e < AMAX * AMAX; e += blockDim.x) {
        const int k = e / AMAX, cc = e % AMAX;
        R[e] = (k < a && cc < a) ? (float)Linv[cc * a + k] : 0.f;
    }
    __syncthreads();
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m;
         i += (uint64_t)gridDim.x * blockDim.x) {
        float row[AMAX], out[AMAX];
        float* ar = A + i * lda;
#pragma unroll
        for (int k = 0; k < AMAX; ++k) {
            row[k] = k < a ? ar[k] : 0.f;
            out[k] = 0.f;
        }
#pragma unroll
        for (int k = 0; k < AMAX; ++k)
#pragma unroll
            for (int cc = k; cc < AMAX; ++cc) out[cc] = fmaf(row[k], R[k * AMAX + cc], out[cc]);
#pragma unroll
        for (int k = 0; k < AMAX; ++k)
            if (k < a) ar[k] = out[k];
    }
}

// In-place Cholesky (lower) of an a x a SPD matrix in one CTA.  status[0] =
// number of pivots that were not positive (replaced by a tiny positive value).
// With drop_tol >= 0 a column whose residual pivot is <= drop_tol times its
// original diagonal is dropped instead: L_kk = 1, L_ik = 0, dropped[k] = 1
// (rank-deficient design columns).  status[0] counts replaced/dropped pivots.
__global__ void k_cholesky(double* __restrict__ G, int a, int* __restrict__ status,
                           double drop_tol, int* __restrict__ dropped, double* __restrict__ work) {
    dependent_start();
    extern __shared__ double S_sm[];
    double* S = work ? work : S_sm;   // global scratch for matrices wider than kMaxSmall
    __shared__ double piv;
    __shared__ int bad;
    __shared__ int drop_k;
    for (int e = threadIdx.x; e < a * a; e += blockDim.x) S[e] = G[e];
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    double dmax = 0.0;
    for (int k = 0; k < a; ++k) dmax = fmax(dmax, fabs(S[k * a + k]));
    for (int k = 0; k < a; ++k) {
        if (threadIdx.x == 0) {
            double v = S[k * a + k];
            drop_k = 0;
            if (drop_tol >= 0.0) {
                if (!(v > drop_tol * fabs(G[k * a + k])) || !(v > 1e-300)) { drop_k = 1; ++bad; v = 1.0; }
            } else if (!(v > 1e-300 + 1e-28 * dmax)) {
                v = 1e-28 * dmax + 1e-300;
                ++bad;
            }
            if (dropped) dropped[k] = drop_k;
            piv = sqrt(v);
            S[k * a + k] = piv;
        }
        __syncthreads();
        for (int i = k + 1 + threadIdx.x; i < a; i += blockDim.x) S[i * a + k] = drop_k ? 0.0 : S[i * a + k] / piv;
        __syncthreads();
        const int rem = a - k - 1;
        for (int e = threadIdx.x; e < rem * rem; e += blockDim.x) {
            const int i = k + 1 + e / rem, j = k + 1 + e % rem;
            if (j <= i) S[i * a + j] -= S[i * a + k] * S[j * a + k];
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < a * a; e += blockDim.x) {
        const int i = e / a, j = e % a;
        G[e] = j <= i ? S[e] : 0.0;
    }
    if (threadIdx.x == 0 && status) status[0] = bad;
}

// Inverse of a lower-triangular matrix: one thread per column.
__global__ void k_tri_inv_lower(const double* __restrict__ L, int a, double* __restrict__ X, int in_smem) {
    dependent_start();
    extern __shared__ double S_sm[];
    const double* S = in_smem ? S_sm : L;   // matrices wider than kMaxSmall are read in place
    if (in_smem) {
        for (int e = threadIdx.x; e < a * a; e += blockDim.x) S_sm[e] = L[e];
        __syncthreads();
    }
    for (int cc = threadIdx.x; cc < a; cc += blockDim.x) {
        for (int i = 0; i < cc; ++i) X[i * a + cc] = 0.0;
        for (int i = cc; i < a; ++i) {
            double s = (i == cc) ? 1.0 : 0.0;
            for (int k = cc; k < i; ++k) s -= S[i * a + k] * X[k * a + cc];
            X[i * a + cc] = s / S[i * a + i];
        }
    }
}

// Cholesky factor and its inverse in one pass: X = L^-1 of G = L L^T (G read
// only), with the pivot rules of k_cholesky.  A thread keeps its elements (i, j),
// j <= i, of the packed lower triangle in registers: element (i, j) is S_ij
// until step j makes it L_ij, then the running right-hand side s_ij of X's
// forward substitution, which step i divides by the pivot.  Step k updates every
// element below row k by one FMA with the same operand pair in both roles,
//   S_ij -= L_ik L_jk (j > k),   s_ij -= L_ik X_kj (j <= k),
// so both recurrences run their terms in the order of k_cholesky and
// k_tri_inv_lower and give the same bits.
//
// One SM issues an FP64 warp instruction per scheduler every 64 cycles
// (sqrt about 690 cycles, a division 570, measured), so a step is the chain
// sqrt, division, FMA, whatever the width up to 32: the division of all a
// elements of the step's column and row is one warp instruction stream.  The
// two kernels it replaces also divided integers per element and ran the
// substitution as one dependent FMA chain per column: 20 x 20 27 + 20 us,
// 30 x 30 28 + 24 us, against 20 and 32 us.
template <int T, int R>
__global__ void __launch_bounds__(T, 1) k_chol_inv(const double* __restrict__ G, int a, double* __restrict__ X,
                                                int transposed, int* __restrict__ status, double drop_tol,
                                                int* __restrict__ dropped) {
    dependent_start();
    __shared__ double vec[2][kMaxDesign];  // step k's column below the diagonal, row up to it
    __shared__ double res[kMaxDesign];     // L_ik (i > k) and X_kj (j <= k)
    __shared__ double diag[kMaxDesign];
    __shared__ double wmax[T / 32];
    const int tid = threadIdx.x, ne = a * (a + 1) / 2;
    int ij[R];  // i << 16 | j; -1: no element
    double val[R];
#pragma unroll
    for (int m = 0; m < R; ++m) {
        const int e = tid + T * m;
        int i = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
        while (i * (i + 1) / 2 > e) --i;
        while ((i + 1) * (i + 2) / 2 <= e) ++i;
        const int j = e - i * (i + 1) / 2;
        ij[m] = e < ne ? (i << 16 | j) : -1;
        val[m] = e < ne ? G[i * a + j] : 0.0;
        if (e < ne && j == 0) vec[0][i] = val[m];
    }
    double dm = 0.0;
    for (int k = tid; k < a; k += T) {
        diag[k] = G[k * a + k];
        dm = fmax(dm, fabs(diag[k]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
    if ((tid & 31) == 0) wmax[tid >> 5] = dm;
    __syncthreads();
    double dmax = 0.0;
    for (int w = 0; w < T / 32; ++w) dmax = fmax(dmax, wmax[w]);
    int bad = 0;
    for (int k = 0; k < a; ++k) {
        const double* v = vec[k & 1];
        if (tid < ((a + 31) & ~31)) {  // whole warps: the pivot is formed by each of them
            double pv = v[k];
            bool drop = false;
            if (drop_tol >= 0.0) {
                if (!(pv > drop_tol * fabs(diag[k])) || !(pv > 1e-300)) { drop = true; ++bad; pv = 1.0; }
            } else if (!(pv > 1e-300 + 1e-28 * dmax)) {
                pv = 1e-28 * dmax + 1e-300;
                ++bad;
            }
            const double piv = sqrt(pv);
            if (tid < a) {
                double q = (tid == k ? 1.0 : v[tid]) / piv;
                if (drop && tid > k) q = 0.0;
                res[tid] = q;
                const double x = tid <= k ? q : 0.0;
                if (transposed) X[tid * a + k] = x;
                else X[k * a + tid] = x;
                if (tid == k && dropped) dropped[k] = drop ? 1 : 0;
            }
        }
        __syncthreads();
        double* nv = vec[(k + 1) & 1];
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const int i = ij[m] >> 16, j = ij[m] & 0xffff;
            if (i > k) {
                val[m] = fma(-res[i], res[j], j == k ? 0.0 : val[m]);
                if (i == k + 1) nv[j] = val[m];
                else if (j == k + 1) nv[i] = val[m];
            }
        }
        __syncthreads();
    }
    if (tid == 0 && status) status[0] = bad;
}

// k_chol_inv for wide matrices: the packed triangle in shared memory, a warp
// per row and step (lanes over its columns); bound by the a^3 / 3 FMAs on one
// SM's FP64 pipe (131 x 131: 0.39 + 0.46 ms in the two kernels, 0.55 ms so).
__global__ void __launch_bounds__(1024, 1) k_chol_inv_wide(const double* __restrict__ G, int a,
                                                           double* __restrict__ X, int transposed,
                                                           int* __restrict__ status, double drop_tol,
                                                           int* __restrict__ dropped) {
    dependent_start();
    extern __shared__ double P[];          // packed lower triangle
    __shared__ double res[kMaxDesign];
    __shared__ double diag[kMaxDesign];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int i = warp; i < a; i += 32)
        for (int j = lane; j <= i; j += 32) P[i * (i + 1) / 2 + j] = G[i * a + j];
    for (int k = tid; k < a; k += blockDim.x) diag[k] = G[k * a + k];
    __syncthreads();
    double dmax = 0.0;
    for (int k = 0; k < a; ++k) dmax = fmax(dmax, fabs(diag[k]));
    int bad = 0;
    for (int k = 0; k < a; ++k) {
        if (tid < ((a + 31) & ~31)) {
            double pv = P[k * (k + 1) / 2 + k];
            bool drop = false;
            if (drop_tol >= 0.0) {
                if (!(pv > drop_tol * fabs(diag[k])) || !(pv > 1e-300)) { drop = true; ++bad; pv = 1.0; }
            } else if (!(pv > 1e-300 + 1e-28 * dmax)) {
                pv = 1e-28 * dmax + 1e-300;
                ++bad;
            }
            const double piv = sqrt(pv);
            if (tid < a) {
                const double v = tid == k ? 1.0 : tid < k ? P[k * (k + 1) / 2 + tid] : P[tid * (tid + 1) / 2 + k];
                double q = v / piv;
                if (drop && tid > k) q = 0.0;
                res[tid] = q;
                const double x = tid <= k ? q : 0.0;
                if (transposed) X[tid * a + k] = x;
                else X[k * a + tid] = x;
                if (tid == k && dropped) dropped[k] = drop ? 1 : 0;
            }
        }
        __syncthreads();
        for (int i = k + 1 + warp; i < a; i += 32) {
            const double li = -res[i];
            double* row = P + i * (i + 1) / 2;
            for (int j = lane; j <= i; j += 32) row[j] = fma(li, res[j], j == k ? 0.0 : row[j]);
        }
        __syncthreads();
    }
    if (tid == 0 && status) status[0] = bad;
}

// LU with partial pivoting in smem; returns 0 if an exactly zero pivot was met.
__device__ bool lu_smem(double* S, int* piv, int a) {
    __shared__ int p_sh;
    __shared__ int ok;
    if (threadIdx.x == 0) ok = 1;
    __syncthreads();
    for (int k = 0; k < a; ++k) {
        if (threadIdx.x == 0) {
            int p = k;
            double best = fabs(S[k * a + k]);
            for (int i = k + 1; i < a; ++i) {
                const double v = fabs(S[i * a + k]);
                if (v > best) { best = v; p = i; }
            }
            p_sh = p;
            piv[k] = p;
            if (best == 0.0) ok = 0;
        }
        __syncthreads();
        if (!ok) return false;
        const int p = p_sh;
        if (p != k)
            for (int j = threadIdx.x; j < a; j += blockDim.x) {
                const double t = S[k * a + j];
                S[k * a + j] = S[p * a + j];
                S[p * a + j] = t;
            }
        __syncthreads();
        const double d = S[k * a + k];
        for (int i = k + 1 + threadIdx.x; i < a; i += blockDim.x) S[i * a + k] /= d;
        __syncthreads();
        const int rem = a - k - 1;
        for (int e = threadIdx.x; e < rem * rem; e += blockDim.x) {
            const int i = k + 1 + e / rem, j = k + 1 + e % rem;
            S[i * a + j] -= S[i * a + k] * S[k * a + j];
        }
        __syncthreads();
    }
    return true;
}

// safe_inv (src/testing.rs:996-1024): invert; on an exactly zero pivot add
// eps = 1e-8 * max(max|diag|, 1e-300) to the diagonal and retry.
// status: 0 ok, 1 regularised, 2 failed.  eps_used[0] = eps (0 if none).
// Matrices wider than kMaxSmall work in `work` (a x a doubles then a ints,
// global memory) instead of shared memory.
__global__ void k_inverse(const double* __restrict__ A, int a, double* __restrict__ X,
                          int* __restrict__ status, double* __restrict__ eps_used, double* __restrict__ work) {
    dependent_start();
    extern __shared__ double S_sm[];
    __shared__ int piv_sm[kMaxSmall];
    double* S = work ? work : S_sm;
    int* piv = work ? reinterpret_cast<int*>(work + (size_t)a * a) : piv_sm;
    __shared__ double eps;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (threadIdx.x == 0) {
            double dmax = 0.0;
            for (int k = 0; k < a; ++k) dmax = fmax(dmax, fabs(A[k * a + k]));
            dmax = fmax(dmax, 1e-300);
            eps = attempt == 0 ? 0.0 : 1e-8 * dmax;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < a * a; e += blockDim.x)
            S[e] = A[e] + ((e / a == e % a) ? eps : 0.0);
        __syncthreads();
        if (lu_smem(S, piv, a)) {
            // solve for each unit vector: one thread per column
            for (int cc = threadIdx.x; cc < a; cc += blockDim.x) {
                double* x = X;  // column cc written strided
                // b = P e_cc
                for (int i = 0; i < a; ++i) x[i * a + cc] = (i == cc) ? 1.0 : 0.0;
                for (int k = 0; k < a; ++k) {
                    const int p = piv[k];
                    if (p != k) {
                        const double t = x[k * a + cc];
                        x[k * a + cc] = x[p * a + cc];
                        x[p * a + cc] = t;
                    }
                }
                for (int i = 0; i < a; ++i) {
                    double s = x[i * a + cc];
                    for (int k = 0; k < i; ++k) s -= S[i * a + k] * x[k * a + cc];
                    x[i * a + cc] = s;
                }
                for (int i = a - 1; i >= 0; --i) {
                    double s = x[i * a + cc];
                    for (int k = i + 1; k < a; ++k) s -= S[i * a + k] * x[k * a + cc];
                    x[i * a + cc] = s / S[i * a + i];
                }
            }
            if (threadIdx.x == 0) {
                if (status) status[0] = attempt;
                if (eps_used) eps_used[0] = eps;
            }
            return;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (status) status[0] = 2;
        if (eps_used) eps_used[0] = eps;
    }
}

__global__ void k_add_diag(double* __restrict__ A, int a, double v) {
    dependent_start();
    for (int i = threadIdx.x; i < a; i += blockDim.x) A[i * a + i] += v;
}

// safe_inv of up to kMaxInverseJobs matrices, one CTA each, by Gauss-Jordan
// elimination of A + shift I (+ eps I) in shared memory, in place: column k,
// done with at step k, holds the inverse's column of the original row that
// the k-th pivot came from (its entries before step k are that identity
// column's, zeros and a one, so they need no storage).  The pivot search (first
// largest |value| in the column, from the diagonal down) and the updates of the
// rows below the pivot are those of lu_smem, so the pivots, and the exact-zero
// test that triggers the eps retry, are the LU's.  A job without X wants
// only that outcome: the rows above the pivot are left alone, a third of the
// work.
//
// Per step: the search on one warp (magnitudes compared as integers, not on the
// FP64 pipe), then every division of the step side by side (the factors of the
// rows, the scaled pivot row), then a x a FMAs, a warp per row.  Bound by one
// SM's FP64 pipe (two FMAs per cycle).
// Widest that one CTA takes (8 a^2 bytes of shared memory); a cluster above.  The
// inverses of 50 columns: 194 us in one CTA, 124 us in a cluster.
constexpr int kInvOneCta = 40;
struct InverseJobs {
    InverseJob job[kMaxInverseJobs];
};

// Inverses up to here are eliminated in shared memory; wider ones keep the LU's
// solves and their bits.
constexpr int kInvShared = 112;

// Order of the pivot candidates, lu_smem's: 1 + the bits of |x|, and 0 for NaN,
// which no comparison prefers; but a NaN on the diagonal, where the search starts,
// is passed by no other, and goes on into the inverse.  1 is an exact zero.
// Where it starts with the first of several columns nothing is left to invert:
// the matrix counts as singular (the factors of a sketch that broke down are NaN
// altogether), up to the widths that the LU does not take.
__device__ __forceinline__ unsigned long long pivot_key(double x, int i, int k, int a) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    if (u > 0x7ff0000000000000ull) return i == k && (k > 0 || a == 1 || a > kInvShared) ? ~0ull : 0ull;
    return u + 1ull;
}

__global__ void __launch_bounds__(1024, 1) k_inverse_jobs(const __grid_constant__ InverseJobs jobs) {
    dependent_start();
    extern __shared__ double S[];  // a x a
    __shared__ double f[kInvOneCta], prow[kInvOneCta];
    __shared__ int rowid[kInvOneCta], from[kInvOneCta];
    __shared__ double eps;
    __shared__ int p_sh, ok;
    const InverseJob& jb = jobs.job[blockIdx.x];
    const double* A = jb.A;
    const int a = jb.a, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    const bool inv = jb.X != nullptr;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (tid == 0) {
            double dmax = 0.0;
            for (int k = 0; k < a; ++k) dmax = fmax(dmax, fabs(A[k * a + k] + jb.shift));
            dmax = fmax(dmax, 1e-300);
            eps = attempt == 0 ? 0.0 : 1e-8 * dmax;
            ok = 1;
        }
        __syncthreads();
        for (int i = warp; i < a; i += nwarps)
            for (int j = lane; j < a; j += 32) S[i * a + j] = i == j ? (A[i * a + j] + jb.shift) + eps : A[i * a + j];
        for (int i = tid; i < a; i += blockDim.x) rowid[i] = i;
        __syncthreads();
        for (int k = 0; k < a; ++k) {
            if (warp == 0) {
                unsigned long long best = 0ull;
                int p = k;
                for (int i = k + lane; i < a; i += 32) {
                    const unsigned long long key = pivot_key(S[i * a + k], i, k, a);
                    if (key > best) { best = key; p = i; }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int op = __shfl_xor_sync(0xffffffffu, p, o);
                    if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
                }
                if (lane == 0) {
                    p_sh = p;
                    if (best <= 1ull) ok = 0;
                    from[k] = rowid[p];
                    rowid[p] = rowid[k];
                }
            }
            __syncthreads();
            if (!ok) break;
            const int p = p_sh;
            const double d = S[p * a + k];
            // the row factors on the first threads, the pivot row on the last
            // ones: row k takes the scaled pivot row, row p what was in row k
            if (tid < a) {
                const int i = tid;
                if (i != k) f[i] = S[(i == p ? k : i) * a + k] / d;
            }
            const int jt = (int)blockDim.x - 1 - tid;
            double scaled = 0.0;
            if (jt < a && jt != k) {
                const double pj = S[p * a + jt], kj = S[k * a + jt];
                prow[jt] = pj;
                if (inv) scaled = pj / d;
                if (p != k) S[p * a + jt] = kj;
                S[k * a + jt] = inv ? scaled : pj;
            }
            __syncthreads();
            const int i0 = inv ? 0 : k + 1, j0 = inv ? 0 : k + 1;
            for (int i = i0 + warp; i < a; i += nwarps) {
                double* row = S + i * a;
                if (i == k) {
                    if (lane == 0) row[k] = 1.0 / d;
                    continue;
                }
                const double fi = -f[i];
                for (int j = j0 + lane; j < a; j += 32) row[j] = j == k ? fi : fma(fi, prow[j], row[j]);
            }
            __syncthreads();
        }
        if (ok) {
            if (inv)
                for (int i = warp; i < a; i += nwarps)
                    for (int j = lane; j < a; j += 32) jb.X[i * a + from[j]] = S[i * a + j];
            if (tid == 0) {
                jb.status[0] = attempt;
                jb.eps[0] = eps;
            }
            return;
        }
        __syncthreads();
    }
    if (tid == 0) {
        jb.status[0] = 2;
        jb.eps[0] = eps;
    }
}

// The same elimination for wide matrices, a job to a cluster of kInvCluster CTAs:
// column j lives column-major in the shared memory of CTA j mod kInvCluster.  Step
// k's owner searches its column and divides it, and leaves the pivot, its row and
// the row factors with every CTA (two sets of them, for even and odd steps: a step's
// are read until the next one's barrier); then each CTA updates its columns, a warp
// per column.  One SM spent a^2 FMAs of its FP64 pipe per step: two launches with
// designs of 100 and 131 columns took 1.41 ms, 0.78 ms so.
constexpr int kInvCluster = 8;
__global__ void __launch_bounds__(1024, 1) k_inverse_cluster(const __grid_constant__ InverseJobs jobs) {
    dependent_start();
    extern __shared__ double S[];  // the CTA's columns, a long each
    __shared__ double f[2][kMaxDesign], piv[2];
    __shared__ int prow[2], found[2];
    __shared__ int rowid[kMaxDesign], from[kMaxDesign];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const InverseJob& jb = jobs.job[blockIdx.x / kInvCluster];
    const double* A = jb.A;
    const int a = jb.a, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    const int ncol = (a - rank + kInvCluster - 1) / kInvCluster;  // columns rank, rank + 8 ..
    const bool inv = jb.X != nullptr;
    for (int attempt = 0; attempt < 2; ++attempt) {
        double dmax = 0.0;
        for (int k = lane; k < a; k += 32) dmax = fmax(dmax, fabs(A[k * a + k] + jb.shift));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        dmax = fmax(dmax, 1e-300);
        const double eps = attempt == 0 ? 0.0 : 1e-8 * dmax;
        for (int e = tid; e < ncol * a; e += blockDim.x) {
            const int jl = e / a, i = e - jl * a, j = rank + kInvCluster * jl;
            S[e] = i == j ? (A[i * a + j] + jb.shift) + eps : A[i * a + j];
        }
        for (int i = tid; i < a; i += blockDim.x) rowid[i] = i;
        bool ok = true;
        cluster.sync();  // every CTA runs, and is done with the last attempt's sets
        for (int k = 0; k < a; ++k) {
            const int b = k & 1;
            if (rank == k % kInvCluster) {
                const double* col = S + (k / kInvCluster) * a;
                if (warp == 0) {
                    unsigned long long best = 0ull;
                    int p = k;
                    for (int i = k + lane; i < a; i += 32) {
                        const unsigned long long key = pivot_key(col[i], i, k, a);
                        if (key > best) { best = key; p = i; }
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                        const int op = __shfl_xor_sync(0xffffffffu, p, o);
                        if (ob > best || (ob == best && op < p)) { best = ob; p = op; }
                    }
                    if (lane < kInvCluster) {
                        cluster.map_shared_rank(prow, lane)[b] = p;
                        cluster.map_shared_rank(found, lane)[b] = best > 1ull;
                        cluster.map_shared_rank(piv, lane)[b] = col[p];
                    }
                }
                __syncthreads();
                const int p = prow[b];
                const double d = piv[b];
                for (int i = tid; i < a; i += blockDim.x) {
                    if (i == k) continue;
                    const double fi = col[i == p ? k : i] / d;
#pragma unroll
                    for (int c = 0; c < kInvCluster; ++c) cluster.map_shared_rank(f[b], c)[i] = fi;
                }
            }
            cluster.sync();
            ok = found[b] != 0;
            if (!ok) break;
            const int p = prow[b];
            const double d = piv[b];
            if (tid == 0) {
                from[k] = rowid[p];
                rowid[p] = rowid[k];
            }
            for (int jl = warp; jl < ncol; jl += nwarps) {
                const int j = rank + kInvCluster * jl;
                double* col = S + jl * a;
                if (j == k) {
                    if (!inv) continue;
                    for (int i = lane; i < a; i += 32) col[i] = i == k ? 1.0 / d : -f[b][i];
                    continue;
                }
                if (!inv && j < k) continue;
                const double pj = col[p], kj = col[k];
                __syncwarp();
                for (int i = (inv ? 0 : (k & ~31)) + lane; i < a; i += 32) {
                    if (i == k) col[i] = inv ? pj / d : pj;
                    else if (inv || i > k) col[i] = fma(-f[b][i], pj, i == p ? kj : col[i]);
                }
            }
            __syncthreads();
        }
        if (ok) {
            if (inv)
                for (int e = tid; e < ncol * a; e += blockDim.x) {
                    const int jl = e / a, i = e - jl * a;
                    jb.X[i * a + from[rank + kInvCluster * jl]] = S[e];
                }
            if (tid == 0 && rank == 0) {
                jb.status[0] = attempt;
                jb.eps[0] = eps;
            }
            return;
        }
        if (attempt == 1 && tid == 0 && rank == 0) {
            jb.status[0] = 2;
            jb.eps[0] = eps;
        }
    }
}

// Columns that k_jacobi_svd gives one CTA; wider ones go to a cluster.  A solve
// with its copies, one CTA against eight: 30 columns 601 and 651 us, 33 columns 848
// and 870, 40 columns 1107 and 1018 (and one CTA holds a column in one element per
// lane up to 32).
constexpr int kEighOneCta = 32;
constexpr int kEighCluster = 8;
constexpr size_t kEighClusterSmem = 200 << 10;  // beside 25 KB of static arrays
// with those arrays a launch passes 48 KB before its dynamic part does
constexpr size_t kEighLimit = (48 << 10) + 1;

__device__ __forceinline__ float warp_sumf(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// x, unknown to the compiler: a sum that starts from plain(0) of one product
// stays a fused multiply-add with zero, whatever the trip count
__device__ __forceinline__ float plain(float x) { asm("" : "+f"(x)); return x; }
__device__ __forceinline__ double plain(double x) { asm("" : "+d"(x)); return x; }

// warp_sum of four values at once, in the same order of additions: the lanes
// split over the values in the first two steps, so that the sums take six FP64
// additions of the warp instead of twenty.  The lane's result is value
// 2 (lane >= 16) + (lane / 8 odd).
__device__ __forceinline__ double warp_sum4(const double (&v)[4]) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16, odd = lane & 8;
    double a = up ? v[2] : v[0], b = up ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
    b += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
    double t = odd ? b : a;
    t += __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// the two halves of a cluster barrier: what a thread reads or writes before its
// arrival comes before what any thread does after its wait
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// slot of the round-robin tournament of m (even) players: player 0 fixed, the
// others rotate
__device__ __forceinline__ int tournament_slot(int idx, int round, int m) {
    if (idx == 0) return 0;
    int s = idx - 1 + round;
    if (s >= m - 1) s -= m - 1;
    return 1 + s;
}

// FP32 one-sided Jacobi sweeps with accumulated V, until a sweep rotates nothing
// or max_sweeps.  column(c) is column c of M (ap long) and `to_v` floats behind
// it that of V; the NC CTAs share the pairs of a round, a warp per pair, NR
// elements of a column per lane (two at least: a lone product would be fused into
// the sum over the lanes).  A round is a chain of five divisions and square
// roots: the angle is computed beside the test of whether it is needed, and the
// columns are read once.  rotated: a flag in each CTA for even and for odd sweeps.
template <int NC, int NR, class Column, class Sync>
__device__ void jacobi_sweeps32(Column column, int to_v, int ap, int rank, float tol, int max_sweeps, int* rotated,
                                float abs_tol, Sync sync_all) {
    const int lane = threadIdx.x & 31, nwarps = NC * (blockDim.x >> 5);
    const int warp = rank + NC * (threadIdx.x >> 5);
    const int npairs = ap / 2;
    for (int sweep = 0; sweep < max_sweeps; ++sweep) {
        int* flag = rotated + (sweep & 1);
        for (int round = 0; round < ap - 1; ++round) {
            for (int pr = warp; pr < npairs; pr += nwarps) {
                const int s0 = tournament_slot(pr, round, ap), s1 = tournament_slot(ap - 1 - pr, round, ap);
                float* mp = column(min(s0, s1));
                float* mq = column(max(s0, s1));
                float x[NR], y[NR], vx[NR], vy[NR];
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    const int r = lane + 32 * q;
                    x[q] = r < ap ? mp[r] : 0.f;
                    y[q] = r < ap ? mq[r] : 0.f;
                    if constexpr (NC > 1) {  // another CTA's memory is far: V's columns come along
                        vx[q] = r < ap ? mp[to_v + r] : 0.f;
                        vy[q] = r < ap ? mq[to_v + r] : 0.f;
                    }
                }
                float al = 0.f, be = 0.f, ga = 0.f;
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    al += x[q] * x[q];
                    be += y[q] * y[q];
                    ga += x[q] * y[q];
                }
                al = warp_sumf(al);
                be = warp_sumf(be);
                ga = warp_sumf(ga);
                const float zeta = (be - al) / (2 * ga);
                const float bound = tol * sqrtf(al * be);
                const float t = (zeta >= 0 ? 1.f : -1.f) / (fabsf(zeta) + sqrtf(1.f + zeta * zeta));
                const float cs = 1.f / sqrtf(1.f + t * t), sn = cs * t;
                const float g = fabsf(ga);
                if (!(g > bound && g > 1e-37f && g > abs_tol)) continue;
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    const int r = lane + 32 * q;
                    if (r >= ap) continue;
                    if constexpr (NC == 1) {
                        vx[q] = mp[to_v + r];
                        vy[q] = mq[to_v + r];
                    }
                    mp[r] = cs * x[q] - sn * y[q];
                    mq[r] = sn * x[q] + cs * y[q];
                    mp[to_v + r] = cs * vx[q] - sn * vy[q];
                    mq[to_v + r] = sn * vx[q] + cs * vy[q];
                }
                if (lane == 0) *flag = 1;
            }
            // the next sweep's flag: every CTA has read it (a round has ended since)
            if (round == ap - 2 && threadIdx.x == 0) rotated[(sweep & 1) ^ 1] = 0;
            sync_all();
        }
        if constexpr (NC == 1) {
            const int any = *flag;
            __syncthreads();
            if (!any) break;
        } else {
            const int* f = lane < NC ? cooperative_groups::this_cluster().map_shared_rank(flag, lane) : flag;
            if (!__any_sync(0xffffffffu, *f)) break;
        }
    }
}

// Classical Gram-Schmidt, twice, of the ap columns of column-major Vs (FP64);
// acc: ap x ap scratch.  Column j's first pass takes its products with the
// column as it came in, so it runs ahead: as soon as column i is final, its
// part leaves every later column, the next one first and the others (warps
// from kTrail on) while the next one's second pass sums its chain and its norm.
// FP64 instructions hold a scheduler for 64 cycles whatever the lanes active,
// so the dot products are summed four to a warp.
constexpr int kTrail = 4;
template <int NR>
__device__ void gs_columns(double* Vs, double* acc, int ap, double* dots) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    constexpr int kChainWarps = NR < kTrail ? NR : kTrail;
    for (int e = threadIdx.x; e < ap * ap; e += blockDim.x) acc[e] = Vs[e];
    __syncthreads();
    // the products of NR elements a lane with four columns from col on (cols past `end` as zero)
    auto dot4 = [&](const double* cols, int col, int end, const double (&v)[NR], double (&t)[4]) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            t[m] = plain(0.0);
            if (col + m < end) {
                const double* c = cols + (col + m) * ap;
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t[m] += c[lane + 32 * q] * v[q];
            }
        }
    };
    auto load = [&](const double* c, double (&v)[NR]) {
#pragma unroll
        for (int q = 0; q < NR; ++q) v[q] = lane + 32 * q < ap ? c[lane + 32 * q] : 0.0;
    };
    for (int j = 0; j < ap; ++j) {
        double* vj = Vs + j * ap;
        double* aj = acc + j * ap;
        if (j > 0) {
            if (warp == 0) {  // the last term of the column's first pass
                const double* vi = vj - ap;
                double t = plain(0.0);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t += vi[lane + 32 * q] * vj[lane + 32 * q];
                t = warp_sum(t);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) aj[lane + 32 * q] -= t * vi[lane + 32 * q];
            }
            __syncthreads();
            // the second pass's products
            for (int i = 4 * warp; i < j; i += 4 * nwarps) {
                double v[NR], t[4];
                load(aj, v);
                dot4(Vs, i, j, v, t);
                const double s = warp_sum4(t);
                if ((lane & 7) == 0 && i + (lane >> 3) < j) dots[i + (lane >> 3)] = s;
            }
            __syncthreads();
        }
        if (warp < kChainWarps) {
            double s[NR];
#pragma unroll
            for (int q = 0; q < NR; ++q) s[q] = 0.0;
#pragma unroll
            for (int q = 0; q < (NR + kChainWarps - 1) / kChainWarps; ++q) {
                const int r = lane + 32 * (warp + q * kChainWarps);
                if (r < ap) {
                    double t = aj[r];
#pragma unroll 4
                    for (int i = 0; i < j; ++i) t -= dots[i] * Vs[i * ap + r];
                    if (kChainWarps == 1) s[q] = t;
                    else vj[r] = t;
                }
            }
            if (kChainWarps > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * kChainWarps) : "memory");
            if (warp == 0) {
                if (kChainWarps > 1) load(vj, s);
                double t = plain(0.0);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t += s[q] * s[q];
                t = warp_sum(t);
                const double inv = t > 0.0 ? 1.0 / sqrt(t) : 0.0;
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) vj[lane + 32 * q] = s[q] * inv;
            }
        } else if (warp >= kTrail && j > 0) {
            // column j - 1 leaves the columns behind j
            const double* vi = vj - ap;
            double v[NR], t[4];
            load(vi, v);
            for (int k = j + 1 + 4 * (warp - kTrail); k < ap; k += 4 * (nwarps - kTrail)) {
                dot4(Vs, k, ap, v, t);
                const double s = warp_sum4(t);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double d = __shfl_sync(0xffffffffu, s, 8 * m);
                    if (k + m < ap) {
                        double* ak = acc + (k + m) * ap;
#pragma unroll
                        for (int q = 0; q < NR; ++q)
                            if (lane + 32 * q < ap) ak[lane + 32 * q] -= d * v[q];
                    }
                }
            }
        }
        __syncthreads();
    }
}

// gs_columns over a cluster: column k and its running first pass belong to CTA k mod
// kEighCluster (own: the first passes, the columns as they came in, the final
// ones, `area` doubles each), which gives the second pass's products with its final
// columns; the chain and the norm stay with the first CTA, where the columns are
// put together (vec).  Per column the owner ends its first pass and hands it to all
// (cur), all hand their products to the first, and that one the final column to
// all (last, for even and odd columns): three barriers.
template <int NR>
__device__ void gs_cluster(double* own, int area, double* vec, int ap, double* dots, double* cur,
                           double (*last)[kMaxDesign]) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr int kN = kEighCluster;
    const int rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    constexpr int kChainWarps = NR < kTrail ? NR : kTrail;
    double *acc = own, *orig = own + area, *fin = own + 2 * area;
    auto load = [&](const double* c, double (&v)[NR]) {
#pragma unroll
        for (int q = 0; q < NR; ++q) v[q] = lane + 32 * q < ap ? c[lane + 32 * q] : 0.0;
    };
    // products of v with four of the CTA's columns from slot s on (slots past `end` as zero)
    auto dot4 = [&](const double* cols, int s, int end, const double (&v)[NR], double (&t)[4]) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            t[m] = plain(0.0);
            if (s + m < end) {
                const double* c = cols + (s + m) * ap;
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t[m] += c[lane + 32 * q] * v[q];
            }
        }
    };
    auto to_all = [&](double* dst, const double (&v)[NR]) {
#pragma unroll
        for (int c = 0; c < kN; ++c) {
            double* d = cluster.map_shared_rank(dst, c);
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (lane + 32 * q < ap) d[lane + 32 * q] = v[q];
        }
    };
    const int slots = (ap - rank + kN - 1) / kN;
    for (int j = 0; j < ap; ++j) {
        const double* prev = last[(j - 1) & 1];
        if (j > 0 && rank == (j - 1) % kN)
            for (int r = tid; r < ap; r += blockDim.x) fin[(j - 1) / kN * ap + r] = prev[r];
        if (rank == j % kN && warp == 0) {
            double x[NR];
            load(acc + j / kN * ap, x);
            if (j > 0) {  // the last term of the column's first pass
                const double* vj = orig + j / kN * ap;
                double t = plain(0.0);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t += prev[lane + 32 * q] * vj[lane + 32 * q];
                t = warp_sum(t);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) x[q] -= t * prev[lane + 32 * q];
            }
            to_all(cur, x);
        }
        cluster.sync();
        const int done = j > rank ? (j - rank + kN - 1) / kN : 0;  // the CTA's final columns
        for (int s = 4 * warp; s < done; s += 4 * nwarps) {
            double v[NR], t[4];
            load(cur, v);
            dot4(fin, s, done, v, t);
            const double d = warp_sum4(t);
            if ((lane & 7) == 0 && s + (lane >> 3) < done)
                cluster.map_shared_rank(dots, 0)[rank + kN * (s + (lane >> 3))] = d;
        }
        cluster.sync();
        const int w = rank == 0 ? warp - kTrail : warp, nw = rank == 0 ? nwarps - kTrail : nwarps;
        if (rank == 0 && warp < kChainWarps) {
            double* vj = vec + j * ap;
#pragma unroll
            for (int q = 0; q < (NR + kChainWarps - 1) / kChainWarps; ++q) {
                const int r = lane + 32 * (warp + q * kChainWarps);
                if (r < ap) {
                    double t = cur[r];
#pragma unroll 4
                    for (int i = 0; i < j; ++i) t -= dots[i] * vec[i * ap + r];
                    vj[r] = t;
                }
            }
            if (kChainWarps > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * kChainWarps) : "memory");
            if (warp == 0) {
                double x[NR];
                load(vj, x);
                double t = plain(0.0);
#pragma unroll
                for (int q = 0; q < NR; ++q)
                    if (lane + 32 * q < ap) t += x[q] * x[q];
                t = warp_sum(t);
                const double inv = t > 0.0 ? 1.0 / sqrt(t) : 0.0;
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    x[q] *= inv;
                    if (lane + 32 * q < ap) vj[lane + 32 * q] = x[q];
                }
                to_all(last[j & 1], x);
            }
        } else if (w >= 0 && j > 0) {
            // column j - 1 leaves the columns behind j
            double v[NR], t[4];
            load(prev, v);
            const int first = j >= rank ? (j - rank) / kN + 1 : 0;
            for (int s = first + 4 * w; s < slots; s += 4 * nw) {
                dot4(orig, s, slots, v, t);
                const double d4 = warp_sum4(t);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const double d = __shfl_sync(0xffffffffu, d4, 8 * m);
                    if (s + m < slots) {
                        double* ak = acc + (s + m) * ap;
#pragma unroll
                        for (int q = 0; q < NR; ++q)
                            if (lane + 32 * q < ap) ak[lane + 32 * q] -= d * v[q];
                    }
                }
            }
        }
        cluster.sync();
    }
}

// Eigen-decomposition of a symmetric positive semi-definite a x a matrix
// (a <= kMaxDesign; the Gram matrices of Step 0, the RSVD and the NMF probe) in
// NC CTAs: A V = V diag(sig), sig descending, V orthonormal; A is overwritten by
// V (its left singular vectors).
//
// GB300 runs FP64 at a small fraction of its FP32 rate, so the bulk of the
// rotation work runs as FP32 one-sided Jacobi sweeps (pairs in parallel,
// round-robin order) to ~1e-5 (at most 12 sweeps: with Gram matrices of
// condition 1e6 and more, FP32 rounding keeps rotating the small columns, and
// the FP64 phase converges quadratically from there anyway); V is
// re-orthonormalised in FP64 (Gram-Schmidt, twice) and B = V^T A V formed in
// FP64.  B is then diagonal up to ~1e-5 of its norm, and two-sided cyclic Jacobi
// sweeps in FP64 (Golub & Van Loan, Algorithm 8.5.2 with the parallel
// round-robin ordering) finish it -- quadratic convergence, typically two sweeps
// -- accumulating their rotations into R; V <- V R and a final Gram-Schmidt.
// Jacobi rotations are bounded (|tan| <= 1), so clusters of equal or nearly
// equal eigenvalues need no special case.  Eigenvalues are v_j^T A v_j of the
// final vectors.
//
// Every round of the FP64 sweeps is the latency of an angle (five divisions and
// square roots) plus the rotations of ap^2 elements at a sixteenth of the FP32
// rate.  One CTA holds it all in shared memory up to kEighOneCta columns.  Wider
// ones run as a cluster of eight: the FP32 matrices' and B's columns and R's rows
// are spread over the CTAs' shared memory, a round's pairs and 2 x 2 blocks are
// shared out and read and written there, and the products take a share of the
// columns each; of Gram-Schmidt the chains and norms stay with the first CTA.
// A solve with its copies (45 us), before and so: 13 columns 275 and 235 us, 20
// 461 and 348, 50 2457 and 1413, 100 14.1 and 4.2 ms, 256 221 and 53 ms (the wait in
// the middle of a round is 1 to 3 % of these).
template <int NC, int NR>
__global__ void __launch_bounds__(1024, 1) k_jacobi_svd(double* __restrict__ A, int a, double* __restrict__ V,
                                                        double* __restrict__ sig, double* ws, long long hold) {
    dependent_start();
    extern __shared__ double sm_dyn[];
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = NC > 1 ? (int)cluster.block_rank() : 0;
    // all CTAs' writes before it are seen by all after it
    auto sync_all = [&]() {
        if (NC > 1) cluster.sync();
        else __syncthreads();
    };
    const int ap = a + (a & 1);     // even number of columns (padded column is zero)
    const int share = (ap + NC - 1) / NC;  // columns (rows of R) of one CTA
    const int c0 = min(ap, rank * share), c1 = min(ap, c0 + share), nc = c1 - c0;
    const int sq = ap * ap;
    // One CTA: three squares of shared memory -- Gram-Schmidt's scratch, T and R;
    // the vectors; the FP32 matrices, B and V R.  A cluster: three squares of
    // global memory for what the CTAs pass on, the first CTA's vectors in shared
    // memory where they fit, and in each a share of the FP32 matrices, then of
    // Gram-Schmidt's columns, then of T or R, and of B.
    double *vec, *scratch = nullptr, *fp32, *T, *Bs, *R, *VR;
    if (NC == 1) {
        scratch = T = R = sm_dyn;
        vec = sm_dyn + sq;
        fp32 = Bs = VR = sm_dyn + 2 * sq;
    } else {
        const bool fits = 2 * (size_t)sq * sizeof(double) <= kEighClusterSmem;
        vec = fits ? sm_dyn + sq : ws + sq;
        fp32 = T = R = sm_dyn;
        Bs = sm_dyn + share * ap;
        VR = ws;
    }
    double* vecs = NC == 1 ? vec : ws + sq;  // the vectors where every CTA reads them
    float* M32 = reinterpret_cast<float*>(fp32);  // the share's columns of M, then of V
    const int to_v = share * ap;
    // Gram-Schmidt over the cluster: the columns rank, rank + NC .. , `area` doubles of them
    const int area = share * ap, mine = (ap - rank + NC - 1) / NC * ap;
    __shared__ int rotated, rotated32[2], nact;
    __shared__ double sg[kMaxDesign];
    __shared__ double dots[kMaxDesign];
    __shared__ double bmax;
    __shared__ int order[kMaxDesign];
    __shared__ int jp[2][kMaxDesign / 2], jq[2][kMaxDesign / 2];
    __shared__ double jc[2][kMaxDesign / 2], js[2][kMaxDesign / 2];
    __shared__ double* bcol[kMaxDesign];  // columns of B, wherever they are
    __shared__ float* mcol[kMaxDesign];   // and of the FP32 matrix
    __shared__ int act[kMaxDesign], rest[kMaxDesign], actflag[kMaxDesign];
    __shared__ float colmax2;
    __shared__ double cur[NC > 1 ? kMaxDesign : 1], last[NC > 1 ? 2 : 1][kMaxDesign];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    // phase 1: FP32 sweeps
    for (int e = threadIdx.x; e < nc * ap; e += blockDim.x) {
        const int col = c0 + e / ap, row = e % ap;
        M32[e] = (row < a && col < a) ? (float)A[row * a + col] : 0.f;
        M32[to_v + e] = (row == col) ? 1.f : 0.f;
    }
    for (int cc = threadIdx.x; cc < ap; cc += blockDim.x) {
        bcol[cc] = NC == 1 ? Bs + cc * ap : cluster.map_shared_rank(Bs, cc / share) + (cc % share) * ap;
        mcol[cc] = NC == 1 ? M32 + cc * ap : cluster.map_shared_rank(M32, cc / share) + (cc % share) * ap;
    }
    // FP32 resolution of the whole matrix: couplings below 1e-7 of the largest
    // squared column norm are left to the FP64 sweeps (columns of a rank-deficient
    // Gram that are zero up to FP32 rounding would otherwise keep rotating
    // until the sweep limit)
    if (threadIdx.x == 0) {
        colmax2 = 0.f;
        rotated32[0] = rotated32[1] = 0;
    }
    sync_all();
    for (int cc = warp; cc < ap; cc += nwarps) {
        float t = 0.f;
        for (int r = lane; r < a; r += 32) t += mcol[cc][r] * mcol[cc][r];
        t = warp_sumf(t);
        if (lane == 0) atomicMax(reinterpret_cast<int*>(&colmax2), __float_as_int(t));
    }
    sync_all();
    jacobi_sweeps32<NC, (NR > 2 ? NR : 2)>([&](int cc) { return NC == 1 ? M32 + cc * ap : mcol[cc]; }, to_v, ap,
                                          rank, 1.0e-5f, 12, rotated32, 1e-7f * colmax2, sync_all);
    sync_all();
    // phase 2: FP64 orthonormal V
    if constexpr (NC == 1) {
        for (int e = threadIdx.x; e < sq; e += blockDim.x) vec[e] = (double)mcol[e / ap][to_v + e % ap];
        __syncthreads();
        gs_columns<NR>(vec, scratch, ap, dots);
    } else {
        for (int e = threadIdx.x; e < mine; e += blockDim.x)
            sm_dyn[area + e] = (double)mcol[rank + NC * (e / ap)][to_v + e % ap];
        sync_all();  // the FP32 matrices are done with
        for (int e = threadIdx.x; e < mine; e += blockDim.x) sm_dyn[e] = sm_dyn[area + e];
        __syncthreads();
        gs_cluster<NR>(sm_dyn, area, vec, ap, dots, cur, last);
        if (rank == 0 && vecs != vec)
            for (int e = threadIdx.x; e < sq; e += blockDim.x) vecs[e] = vec[e];
    }
    sync_all();
    // phase 3: the share's columns of T = A V and of B = V^T T
    for (int e = threadIdx.x; e < nc * ap; e += blockDim.x) {
        const int col = c0 + e / ap, row = e % ap;
        double t = 0.0;
        if (row < a)
            for (int k = 0; k < a; ++k) t += A[row * a + k] * vecs[col * ap + k];
        T[e] = t;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nc * ap; e += blockDim.x) {
        const int col = e / ap, row = e % ap;
        double t = 0.0;
        for (int k = 0; k < ap; ++k) t += vecs[row * ap + k] * T[col * ap + k];
        Bs[e] = t;  // B[col * ap + row] = v_row^T A v_col
    }
    sync_all();
    if (warp == 0) {
        double m = 0.0;
        for (int j = lane; j < ap; j += 32) m = fmax(m, fabs(bcol[j][j]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) bmax = m;
    }
    // phase 4: FP64 two-sided Jacobi on B, rotations accumulated in R (the
    // share's rows, column-major).
    // Each sweep pairs only the active columns, those with an off-diagonal
    // entry above the skip level, in the round-robin order over them: a
    // column whose couplings are all at that level stays there while the
    // others rotate (a rotation of p and q mixes B_ip and B_iq and keeps
    // their norm), and the sweeps after the first usually have a few
    // columns left, the ones of the small eigenvalues the FP32 phase could
    // not resolve -- a sweep over all columns costs ap - 1 rounds of block
    // barriers and FP64 rotation angles whatever the number rotated.
    for (int e = threadIdx.x; e < ap * nc; e += blockDim.x) R[e] = (e / nc == c0 + e % nc) ? 1.0 : 0.0;
    __syncthreads();
    const double skip = 4e-16 * bmax;  // off-diagonals at the rounding level of B
    const int np2 = ap / 2;            // pairs, those of columns at rest among them
    const int kshare = (np2 + NC - 1) / NC, k0 = min(np2, rank * kshare), nk = min(np2, k0 + kshare) - k0;
    // warps 0 .. angle_warps - 1 compute a round's angles; R's rotations run beside
    // them on the schedulers (warp mod 4) that no angle's chain is on
    const int angle_warps = (np2 + 31) / 32, free_sched = 4 - angle_warps;
    const int r_warps = free_sched ? nwarps / 4 * free_sched : nwarps - 4;
    const int r_warp = free_sched ? (warp & 3) < angle_warps ? -1 : (warp >> 2) * free_sched + (warp & 3) - angle_warps
                                  : warp - 4;
    int buf = 0;
    bool pending = false;  // the last round's rotations are not in R yet
    // R <- R J of the rotations in buffer b, by thread `t` of `step`
    auto rotate_r = [&](int b, int t, int step) {
        for (int e = t; e < np2 * nc; e += step) {
            const int k = e / nc, i = e - k * nc;
            const double cs = jc[b][k], sn = js[b][k];
            if (sn == 0.0) continue;
            double* rp = R + jp[b][k] * nc;
            double* rq = R + jq[b][k] * nc;
            const double x = rp[i], y = rq[i];
            rp[i] = cs * x - sn * y;
            rq[i] = sn * x + cs * y;
        }
    };
    for (int sweep = 0; sweep < 12; ++sweep) {
        if (threadIdx.x == 0) rotated = 0;
        for (int cc = c0 + warp; cc < c1; cc += nwarps) {
            bool any = false;
            for (int r = lane; r < ap; r += 32) any |= r != cc && fabs(bcol[cc][r]) > skip;
            any = __any_sync(0xffffffffu, any);
            if (lane < NC) {
                int* f = NC == 1 ? actflag : cluster.map_shared_rank(actflag, lane);
                f[cc] = any ? 1 : 0;
            }
        }
        sync_all();
        if (warp == 0) {  // the active columns in ascending order, and the others
            int run = 0, idle = 0;
            for (int base = 0; base < ap; base += 32) {
                const bool in = base + lane < ap, f = in && actflag[base + lane];
                const unsigned m = __ballot_sync(0xffffffffu, f), z = __ballot_sync(0xffffffffu, in && !f);
                if (f) act[run + __popc(m & ((1u << lane) - 1u))] = base + lane;
                else if (in) rest[idle + __popc(z & ((1u << lane) - 1u))] = base + lane;
                run += __popc(m);
                idle += __popc(z);
            }
            if (lane == 0) nact = run;
        }
        __syncthreads();
        const int na = nact;
        if (na < 2) break;
        const int nap = na + (na & 1);  // even; position na (odd na) pairs with a column at rest
        const int npairs = nap / 2;
        for (int round = 0; round < nap - 1; ++round) {
            // test hook: one CTA comes late to its reads
            if (NC > 1 && hold > 0 && rank == 1)
                for (const long long t0 = clock64(); clock64() - t0 < hold;) {}
            const int k = threadIdx.x;
            int pc = 0, qc = 0;
            bool meet = false;  // a pair of active columns
            double app = 0.0, aqq = 0.0, apq = 0.0;
            if (warp < angle_warps) {
                if (k < npairs) {
                    const int x = tournament_slot(k, round, nap), y = tournament_slot(nap - 1 - k, round, nap);
                    if (x < na && y < na) {
                        pc = act[x];
                        qc = act[y];
                        if (pc > qc) { const int t = pc; pc = qc; qc = t; }
                        meet = true;
                        app = bcol[pc][pc];
                        aqq = bcol[qc][qc];
                        apq = bcol[qc][pc];
                    } else {
                        pc = act[x < na ? x : y];
                        qc = rest[0];
                    }
                } else if (k < np2) {
                    pc = rest[(na & 1) + 2 * (k - npairs)];
                    qc = rest[(na & 1) + 2 * (k - npairs) + 1];
                }
            }
            // Every CTA forms every angle, from elements that lie with the CTAs that
            // rotate them below: no block is written before all have read.  The wait
            // is behind the angles, which take longer than the barrier.
            if (NC > 1) cluster_arrive();
            if (warp < angle_warps) {
                double cs = 1.0, sn = 0.0;
                if (meet && fabs(apq) > skip && apq != 0.0) {
                    const double tau = (aqq - app) / (2.0 * apq);
                    const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                    cs = 1.0 / sqrt(1.0 + t * t);
                    sn = t * cs;
                    rotated = 1;
                }
                if (k < np2) {
                    jp[buf][k] = pc; jq[buf][k] = qc; jc[buf][k] = cs; js[buf][k] = sn;
                }
            } else if (pending && r_warp >= 0) {
                rotate_r(buf ^ 1, 32 * r_warp + lane, 32 * r_warps);
            }
            __syncthreads();
            if (NC > 1) cluster_wait();
            // B <- J^T (B J), the 2 x 2 blocks of the share's pairs of columns
            // with every pair of rows
            for (int e = threadIdx.x; e < nk * np2; e += blockDim.x) {
                const int k = k0 + e / np2, l = e % np2;
                const double sk = js[buf][k], sl = js[buf][l];
                if (sk == 0.0 && sl == 0.0) continue;
                double* bp = bcol[jp[buf][k]];
                double* bq = bcol[jq[buf][k]];
                const int pr = jp[buf][l], qr = jq[buf][l];
                double pp = bp[pr], pq = bp[qr], qp = bq[pr], qq = bq[qr];
                if (sk != 0.0) {
                    const double cs = jc[buf][k], sn = sk;
                    double x = pp, y = qp;
                    pp = cs * x - sn * y;
                    qp = sn * x + cs * y;
                    x = pq; y = qq;
                    pq = cs * x - sn * y;
                    qq = sn * x + cs * y;
                }
                if (sl != 0.0) {
                    const double cs = jc[buf][l], sn = sl;
                    double x = pp, y = pq;
                    pp = cs * x - sn * y;
                    pq = sn * x + cs * y;
                    x = qp; y = qq;
                    qp = cs * x - sn * y;
                    qq = sn * x + cs * y;
                }
                bp[pr] = pp; bp[qr] = pq; bq[pr] = qp; bq[qr] = qq;
            }
            sync_all();
            buf ^= 1;
            pending = true;
        }
        const int any = rotated;
        __syncthreads();
        if (!any) break;
    }
    if (pending) rotate_r(buf ^ 1, threadIdx.x, blockDim.x);
    // V <- V R
    double* Rall = R;
    if (NC > 1) {
        Rall = ws + 2 * sq;
        __syncthreads();
        for (int e = threadIdx.x; e < ap * nc; e += blockDim.x) Rall[(e / nc) * ap + c0 + e % nc] = R[e];
    }
    sync_all();
    for (int e = threadIdx.x; e < nc * ap; e += blockDim.x) {
        const int col = c0 + e / ap, row = e % ap;
        double t = 0.0;
        for (int i = 0; i < ap; ++i) t += vecs[i * ap + row] * Rall[col * ap + i];
        VR[col * ap + row] = t;
    }
    sync_all();
    double* fin = VR;
    if constexpr (NC == 1) {
        gs_columns<NR>(fin, scratch, ap, dots);
    } else {
        for (int e = threadIdx.x; e < mine; e += blockDim.x)
            sm_dyn[e] = sm_dyn[area + e] = VR[(rank + NC * (e / ap)) * ap + e % ap];
        __syncthreads();
        gs_cluster<NR>(sm_dyn, area, vec, ap, dots, cur, last);
        if (rank == 0 && vecs != vec)
            for (int e = threadIdx.x; e < sq; e += blockDim.x) vecs[e] = vec[e];
    }
    if (NC > 1) fin = vecs;
    sync_all();
    // phase 5: eigenvalues v_j^T A v_j, descending order
    for (int cc = c0 + warp; cc < c1; cc += nwarps) {
        double s = 0.0;
        for (int r = lane; r < a; r += 32) {
            double t = 0.0;
            for (int k = 0; k < a; ++k) t += A[r * a + k] * fin[cc * ap + k];
            s += fin[cc * ap + r] * t;
        }
        s = warp_sum(s);
        if (lane == 0) *(NC == 1 ? sg + cc : cluster.map_shared_rank(sg, 0) + cc) = fabs(s);
    }
    sync_all();
    if (rank != 0) return;
    // a column's place is the number of larger ones (compared as integers: no
    // value is negative); equal values, and NaN, are put where a selection sort
    // does, the first largest of the rest swapped to the front
    bool plain_order = true;
    for (int i = threadIdx.x; i < a; i += blockDim.x) {
        const long long key = __double_as_longlong(sg[i]);
        int place = 0;
        for (int j = 0; j < a; ++j) {
            const long long other = __double_as_longlong(sg[j]);
            place += other > key;
            plain_order = plain_order && (other != key || j == i);
        }
        plain_order = plain_order && !isnan(sg[i]);
        order[place] = i;
    }
    if (!__syncthreads_and(plain_order)) {
        if (threadIdx.x == 0) {
            for (int i = 0; i < a; ++i) order[i] = i;
            for (int i = 0; i < a; ++i) {
                int best = i;
                for (int j = i + 1; j < a; ++j)
                    if (sg[order[j]] > sg[order[best]]) best = j;
                const int t = order[i]; order[i] = order[best]; order[best] = t;
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < a * a; e += blockDim.x) {
        const int row = e / a, cc = e % a;
        V[e] = A[e] = fin[order[cc] * ap + row];
    }
    for (int cc = threadIdx.x; cc < a; cc += blockDim.x) sig[cc] = sg[order[cc]];
}

// SplitMix64 counter RNG + Box-Muller (identical stream definition in the
// CPU oracle): element (i, c) of a rows x cols matrix is draw i*cols+c.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_normal(uint64_t seed, uint64_t total, double* __restrict__ out) {
    dependent_start();
    const uint64_t key = mix64(seed + 0x9E3779B97F4A7C15ull);
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t a = mix64(key + (2 * t + 1) * 0x9E3779B97F4A7C15ull);
        const uint64_t b = mix64(key + (2 * t + 2) * 0x9E3779B97F4A7C15ull);
        const double u1 = ((double)(a >> 11) + 1.0) * 0x1.0p-53;
        const double u2 = (double)(b >> 11) * 0x1.0p-53;
        out[t] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
    }
}

__global__ void k_f64_to_f32_pad(const double* __restrict__ A, uint64_t m, int a, int lda,
                                 float* __restrict__ out, uint64_t m_pad, int ldo) {
    dependent_start();
    const uint64_t total = m_pad * ldo;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / ldo;
        const int cc = (int)(t - i * ldo);
        out[t] = (i < m && cc < a) ? (float)A[i * lda + cc] : 0.f;
    }
}

__global__ void k_f32_to_f64(const float* __restrict__ A, uint64_t m, int a, int lda,
                             double* __restrict__ out, int ldo) {
    dependent_start();
    const uint64_t total = m * a;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / a;
        const int cc = (int)(t - i * a);
        out[i * ldo + cc] = (double)A[i * lda + cc];
    }
}

__global__ void k_fill(double* __restrict__ x, uint64_t n, double v) {
    dependent_start();
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < n; t += (uint64_t)gridDim.x * blockDim.x)
        x[t] = v;
}

__global__ void k_transpose(const double* __restrict__ A, int rows, int cols, double* __restrict__ At) {
    dependent_start();
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < rows * cols; e += gridDim.x * blockDim.x) {
        const int i = e / cols, j = e % cols;
        At[j * rows + i] = A[e];
    }
}

__global__ void k_scale_cols(double* __restrict__ A, uint64_t m, int a, int lda,
                             const double* __restrict__ f) {
    dependent_start();
    const uint64_t total = m * a;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / a;
        const int cc = (int)(t - i * a);
        A[i * lda + cc] *= f[cc];
    }
}

// C = [1 | X | U] (n x (1+d+K))
__global__ void k_build_design(const double* __restrict__ X, int d, const double* __restrict__ U, int K,
                               uint64_t n, double* __restrict__ C) {
    dependent_start();
    const int w = 1 + d + K;
    const uint64_t total = n * w;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / w;
        const int cc = (int)(t - i * w);
        C[t] = cc == 0 ? 1.0 : (cc <= d ? X[i * d + cc - 1] : U[i * K + cc - 1 - d]);
    }
}

size_t smem_sq(int a) { return (size_t)a * a * sizeof(double); }

// rows of a narrow FP32 matrix the tiled kernels can take
bool narrow_tiled(const float* A, int lda) {
    return lda % 4 == 0 && lda <= 32 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
}

void set_smem(const void* fn, size_t bytes) { raise_dynamic_smem(fn, bytes); }

}  // namespace

// column means of a tall matrix: rows in ranges of kColRows per block, then
// the partials summed in order and divided by m (one block per column left
// too few blocks on the GPU: 30 blocks each walking 20 000 rows)
constexpr uint64_t kColRows = 2048;

__global__ void k_colsum_split(const double* __restrict__ A, uint64_t m, int a, int lda, uint64_t per,
                               double* __restrict__ part);

__global__ void k_mean_partials(const double* __restrict__ part, int splits, int a, uint64_t m,
                                double* __restrict__ out) {
    dependent_start();
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= a) return;
    double s = 0.0;
    for (int k = 0; k < splits; ++k) s += part[(uint64_t)k * a + col];
    out[col] = m ? s / (double)m : 0.0;
}

void launch_colmeans(Ctx& c, const double* A, uint64_t m, int a, int lda, double* out) {
    if (a == 0) return;
    if (m <= 2 * kColRows) {
        launch_next(c, k_colmeans, a, 256, 0, A, m, lda, out, 1);
        SLFMM_LAUNCHED(c, "k_colmeans");
        return;
    }
    const uint64_t splits = std::min<uint64_t>(ceil_div(m, kColRows), 512);
    const uint64_t per = ceil_div(m, splits);
    DBuf<double> part(splits * a, c.stream);
    launch_next(c, k_colsum_split, dim3(a, (unsigned)splits), 256, 0, A, m, a, lda, per, part.get());
    SLFMM_LAUNCHED(c, "k_colsum_split");
    launch_next(c, k_mean_partials, (unsigned)ceil_div((uint64_t)a, 128), 128, 0, part.get(), (int)splits, a, m,
                                                                                 out);
    SLFMM_LAUNCHED(c, "k_mean_partials");
}

// column sums of a tall matrix: row ranges of `per` rows in parallel, then
// the partials summed in order
__global__ void k_colsum_split(const double* __restrict__ A, uint64_t m, int a, int lda, uint64_t per,
                               double* __restrict__ part) {
    dependent_start();
    __shared__ double red[32];
    const int col = blockIdx.x;
    const uint64_t r0 = (uint64_t)blockIdx.y * per, r1 = min(m, r0 + per);
    double s = 0.0;
    for (uint64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) s += A[i * lda + col];
    s = block_sum(s, red);
    if (threadIdx.x == 0) part[(uint64_t)blockIdx.y * a + col] = s;
}

void launch_colsums(Ctx& c, const double* A, uint64_t m, int a, int lda, double* out) {
    if (a == 0) return;
    if (m <= 2 * kColRows) {
        launch_next(c, k_colmeans, a, 256, 0, A, m, lda, out, 0);
        SLFMM_LAUNCHED(c, "k_colsums");
        return;
    }
    const uint64_t splits = std::min<uint64_t>(ceil_div(m, m <= 65536 ? kColRows : 16384), 512);
    const uint64_t per = ceil_div(m, splits);
    DBuf<double> part(splits * a, c.stream);
    launch_next(c, k_colsum_split, dim3(a, (unsigned)splits), 256, 0, A, m, a, lda, per, part.get());
    SLFMM_LAUNCHED(c, "k_colsum_split");
    launch_sum_partials(c, part.get(), (int)splits, (uint64_t)a, out);
}

void launch_sum_partials(Ctx& c, const double* part, int splits, uint64_t count, double* out) {
    if (!count) return;
    if (splits >= 32) {
        launch_next(c, k_sum_partials_wide, (unsigned)std::min<uint64_t>(count, 65535), 128, 0, part, splits, count,
                                                                                             out);
        SLFMM_LAUNCHED(c, "k_sum_partials_wide");
        return;
    }
    launch_next(c, k_sum_partials, grid_for(c, count, 256), 256, 0, part, splits, count, out);
    SLFMM_LAUNCHED(c, "k_sum_partials");
}

void launch_center_cols(Ctx& c, double* A, uint64_t m, int a, int lda, const double* means) {
    if (a == 0 || m == 0) return;
    launch_next(c, k_center_cols, grid_for(c, m * a, 256), 256, 0, A, m, a, lda, means);
    SLFMM_LAUNCHED(c, "k_center_cols");
}

void launch_scale_cols_sd(Ctx& c, double* A, uint64_t m, int a, int lda) {
    if (a == 0) return;
    launch_next(c, k_scale_cols_sd, a, 256, 0, A, m, lda);
    SLFMM_LAUNCHED(c, "k_scale_cols_sd");
}

template <typename T>
static void atb_impl(Ctx& c, const T* A, int lda, const T* B, int ldb, uint64_t m, int a, int b,
                     double* out) {
    // FP64-bound (GB300 runs FP64 at a small fraction of FP32): enough row
    // splits that every SM holds a few CTAs (64 rows each at least)
    if (a > 0 && b > 0 && a * b <= 256 * 16 * 4 && a <= 128 && b <= 128) {
        const int ab = a * b;
        const int R = ab <= 256 ? 1 : ab <= 512 ? 2 : ab <= 1024 ? 4 : ab <= 2048 ? 8 : 16;
        const int blocks_o = (int)ceil_div((uint64_t)ab, (uint64_t)256 * R);
        uint64_t splits = std::max<uint64_t>(
            1, std::min<uint64_t>(ceil_div(m, 64), ceil_div((uint64_t)c.sm_count * 8, (uint64_t)blocks_o)));
        splits = std::min<uint64_t>(splits, 65535);
        const uint64_t per = round_up(ceil_div(std::max<uint64_t>(m, 1), splits), 32);
        splits = std::max<uint64_t>(1, ceil_div(m, per));
        DBuf<double> part(splits * ab, c.stream);
        const size_t smem = (size_t)32 * (a + b) * sizeof(double);
        dim3 grid(blocks_o, (unsigned)splits);
#define SLFMM_ATB_FLAT(RR)                                                                        \
    do {                                                                                          \
        raise_dynamic_smem((const void*)k_atb_flat<T, RR>, smem);                                 \
        launch_next(c, k_atb_flat<T, RR>, grid, 256, smem, A, lda, B, ldb, m, a, b, per, part.get()); \
    } while (0)
        switch (R) {
            case 1: SLFMM_ATB_FLAT(1); break;
            case 2: SLFMM_ATB_FLAT(2); break;
            case 4: SLFMM_ATB_FLAT(4); break;
            case 8: SLFMM_ATB_FLAT(8); break;
            default: SLFMM_ATB_FLAT(16); break;
        }
#undef SLFMM_ATB_FLAT
        SLFMM_LAUNCHED(c, "k_atb_flat");
        launch_sum_partials(c, part.get(), (int)splits, (uint64_t)ab, out);
        return;
    }
    const int ta = (int)ceil_div(a, 32), tb = (int)ceil_div(b, 32);
    uint64_t splits = std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(m, 64),
                                          ceil_div((uint64_t)c.sm_count * 8, (uint64_t)ta * tb)));
    splits = std::min<uint64_t>(splits, 65535);
    const uint64_t per = round_up(ceil_div(std::max<uint64_t>(m, 1), splits), 32);
    splits = std::max<uint64_t>(1, ceil_div(m, per));
    DBuf<double> part(splits * a * b, c.stream);
    dim3 grid(ta, tb, (unsigned)splits);
    launch_next(c, k_atb<T>, grid, 256, 0, A, lda, B, ldb, m, a, b, per, part.get());
    SLFMM_LAUNCHED(c, "k_atb");
    launch_sum_partials(c, part.get(), (int)splits, (uint64_t)a * b, out);
}

void launch_atb(Ctx& c, const double* A, int lda, const double* B, int ldb, uint64_t m, int a, int b,
                double* out) {
    atb_impl<double>(c, A, lda, B, ldb, m, a, b, out);
}

void launch_gram_f32(Ctx& c, const float* A, int lda, uint64_t m, int a, double* out) {
    if (a <= 32) {
        if (narrow_tiled(A, lda)) {
            const uint64_t tb = std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(m, (uint64_t)kNarrowTile),
                                                                        (uint64_t)c.sm_count));
            const size_t sm = kPipeRing + (size_t)(kPipeThreads / 32) * 32 * 32 * sizeof(double);
            DBuf<double> tpart(tb * a * a, c.stream);
            set_smem((const void*)k_gram_tile, sm);
            launch_next(c, k_gram_tile, (unsigned)tb, kPipeThreads, sm, A, lda, m, a, tpart.get());
            SLFMM_LAUNCHED(c, "k_gram_tile");
            launch_sum_partials(c, tpart.get(), (int)tb, (uint64_t)a * a, out);
            return;
        }
        const uint64_t runs = std::max<uint64_t>(1, ceil_div(m, (uint64_t)kGramRun));
        const uint64_t blocks = std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(runs, 8), (uint64_t)c.sm_count * 4));
        DBuf<double> part(blocks * a * a, c.stream);
        set_smem((const void*)k_gram_narrow, kGramNarrowSmem);
        launch_next(c, k_gram_narrow, (unsigned)blocks, 256, kGramNarrowSmem, A, lda, m, a, part.get());
        SLFMM_LAUNCHED(c, "k_gram_narrow");
        launch_sum_partials(c, part.get(), (int)blocks, (uint64_t)a * a, out);
        return;
    }
    const int ta = (int)ceil_div(a, 32);
    uint64_t splits = std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(m, 1024),
                                          ceil_div((uint64_t)c.sm_count * 8, (uint64_t)ta * ta)));
    splits = std::min<uint64_t>(splits, 65535);
    const uint64_t per = round_up(ceil_div(std::max<uint64_t>(m, 1), splits), 32);
    splits = std::max<uint64_t>(1, ceil_div(m, per));
    DBuf<double> part(splits * a * a, c.stream);
    dim3 grid(ta, ta, (unsigned)splits);
    launch_next(c, k_gram_f32, grid, 256, 0, A, lda, m, a, per, part.get());
    SLFMM_LAUNCHED(c, "k_gram_f32");
    launch_sum_partials(c, part.get(), (int)splits, (uint64_t)a * a, out);
}

void launch_gemm_small(Ctx& c, const double* A, int lda, uint64_t m, int a, const double* B, int ldb,
                       int b, double alpha, double beta, double* C, int ldc) {
    if (m == 0 || b == 0) return;
    // B in shared memory: column blocks of B (and C) for wide products
    const int bb = std::max(1, std::min(b, (int)((200 * 1024) / (sizeof(double) * (size_t)std::max(a, 1)))));
    for (int c0 = 0; c0 < b; c0 += bb) {
        const int nb = std::min(bb, b - c0);
        const size_t sm = (size_t)a * nb * sizeof(double);
        set_smem((const void*)k_gemm_small<double>, sm);
        launch_next(c, k_gemm_small<double>, grid_for(c, m * nb, 256), 256, sm, A, lda, m, a, B + c0, ldb, nb, alpha,
                                                                              beta, C + c0, ldc);
        SLFMM_LAUNCHED(c, "k_gemm_small");
    }
}

void launch_trmul_f32(Ctx& c, float* A, int lda, uint64_t m, int a, const double* Linv) {
    SLFMM_REQUIRE(a <= 64, SLFMM_ERR_BAD_ARG, "sketch width must be <= 64");
    if (m == 0) return;
    if (a <= 32) {
        if (narrow_tiled(A, lda)) {
            launch_next(c, k_trmul_rows, grid_for(c, ceil_div(m, (uint64_t)kTrmulRows), 256), 256, 0, A, lda, m, a,
                        Linv);
            SLFMM_LAUNCHED(c, "k_trmul_rows");
            return;
        }
        launch_next(c, k_trmul_narrow, grid_for(c, m, 32), 256, 0, A, lda, m, a, Linv);
        SLFMM_LAUNCHED(c, "k_trmul_narrow");
        return;
    }
    launch_next(c, k_trmul_f32<64>, grid_for(c, m, 128), 128, 0, A, lda, m, a, Linv);
    SLFMM_LAUNCHED(c, "k_trmul_f32");
}

// The small dense solvers keep the matrix in shared memory up to kMaxSmall
// columns and work in global memory (L2-resident) up to kMaxDesign.
void launch_cholesky(Ctx& c, double* A, int a, int* status, double drop_tol, int* dropped) {
    SLFMM_REQUIRE(a <= kMaxDesign, SLFMM_ERR_BAD_ARG, "matrix too large for the small Cholesky");
    if (a <= kMaxSmall) {
        set_smem((const void*)k_cholesky, smem_sq(a));
        launch_next(c, k_cholesky, 1, 512, smem_sq(a), A, a, status, drop_tol, dropped, nullptr);
    } else {
        DBuf<double> work((size_t)a * a, c.stream);
        launch_next(c, k_cholesky, 1, 1024, 0, A, a, status, drop_tol, dropped, work.get());
    }
    SLFMM_LAUNCHED(c, "k_cholesky");
}

// X = L^-1 (or its transpose) of the Cholesky factor of G.  The fused kernel
// keeps the packed triangle in registers up to 127 columns and in shared memory
// up to 236; wider designs take the two separate kernels, on a copy of G.
void launch_chol_inv(Ctx& c, const double* G, int a, double* X, bool transposed, int* status, double drop_tol,
                     int* dropped) {
    SLFMM_REQUIRE(a <= kMaxDesign, SLFMM_ERR_BAD_ARG, "matrix too large for the small Cholesky");
    if (a < 1) return;
    const int ne = a * (a + 1) / 2, tr = transposed ? 1 : 0;
#define SLFMM_CHOL_INV(T, R) launch_next(c, k_chol_inv<T, R>, 1, T, 0, G, a, X, tr, status, drop_tol, dropped)
    if (ne <= 256) SLFMM_CHOL_INV(256, 1);
    else if (ne <= 256 * 2) SLFMM_CHOL_INV(256, 2);
    else if (ne <= 256 * 4) SLFMM_CHOL_INV(256, 4);
    else if (ne <= 256 * 9) SLFMM_CHOL_INV(256, 9);
    else if (ne <= 512 * 16) SLFMM_CHOL_INV(512, 16);
    else if (ne * sizeof(double) <= 220 * 1024) {
        const size_t sm = ne * sizeof(double);
        set_smem((const void*)k_chol_inv_wide, sm);
        launch_next(c, k_chol_inv_wide, 1, 1024, sm, G, a, X, tr, status, drop_tol, dropped);
    } else {
        DBuf<double> L((size_t)a * a, c.stream), lower((size_t)a * a, c.stream);
        SLFMM_CUDA(cudaMemcpyAsync(L.get(), G, (size_t)a * a * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
        launch_cholesky(c, L.get(), a, status, drop_tol, dropped);
        launch_tri_inv_lower(c, L.get(), a, transposed ? lower.get() : X);
        if (transposed) launch_transpose(c, lower.get(), a, a, X);
        return;
    }
#undef SLFMM_CHOL_INV
    SLFMM_LAUNCHED(c, "k_chol_inv");
}

void launch_tri_inv_lower(Ctx& c, const double* L, int a, double* Linv) {
    SLFMM_REQUIRE(a <= kMaxDesign, SLFMM_ERR_BAD_ARG, "matrix too large for the triangular inverse");
    const bool sm = a <= kMaxSmall;
    if (sm) set_smem((const void*)k_tri_inv_lower, smem_sq(a));
    launch_next(c, k_tri_inv_lower, 1, sm ? 128 : 256, sm ? smem_sq(a) : 0, L, a, Linv, sm ? 1 : 0);
    SLFMM_LAUNCHED(c, "k_tri_inv_lower");
}

// The elimination in shared memory takes every status-only job, and inverses up
// to kInvShared columns.
static bool inverse_in_shared(const InverseJob& j) { return j.a <= (j.X ? kInvShared : kMaxDesign); }

void launch_inverses(Ctx& c, const InverseJob* jobs, int n) {
    SLFMM_REQUIRE(n <= kMaxInverseJobs, SLFMM_ERR_BAD_ARG, "too many matrices for one inversion launch");
    double work = 0.0;
    for (int i = 0; i < n; ++i) {
        SLFMM_REQUIRE(jobs[i].a <= kMaxDesign, SLFMM_ERR_BAD_ARG, "matrix too large for the small inverse");
        work += 2.0 * jobs[i].a * jobs[i].a * jobs[i].a;
    }
    ProfScope ps(c, "small_inverse", 0.0, work);
    InverseJobs js{};
    int m = 0, amax = 0;
    for (int i = 0; i < n; ++i)
        if (inverse_in_shared(jobs[i])) {
            js.job[m++] = jobs[i];
            amax = std::max(amax, jobs[i].a);
        }
    if (amax > kInvOneCta) {
        const size_t sm = ceil_div(amax, kInvCluster) * amax * sizeof(double);
        set_smem((const void*)k_inverse_cluster, std::max(sm, kEighLimit));
        launch_next_clusters(c, k_inverse_cluster, m, kInvCluster, 1024, sm, js);
        SLFMM_LAUNCHED(c, "k_inverse_cluster");
    } else if (m) {
        launch_next(c, k_inverse_jobs, m, 1024, smem_sq(amax), js);
        SLFMM_LAUNCHED(c, "k_inverse_jobs");
    }
    for (int i = 0; i < n; ++i) {
        const InverseJob& j = jobs[i];
        if (inverse_in_shared(j)) continue;
        DBuf<double> A;
        const double* src = j.A;
        if (j.shift != 0.0) {
            A.alloc((size_t)j.a * j.a, c.stream);
            SLFMM_CUDA(cudaMemcpyAsync(A.get(), j.A, A.bytes(), cudaMemcpyDeviceToDevice, c.stream));
            launch_next(c, k_add_diag, 1, 256, 0, A.get(), j.a, j.shift);
            SLFMM_LAUNCHED(c, "k_add_diag");
            src = A.get();
        }
        if (j.a <= kMaxSmall) {
            set_smem((const void*)k_inverse, smem_sq(j.a));
            launch_next(c, k_inverse, 1, 256, smem_sq(j.a), src, j.a, j.X, j.status, j.eps, nullptr);
        } else {
            DBuf<double> work((size_t)j.a * j.a + (size_t)(j.a + 1) / 2, c.stream);  // matrix, then a pivot ints
            launch_next(c, k_inverse, 1, 1024, 0, src, j.a, j.X, j.status, j.eps, work.get());
        }
        SLFMM_LAUNCHED(c, "k_inverse");
    }
}

void launch_inverse(Ctx& c, const double* A, int a, double* Ainv, int* status, double* eps_used) {
    const InverseJob j{A, a, 0.0, Ainv, status, eps_used};
    launch_inverses(c, &j, 1);
}

void launch_jacobi_svd(Ctx& c, const double* A, int a, double* V, double* sig) {
    SLFMM_REQUIRE(a >= 1 && a <= kMaxDesign, SLFMM_ERR_BAD_ARG,
                  "small eigen-solve limited to " + std::to_string(kMaxDesign) + " x " + std::to_string(kMaxDesign));
    const int ap = a + (a & 1);
    ProfScope ps(c, "small_eigh", 16.0 * a * a, 0.0);
    const size_t square = (size_t)ap * ap * sizeof(double);
    if (a <= kEighOneCta) {
        // a warp per pair of columns, in fours, and those of Gram-Schmidt
        const int threads = std::max(256, (int)round_up(32 * (uint64_t)(ap / 2), 128));
        static_assert(kEighOneCta <= 32 && 3 * 32 * 32 * sizeof(double) + (20 << 10) <= (48 << 10), "");
        launch_next(c, k_jacobi_svd<1, 1>, 1, threads, 3 * square, const_cast<double*>(A), a, V, sig, nullptr, 0ll);
    } else {
        DBuf<double> ws(3 * (size_t)ap * ap, c.stream);
        const size_t share = 3 * ceil_div(ap, kEighCluster) * ap * sizeof(double);
        const size_t sm = 2 * square <= kEighClusterSmem ? std::max(2 * square, share) : share;
        auto go = [&](auto kern) {
            set_smem((const void*)kern, std::max(sm, kEighLimit));
            launch_next_clusters(c, kern, 1, kEighCluster, 1024, sm, const_cast<double*>(A), a, V, sig, ws.get(),
                                 c.hold_next_solve);
            c.hold_next_solve = 0;
        };
        if (ap <= 64) go(k_jacobi_svd<kEighCluster, 2>);
        else if (ap <= 128) go(k_jacobi_svd<kEighCluster, 4>);
        else go(k_jacobi_svd<kEighCluster, 8>);
    }
    SLFMM_LAUNCHED(c, "k_jacobi_svd");
}

void launch_fill(Ctx& c, double* x, uint64_t n, double v) {
    if (!n) return;
    launch_next(c, k_fill, grid_for(c, n, 256), 256, 0, x, n, v);
    SLFMM_LAUNCHED(c, "k_fill");
}

void launch_transpose(Ctx& c, const double* A, int rows, int cols, double* At) {
    if (!rows || !cols) return;
    launch_next(c, k_transpose, grid_for(c, (uint64_t)rows * cols, 256), 256, 0, A, rows, cols, At);
    SLFMM_LAUNCHED(c, "k_transpose");
}

void launch_scale_cols(Ctx& c, double* A, uint64_t m, int a, int lda, const double* f) {
    if (!m || !a) return;
    launch_next(c, k_scale_cols, grid_for(c, m * a, 256), 256, 0, A, m, a, lda, f);
    SLFMM_LAUNCHED(c, "k_scale_cols");
}

void launch_build_design(Ctx& c, const double* X, int d, const double* U, int K, uint64_t n, double* C) {
    if (!n) return;
    launch_next(c, k_build_design, grid_for(c, n * (1 + d + K), 256), 256, 0, X, d, U, K, n, C);
    SLFMM_LAUNCHED(c, "k_build_design");
}

void launch_normal(Ctx& c, uint64_t seed, uint64_t rows, int cols, double* out) {
    const uint64_t total = rows * cols;
    if (!total) return;
    launch_next(c, k_normal, grid_for(c, total, 256), 256, 0, seed, total, out);
    SLFMM_LAUNCHED(c, "k_normal");
}

void launch_f64_to_f32_pad(Ctx& c, const double* A, uint64_t m, int a, int lda, float* out,
                           uint64_t m_pad, int ldo) {
    if (!m_pad || !ldo) return;
    launch_next(c, k_f64_to_f32_pad, grid_for(c, m_pad * ldo, 256), 256, 0, A, m, a, lda, out, m_pad, ldo);
    SLFMM_LAUNCHED(c, "k_f64_to_f32_pad");
}

void launch_f32_to_f64(Ctx& c, const float* A, uint64_t m, int a, int lda, double* out, int ldo) {
    if (!m || !a) return;
    launch_next(c, k_f32_to_f64, grid_for(c, m * a, 256), 256, 0, A, m, a, lda, out, ldo);
    SLFMM_LAUNCHED(c, "k_f32_to_f64");
}

}  // namespace slfmm
