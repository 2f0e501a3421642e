// The reference's Gaussian sketch stream (host_rng.cpp defines it) drawn on the
// device, equal to the host's draw bit for bit.
//
// The sampler is sequential: a draw takes one 64-bit output when the ziggurat's
// first test accepts (98.8 %), two for a wedge test, three or more in the tail,
// so where draw e starts depends on every draw before it.  But what a draw that
// starts at output s does depends on the outputs from s on alone.  So every
// output is tested as if a draw started there, which gives the outputs it would
// take; an output that no earlier one reaches over is a draw start whatever
// came before, and such an output is never far.  From there the starts follow
// by walking.
//
// The first test, a wedge's two products and its sum are exact IEEE operations.
// A wedge's exp and a tail's logarithms decide comparisons only, and where the
// device's result is too close to the threshold for its last bits not to matter
// the whole draw is made by the host instead (about once in 1e11 draws).  A tail
// value needs the host's logarithm itself: the accepted uniforms (2.6 draws in
// 10 000) are read back and their values sent.
//
// Drawn on 16 host threads and copied, 8 500 x 20 took 1.5-2 ms, with the
// device idle; here 9 us in two launches and a read-back under Step 0.
#include "chacha8.cuh"
#include "slfmm_internal.h"

namespace slfmm {

struct Ctx::NormalTails {
    struct Entry {
        uint64_t slot;  // in the scratch values, times two, plus one for the negative side
        double a;
    };
    unsigned long long drawn;  // draws made
    unsigned int n;            // tail entries (past the list's end too)
    unsigned int undecided;    // a comparison too close, or a walk too long, for the device
    Entry e[1];
};

namespace {
using Tails = Ctx::NormalTails;

// A block takes kDrawOwn outputs (eight per thread) and looks at kDrawEdge on
// either side: before them for an output that nothing reaches over, after them
// for what the last draws take.
constexpr int kDrawThreads = 256;
constexpr int kDrawWindow = kDrawThreads * 8;
constexpr int kDrawEdge = 64;
constexpr int kDrawOwn = kDrawWindow - 2 * kDrawEdge;
constexpr int kDrawReach = 17;  // outputs of the longest draw followed: eight tail pairs
constexpr int kDrawQueue = 512;
constexpr uint8_t kDrawCount = 31, kDrawValue = 32, kDrawTail = 64;
static_assert(kDrawOwn % 8 == 0 && kDrawReach < kDrawEdge && kDrawReach <= kDrawCount, "");

__device__ __forceinline__ double strip_u(uint64_t bits) {
    return __dadd_rn(__longlong_as_double((1024ll << 52) | (long long)(bits >> 12)), -3.0);
}
__device__ __forceinline__ double open_u(uint64_t bits) {
    return __dadd_rn(__longlong_as_double((1023ll << 52) | (long long)(bits >> 12)), -(1.0 - 0x1.0p-53));
}

// a < b; `near` when the two are too close for results a few ulps off
__device__ __forceinline__ bool less_or_near(double a, double b, bool& near) {
    near = near || fabs(a - b) <= 1e-12 * (fabs(a) + fabs(b));
    return a < b;
}

__global__ void __launch_bounds__(kDrawThreads) k_draw(uint64_t seed, const double* __restrict__ tables, unsigned cap,
                                                       double* __restrict__ vals, unsigned* __restrict__ counts,
                                                       Tails* __restrict__ tails) {
    dependent_start();
    __shared__ uint64_t bits[kDrawWindow];
    __shared__ double x[257], f[257];
    __shared__ uint8_t cons[kDrawWindow];
    __shared__ uint16_t queue[kDrawQueue];
    __shared__ unsigned queued, warp_sum[kDrawThreads / 32];
    const int t = threadIdx.x, lane = t & 31;
    // window position w is output first + w; there is none below 0
    const int64_t first = (int64_t)blockIdx.x * kDrawOwn - kDrawEdge;
    const int lo = first < 0 ? (int)-first : 0;
    bool undecided = false;
    for (int i = t; i < 257; i += kDrawThreads) {
        x[i] = tables[i];
        f[i] = tables[257 + i];
    }
    if (t == 0) queued = 0;
    if (8 * t >= lo) {
        ChaCha8Draws cc(seed);
        cc.blk = (uint64_t)(first + 8 * t) / 8;
        cc.refill();
#pragma unroll
        for (int j = 0; j < 8; ++j) bits[8 * t + j] = cc.word(j);
    }
    __syncthreads();
    // the first test of every output that a draw may start at; those that need
    // more are queued, so that their exp and log run on full warps
    for (int w = t; w < kDrawEdge + kDrawOwn; w += kDrawThreads) {
        uint8_t v = 0;
        if (w >= lo) {
            const uint64_t b = bits[w];
            const int i = (int)(b & 0xff);
            v = 1 | kDrawValue;
            if (!(fabs(__dmul_rn(strip_u(b), x[i])) < x[i + 1])) {
                const unsigned q = atomicAdd(&queued, 1u);
                if (q < kDrawQueue) queue[q] = (uint16_t)w;
                else undecided = true;
            }
        }
        cons[w] = v;
    }
    __syncthreads();
    for (int q = t; q < (int)min(queued, (unsigned)kDrawQueue); q += kDrawThreads) {
        const int w = queue[q];
        const int i = (int)(bits[w] & 0xff);
        bool near = false;
        if (i == 0) {
            int at = w + 1;
            bool again = true;
            while (again && at + 2 <= w + kDrawReach) {
                const double ex = log(open_u(bits[at])) / x[1];
                const double ey = log(open_u(bits[at + 1]));
                again = less_or_near(-2.0 * ey, ex * ex, near);
                at += 2;
            }
            near = near || again;
            cons[w] = (uint8_t)(at - w) | kDrawValue | kDrawTail;
        } else {
            const double xv = __dmul_rn(strip_u(bits[w]), x[i]);
            const double u01 = (double)(bits[w + 1] >> 11) * 0x1.0p-53;
            const double h = __dadd_rn(f[i + 1], __dmul_rn(__dadd_rn(f[i], -f[i + 1]), u01));
            cons[w] = 2 | (less_or_near(h, exp(__dmul_rn(-xv, xv) * 0.5), near) ? kDrawValue : 0);
        }
        undecided = undecided || near;
    }
    __syncthreads();
    // the draw starts among the thread's own eight outputs, from the nearest
    // output at or before them that nothing reaches over
    unsigned starts = 0;  // those with a value
    const int own = kDrawEdge + 8 * t;
    if (8 * t < kDrawOwn) {
        int s = own;
        for (; s > lo; --s) {
            if (s < kDrawReach) {  // too near the window's edge to tell
                undecided = true;
                break;
            }
            bool reached = false;
            for (int j = 1; j < kDrawReach; ++j) reached = reached || (cons[s - j] & kDrawCount) > j;
            if (!reached) break;
        }
        while (s < own) s += max(cons[s] & kDrawCount, 1);
        for (; s < own + 8; s += max(cons[s] & kDrawCount, 1))
            if (cons[s] & kDrawValue) starts |= 1u << (s - own);
    }
    const unsigned mine = __popc(starts);
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_sum[t >> 5] = incl;
    __syncthreads();
    unsigned at = incl - mine, total = 0;
#pragma unroll
    for (int k = 0; k < kDrawThreads / 32; ++k) {
        if (k < (t >> 5)) at += warp_sum[k];
        total += warp_sum[k];
    }
    const uint64_t base = (uint64_t)blockIdx.x * kDrawOwn;
    for (; starts; starts &= starts - 1, ++at) {
        const int w = own + __ffs(starts) - 1;
        const uint64_t b = bits[w];
        const double u = strip_u(b);
        if (cons[w] & kDrawTail) {
            const unsigned k = atomicAdd(&tails->n, 1u);
            if (k < cap) {
                // the accepted pair is the draw's last
                tails->e[k].slot = 2 * (base + at) + (u < 0.0 ? 1 : 0);
                tails->e[k].a = open_u(bits[w + (cons[w] & kDrawCount) - 2]);
            }
        } else {
            vals[base + at] = __dadd_rn(0.0, __dmul_rn(u, x[b & 0xff]));
        }
    }
    if (undecided) tails->undecided = 1;
    if (t == 0) {
        counts[blockIdx.x] = total;
        atomicAdd(&tails->drawn, (unsigned long long)total);
    }
}

// the tail values, computed by the host, into the scratch
__global__ void k_draw_tails(const Tails* __restrict__ tails, const double* __restrict__ tail_vals, unsigned n,
                             double* __restrict__ vals) {
    dependent_start();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) vals[tails->e[i].slot >> 1] = tail_vals[i];
}

// the blocks' values one after the other: block b's follow the counts before it
__global__ void __launch_bounds__(kDrawThreads) k_draw_place(const double* __restrict__ vals,
                                                             const unsigned* __restrict__ counts, uint64_t count,
                                                             double* __restrict__ out) {
    dependent_start();
    __shared__ unsigned long long part[kDrawThreads / 32];
    unsigned long long before = 0;
    for (unsigned b = threadIdx.x; b < blockIdx.x; b += kDrawThreads) before += counts[b];
#pragma unroll
    for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int k = 0; k < kDrawThreads / 32; ++k) before += part[k];
    const unsigned n = counts[blockIdx.x];
    const double* v = vals + (uint64_t)blockIdx.x * kDrawOwn;
    for (unsigned i = threadIdx.x; i < n && before + i < count; i += kDrawThreads) out[before + i] = v[i];
}

// A draw of up to this many values that nobody has started ahead is the host's: the
// device's takes two trips whatever its size (generate_omega of 16, 2 048, 4 096 and
// 8 192 values: 59, 60, 64 and 63 us by the device, 32, 48, 63 and 94 by the host).
constexpr uint64_t kDrawHost = 4096;

// tail entries to expect among `count` draws, with room: 2.6 in 10 000
unsigned tail_cap(uint64_t count) { return (unsigned)(count / 2000 + 64); }
}  // namespace

struct Ctx::PendingNormal {
    uint64_t seed = 0, rows = 0;
    int cols = 0;
    unsigned blocks = 0, cap = 0;
    DBuf<double> tables, vals;
    DBuf<unsigned> counts;
    DBuf<unsigned char> tails;
};

namespace {
// null: no room for the scratch (the host draws then)
std::shared_ptr<Ctx::PendingNormal> start_draw(Ctx& c, uint64_t seed, uint64_t rows, int cols) {
    c.pending_normal.reset();
    auto p = std::make_shared<Ctx::PendingNormal>();
    p->seed = seed;
    p->rows = rows;
    p->cols = cols;
    const uint64_t count = rows * (uint64_t)cols;
    // a draw takes 1.0139 outputs on average
    const uint64_t blocks = ceil_div(count + count / 32 + 1024, (uint64_t)kDrawOwn);
    if (blocks > 0x7fffffffu) return nullptr;
    p->blocks = (unsigned)blocks;
    p->cap = tail_cap(count);
    const size_t bytes = sizeof(Tails) + p->cap * sizeof(Tails::Entry);
    if (!c.draw_done) SLFMM_CUDA(cudaEventCreateWithFlags(&c.draw_done, cudaEventDisableTiming));
    if (bytes > c.draw_tails_bytes) {
        SLFMM_CUDA(cudaEventSynchronize(c.draw_done));  // the last copy into it (none: at once)
        if (c.draw_tails) cudaFreeHost(c.draw_tails);
        c.draw_tails = nullptr;
        c.draw_tails_bytes = 0;
        if (cudaMallocHost((void**)&c.draw_tails, bytes) != cudaSuccess) {
            cudaGetLastError();
            c.draw_tails = nullptr;
            return nullptr;
        }
        c.draw_tails_bytes = bytes;
    }
    try {
        p->tables.alloc(2 * 257, c.stream);
        p->vals.alloc(blocks * kDrawOwn, c.stream);
        p->counts.alloc(blocks, c.stream);
        p->tails.alloc(bytes, c.stream);
    } catch (const Error& e) {
        if (e.code != SLFMM_ERR_NOMEM) throw;
        cudaGetLastError();
        return nullptr;
    }
    SLFMM_CUDA(cudaMemcpyAsync(p->tables.get(), normal_tables(), p->tables.bytes(), cudaMemcpyHostToDevice, c.stream));
    SLFMM_CUDA(cudaMemsetAsync(p->tails.get(), 0, sizeof(Tails), c.stream));
    Tails* tails = reinterpret_cast<Tails*>(p->tails.get());
    launch_next(c, k_draw, p->blocks, kDrawThreads, 0, seed, p->tables.get(), p->cap, p->vals.get(), p->counts.get(),
                tails);
    SLFMM_LAUNCHED(c, "k_draw");
    SLFMM_CUDA(cudaMemcpyAsync(c.draw_tails, tails, bytes, cudaMemcpyDeviceToHost, c.stream));
    SLFMM_CUDA(cudaEventRecord(c.draw_done, c.stream));
    return p;
}
}  // namespace

void prefetch_normal(Ctx& c, uint64_t seed, uint64_t rows, int cols) {
    if (c.rng != SLFMM_RNG_CHACHA8 || rows == 0 || cols <= 0 || cols > 64) return;  // the fit checks the shape
    if (c.pending_normal && c.pending_normal->seed == seed && c.pending_normal->rows == rows &&
        c.pending_normal->cols == cols)
        return;
    c.pending_normal = start_draw(c, seed, rows, cols);
}

void draw_normal(Ctx& c, uint64_t seed, uint64_t rows, int cols, double* out) {
    if (c.rng != SLFMM_RNG_CHACHA8) {
        launch_normal(c, seed, rows, cols, out);
        return;
    }
    const uint64_t count = rows * (uint64_t)cols;
    if (!count) return;
    std::shared_ptr<Ctx::PendingNormal> p = std::move(c.pending_normal);
    c.pending_normal.reset();
    if (!p || p->seed != seed || p->rows != rows || p->cols != cols)
        p = count > kDrawHost ? start_draw(c, seed, rows, cols) : nullptr;
    bool made = false;
    if (p) {
        SLFMM_CUDA(cudaEventSynchronize(c.draw_done));
        const Tails& t = *c.draw_tails;
        made = !t.undecided && t.drawn >= count && t.n <= p->cap;
        if (made) {
            if (t.n) {
                std::vector<double> tv(t.n);
                for (unsigned i = 0; i < t.n; ++i) tv[i] = normal_tail_value(t.e[i].a, t.e[i].slot & 1);
                DBuf<double> tvd(tv.size(), c.stream);
                SLFMM_CUDA(cudaMemcpyAsync(tvd.get(), hold(c, std::move(tv)), tvd.bytes(), cudaMemcpyHostToDevice,
                                           c.stream));
                launch_next(c, k_draw_tails, (unsigned)ceil_div(t.n, 128), 128, 0,
                    reinterpret_cast<const Tails*>(p->tails.get()), tvd.get(), t.n, p->vals.get());
                SLFMM_LAUNCHED(c, "k_draw_tails");
            }
            launch_next(c, k_draw_place, p->blocks, kDrawThreads, 0, p->vals.get(), p->counts.get(), count, out);
            SLFMM_LAUNCHED(c, "k_draw_place");
        }
    }
    if (!made) {
        std::vector<double> own(count);
        reference_normal(seed, rows, (uint64_t)cols, own.data());
        SLFMM_CUDA(cudaMemcpyAsync(out, own.data(), count * sizeof(double), cudaMemcpyHostToDevice, c.stream));
        SLFMM_CUDA(cudaStreamSynchronize(c.stream));
    }
}

void release_draws(Ctx& c) {
    c.pending_normal.reset();
    if (c.draw_done) {
        cudaEventSynchronize(c.draw_done);
        cudaEventDestroy(c.draw_done);
    }
    if (c.draw_tails) cudaFreeHost(c.draw_tails);
    c.draw_done = nullptr;
    c.draw_tails = nullptr;
    c.draw_tails_bytes = 0;
}

}  // namespace slfmm
