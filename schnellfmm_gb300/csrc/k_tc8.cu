// Split-FP8 tcgen05 contraction of the packed genotype matrix (kind::f8f6f4).
//
//   P[r, c] = sum_t s_t[c] * sum_k g(r, k) * B_t[c, k]              (main)
//   M[r, c] = sum_t m_t[c] * sum_k [g(r, k) missing] * E_t[c, k]    (indicator)
//
// Genotypes {0, 1, 2} are exact in E4M3 and are expanded from the 2-bit codes
// in registers (PRMT, no shared-memory tables) straight into TMEM as the A
// operand.  The float operand W is split into power-of-two-scaled E4M3 terms:
// term t holds round_e4m3((W - terms_<t) * 2^(e0 + 4t)), so four terms carry
// about 16 significant bits per column (the "split-FP8" precision pattern);
// the per-(term, column) scales are applied in FP32 in the epilogue.  The
// optional second A operand is the missing-call indicator, multiplied by a
// second set of terms, which makes the mean-imputation correction of missing
// calls exact without any gather over the missing-call lists.
//
// Every CTA streams its own W stages; a stage is reloaded only after the
// CTA's MMAs on it have completed (per-stage "B empty" barriers).  The W
// operand is stored stage-major in global memory -- each 256-sample stage one
// contiguous blob [half][row][128 B] with the 128-byte swizzle already applied
// -- so a stage lands with ONE bulk copy.  On GB300 the copies one thread
// issues complete one after another at a near-constant ~500-750 cycles each
// whatever their size (4 KB to 64 KB, L2 or HBM), so the number of copies per
// stage, not their bytes, sets how fast a single producer can feed the MMAs.
//
// Replaces the reference's per-chunk FP64 dgemms (src/rsvd.rs:61-69, :88-97,
// :117-125, :144-153; src/testing.rs:355-374) and, through the indicator
// operand, the NaN -> column-mean fill of decode_single_snp
// (src/bed.rs:349-378) inside them.
#include <cuda.h>
#include <cuda_fp8.h>

#include <cstdlib>

#include "fp_convert.cuh"
#include "slfmm_internal.h"
#include "tc_common.cuh"

namespace slfmm {
namespace {
using namespace tc;

constexpr int kM = 128;
constexpr int kTileK = 128;                        // samples (codes) per tile block
constexpr int kTileBytes = kM * kTileK / 4;        // 4 KiB: 128 rows x 32 B
constexpr int kHalves = 2;                         // tile blocks per pipeline stage
constexpr int kStageK = kTileK * kHalves;          // 256 samples per stage
constexpr int kStageBytes = kTileBytes * kHalves;  // packed bytes per stage
// Warps: code copies, W copies, two for the MMAs, then the unpack sets of four,
// then the epilogue, two per TMEM lane quarter.  Three and four unpack sets were
// slower (80 registers a thread: column pass 2.66 ms against 2.54 ms with two
// sets at 1 M SNPs x 20 000 samples), and so were four epilogue warps where a
// unit is short (5003 samples: row pass 375 us against 283 us).
constexpr int kUnpackSets = 2;
constexpr int kEpiWarps = 8;
constexpr int kCtlWarps = 4;
constexpr int kThreads = 32 * (kCtlWarps + 4 * kUnpackSets + kEpiWarps);
constexpr int kMainTerms = 4;
constexpr int kIndTerms = 3;
constexpr uint32_t kTabGeno = 0x40380000u;  // code 00,01 -> 0; 10 -> 1.0; 11 -> 2.0 (E4M3 bytes)
constexpr uint32_t kTabMiss = 0x00003800u;  // code 01 (missing) -> 1.0

struct Tc8Args {
    uint32_t rows, kb_total, kb_per_split;
    uint32_t wpad;          // output columns
    uint32_t n_main;        // kMainTerms * wpad
    uint32_t n_ind;         // kIndTerms * wpad or 0
    uint32_t n_total;       // B rows (n_main + n_ind, or n_main when ind_shared)
    uint32_t ind_shared;    // indicator MMAs read B rows [0, n_ind) of the main terms
    uint32_t d_cols;        // TMEM columns reserved for D
    uint32_t a_cols;        // TMEM columns per A slot: a stage's genotypes, or half a stage's with the indicator
    uint32_t parts;         // A slots per stage: 1, or 2 (a slot per half, with the indicator)
    uint32_t slots, tmem_cols;   // A operand ring depth in slots (TMEM)
    uint32_t wstages;       // W operand ring depth (shared memory)
    uint32_t pstages;       // packed-code prefetch depth
    uint32_t group;         // K blocks per group of an accumulator copy
    uint32_t kcopies;       // accumulator copies (2: alternate K groups)
    uint32_t a_base;        // first TMEM column of the A stages
    uint32_t usets;         // unpack sets in use
    uint32_t none;          // 0 (see tc8_unpack)
    uint32_t b_stage_bytes; // n_total * 256: one stage of the stage-major W operand
    const float* inv_scale; // n_total: 2^-(e0 + 4t) per B row
    const uint8_t* wop;     // stage-major, pre-swizzled W operand
    int mode;               // 0: out = P + M; 1: out = s_r (P - mu_r (cs_c - M))
    long long expire_cycles;  // > 0: test hook, see below
    uint32_t tile0;           // matrix index of the tile of unit 0
    uint32_t units, gx;       // work units (row tiles x K splits) and row tiles
    uint32_t rotate;          // stagger the K order of the tiles (see below)
    const double* row_mean;
    const double* row_scale;
    const double* cs;
    float* out;
    uint32_t ldo;
    uint64_t split_stride;
    const uint8_t* tiles;   // tile-major packed codes
    uint64_t tile_bytes;    // kbt * 4096
    int* err;
};

// Pins 32 values in registers at this point of the program (an empty asm
// that reads them), so the compiler cannot sink their computation past a
// following wait.
__device__ __forceinline__ void keep32(const uint32_t (&v)[32]) {
    asm volatile("" ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
                 "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
                 "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
                 "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]));
}

// Warp-wide bounded wait polled by every lane, with warp votes as the only
// branch conditions: the compiler then knows that the warp stays converged
// and keeps the loop around it (ring positions, descriptors) in uniform
// registers, which the tensor-core and bulk-copy instructions take their
// operands from.  (A wait polled by lane 0 and passed on by a shuffle took
// about 250 cycles on a barrier that was already complete.)
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
    const uint32_t addr = smem_u32(bar);
    if (__all_sync(0xffffffffu, mbar_try(addr, parity))) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (__all_sync(0xffffffffu, mbar_try(addr, parity))) return true;
        if ((it & 1023u) == 0) {
            const bool stop = *(volatile int*)err != 0 || clock64() - t0 > kWaitCycles;
            if (__any_sync(0xffffffffu, stop)) {
                if ((threadIdx.x & 31) == 0) atomicCAS(err, 0, code);
                return false;
            }
        }
    }
}

// Ring position: slot index and the parity of its current use.  The positions
// are carried along in 32 bits: forming them from a stage counter took two
// 64-bit divisions per ring and stage in every role, several hundred cycles
// of each handshake (column pass at n = 20 000: 1821 cycles per stage).
struct Ring {
    uint32_t slot, phase;
    __device__ __forceinline__ void advance(uint32_t by, uint32_t n) {  // by: a few slots
        slot += by;
        while (slot >= n) {
            slot -= n;
            phase ^= 1u;
        }
    }
};

// Waits for the copies of every slot a producer has filled (`next`: the
// position it would fill next; `lapped`: it has filled every slot at least
// once), so that no CTA leaves with copies in flight into its shared memory.
__device__ __forceinline__ void drain_ring(uint64_t* full, const Ring& next, bool lapped, uint32_t n, int* err,
                                           int code) {
    for (uint32_t s = 0; s < n; ++s) {
        if (s < next.slot) warp_wait(full + s, next.phase, err, code);
        else if (lapped) warp_wait(full + s, next.phase ^ 1u, err, code);
    }
}

// MMA issue of one warp's share of a work unit (nkb stages from ring positions
// st, sw, which are carried on).  The whole warp runs the loop and each tcgen05
// instruction is predicated on one elected lane: with the loop under
// `lane == 0` instead, every MMA took at least 116 cycles to issue whatever its
// width, since its operands went from vector to uniform registers one
// instruction at a time (measured, 128 x N x 32 E4M3: 116 cycles at N = 32 ...
// 192; this form N / 2 cycles, the pipe's rate).
//
// Two warps issue.  A barrier wait of a warp comes back only once the MMAs that
// it issued before have left its queue, so the pipe runs dry at every wait of
// a single issuer (875 of 1390 cycles per stage busy); the other warp's MMAs
// fill that time.  The warps' accumulators are disjoint and each sees its own
// in K order: with two accumulator copies they take alternate groups of
// a.group stages; with the indicator one takes the genotype and one the
// indicator MMAs; otherwise each takes half of the output columns.
struct MmaShare {
    uint32_t idesc;      // instruction descriptor (its N)
    uint32_t d;          // first accumulator column
    uint32_t a_off;      // TMEM column offset of its operand in an A slot
    uint32_t b_off;      // first B row of its operand, in descriptor units
    uint32_t copy;       // its accumulator copy (kcopies == 2)
};

template <int PARTS>
__device__ __forceinline__ bool tc8_mma_unit(const Tc8Args& a, const MmaShare& m, uint32_t a0, uint64_t bdesc0,
                                             uint64_t* full_b, uint64_t* full_a, uint64_t* a_empty,
                                             uint64_t* b_empty, Ring& st, Ring& sw, uint32_t nkb,
                                             uint32_t elected) {
    constexpr int kSteps = kStageK / 32 / PARTS;           // MMA K steps per A slot
    const uint32_t S = a.slots, SW = a.wstages;
    const uint64_t bstep = a.b_stage_bytes >> 4;           // descriptor address units per stage
    const uint64_t hstep = (uint64_t)a.n_total * (128 >> 4);  // next 128-sample half of the stage
    const bool alternate = a.kcopies == 2;
    uint32_t copy = 0, in_group = 0, acc = 0;  // copy of this stage, its place in the group; 0 clears D
    for (uint32_t i = 0; i < nkb; ++i) {
        if (!alternate || copy == m.copy) {
            const uint64_t bd = bdesc0 + sw.slot * bstep + m.b_off;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
                if (part == 0 && !warp_wait(full_b + sw.slot, sw.phase, a.err, 25)) return false;
                if (!warp_wait(full_a + st.slot, st.phase, a.err, 26)) return false;
                fence_after();
                const uint32_t ad = a0 + st.slot * a.a_cols + m.a_off;
#pragma unroll
                for (int s = 0; s < kSteps; ++s) {
                    const int kk = part * kSteps + s;
                    mma_ts_f8(m.d, ad + s * 8, bd + (kk >> 2) * hstep + (kk & 3) * 2, m.idesc, acc, elected);
                    acc = 1u;
                }
                mma_commit(a_empty + st.slot, elected);
                st.advance(1, S);
            }
            mma_commit(b_empty + sw.slot, elected);
        } else {
            st.advance(PARTS, S);
        }
        sw.advance(1, SW);
        if (alternate && ++in_group == a.group) {
            in_group = 0;
            copy ^= 1u;
        }
    }
    return true;
}

// Half a row (128 codes, 32 B) of a stage.
__device__ __forceinline__ void load_half(const uint8_t* tile, uint32_t row, uint32_t* w) {
    const uint4* rp = reinterpret_cast<const uint4*>(tile + row * (kTileK / 4));
    const uint4 x = rp[0], y = rp[1];
    w[0] = x.x;
    w[1] = x.y;
    w[2] = x.z;
    w[3] = x.w;
    w[4] = y.x;
    w[5] = y.y;
    w[6] = y.z;
    w[7] = y.w;
}

// The E4M3 bytes of half a row (128 codes): a 32-bit word holds 16 two-bit
// codes; masking the even / odd codes into nibbles gives PRMT selectors
// directly (4 codes per PRMT), and the B operand stores K in the matching
// even-then-odd order.  With IND also the missing-call indicator's bytes.
template <bool IND>
__device__ __forceinline__ void expand_half(const uint32_t* w, uint32_t (&gv)[32], uint32_t (&mv)[32]) {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const uint32_t e0 = w[t] & 0x33333333u, o0 = (w[t] >> 2) & 0x33333333u;
        const uint32_t e1 = e0 >> 16, o1 = o0 >> 16;
        gv[4 * t] = __byte_perm(kTabGeno, 0u, e0);
        gv[4 * t + 1] = __byte_perm(kTabGeno, 0u, e1);
        gv[4 * t + 2] = __byte_perm(kTabGeno, 0u, o0);
        gv[4 * t + 3] = __byte_perm(kTabGeno, 0u, o1);
        if (IND) {
            mv[4 * t] = __byte_perm(kTabMiss, 0u, e0);
            mv[4 * t + 1] = __byte_perm(kTabMiss, 0u, e1);
            mv[4 * t + 2] = __byte_perm(kTabMiss, 0u, o0);
            mv[4 * t + 3] = __byte_perm(kTabMiss, 0u, o1);
        }
    }
}

// One unpack warp's part of the CTA's items (all its units in sequence), a row
// per lane expanded into TMEM.  An item, one A slot, is a stage's genotypes or,
// with the indicator, half a stage's genotypes and indicator: that doubles the
// ring where TMEM holds two stages only (D takes 224 of its 512 columns at 32
// outputs).  A set takes items set, set + usets, ...  Everything is expanded
// before the wait for the slot, so a freed slot is refilled by its stores alone.
//
// A packed slot is released once its codes are in registers.  The arrival's
// count depends on them (`none` is 0), so it cannot be issued before the loads
// have returned: released right behind the loads, the refill has been seen to
// overtake them.
template <bool IND>
__device__ __forceinline__ void tc8_unpack(const Tc8Args& a, uint32_t a0, const uint8_t* psm, uint32_t row,
                                           uint64_t* p_full, uint64_t* p_empty, uint64_t* full_a, uint64_t* a_empty,
                                           uint32_t set, uint32_t stages) {
    const uint32_t S = a.slots, P = a.pstages, nsets = a.usets;
    const bool lane0 = (threadIdx.x & 31) == 0;
    constexpr uint32_t kPerStage = IND ? 2 : 1;
    const uint32_t items = stages * kPerStage;
    Ring pr{set / kPerStage, 0}, st{set, 0};
    for (uint32_t i = set; i < items; i += nsets) {
        uint32_t w[IND ? 8 : 16], x[32], y[32];
        if (!warp_wait(p_full + pr.slot, pr.phase, a.err, 27)) return;
        const uint8_t* tile = psm + pr.slot * kStageBytes;
        uint32_t seen;
        if constexpr (IND) {
            load_half(tile + (i & 1u) * kTileBytes, row, w);
            seen = w[0] | w[4];
        } else {
            load_half(tile, row, w);
            load_half(tile + kTileBytes, row, w + 8);
            seen = w[0] | w[4] | w[8] | w[12];
        }
        __syncwarp();
        if (lane0) mbar_arrive_n(p_empty + pr.slot, 1u + (seen & a.none));
        pr.advance((i + nsets) / kPerStage - i / kPerStage, P);
        if constexpr (IND) {
            expand_half<true>(w, x, y);
        } else {
            expand_half<false>(w, x, x);
            expand_half<false>(w + 8, y, y);
        }
        keep32(x);  // expanded before the slot wait: only the stores follow it
        keep32(y);
        const uint32_t a_col = a0 + st.slot * a.a_cols;
        if (!warp_wait(a_empty + st.slot, st.phase ^ 1u, a.err, 28)) return;
        tmem_st_x32(a_col, x);
        tmem_st_x32(a_col + 32, y);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        fence_before();
        __syncwarp();
        if (lane0) mbar_arrive(full_a + st.slot);
        st.advance(nsets, S);
    }
}

__device__ __forceinline__ void fma16(const float* scl, const float (&v)[16], float (&acc)[16]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 f = reinterpret_cast<const float4*>(scl)[q];
        acc[4 * q] = fmaf(f.x, v[4 * q], acc[4 * q]);
        acc[4 * q + 1] = fmaf(f.y, v[4 * q + 1], acc[4 * q + 1]);
        acc[4 * q + 2] = fmaf(f.z, v[4 * q + 2], acc[4 * q + 2]);
        acc[4 * q + 3] = fmaf(f.w, v[4 * q + 3], acc[4 * q + 3]);
    }
}

// 16 columns c0 .. of a warp's 32 rows from the accumulators: pm = sum_t
// scale_t (sum of the copies), pi the indicator's terms.
__device__ __forceinline__ void read_terms(const Tc8Args& a, uint32_t d0, const float* scl, uint32_t c0,
                                           bool second_copy, float (&pm)[16], float (&pi)[16]) {
    float v[16], v2[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) pm[k] = pi[k] = 0.f;
    if (second_copy) {
#pragma unroll 1
        for (int t = 0; t < kMainTerms; ++t) {
            const uint32_t col = t * a.wpad + c0;
            tmem_ld_x16_async(d0 + col, v);
            tmem_ld_x16_async(d0 + a.d_cols + col, v2);
            tmem_ld_wait();
            pin16(v);
            pin16(v2);
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] += v2[k];
            fma16(scl + col, v, pm);
        }
        return;
    }
#pragma unroll 1
    for (int t = 0; t < kMainTerms; t += 2) {
        const uint32_t col = t * a.wpad + c0;
        tmem_ld_x16_async(d0 + col, v);
        tmem_ld_x16_async(d0 + col + a.wpad, v2);
        tmem_ld_wait();
        pin16(v);
        pin16(v2);
        fma16(scl + col, v, pm);
        fma16(scl + col + a.wpad, v2, pm);
    }
    if (a.n_ind) {
        const uint32_t dcol = a.n_main + c0, scol = (a.ind_shared ? 0u : a.n_main) + c0;
        tmem_ld_x16_async(d0 + dcol, v);
        tmem_ld_x16_async(d0 + dcol + a.wpad, v2);
        tmem_ld_wait();
        pin16(v);
        pin16(v2);
        fma16(scl + scol, v, pi);
        tmem_ld_x16_async(d0 + dcol + 2 * a.wpad, v);
        fma16(scl + scol + a.wpad, v2, pi);
        tmem_ld_wait();
        pin16(v);
        fma16(scl + scol + 2 * a.wpad, v, pi);
    }
}

// One CTA per SM runs work units u = blockIdx.x, blockIdx.x + gridDim.x, ...
// (unit u: row tile u % gx, K split u / gx); a launch with one CTA per unit
// is the same code with one unit each.  The copy and MMA rings run on across
// a CTA's units (stage g of the CTA's sequence sits in slot g % depth), so the
// producers prefetch the next unit's operands while the current unit's last
// stages and epilogue run; D is reused once the epilogue has read it
// (d_empty).  A unit's accumulation order depends only on its tile and
// split, so every grid gives the same bits.
__global__ void __launch_bounds__(kThreads, 1) k_tc8_rows(const __grid_constant__ Tc8Args a) {
    dependent_wait();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t S = a.slots, SW = a.wstages, P = a.pstages;
    uint8_t* bsm = smem;
    uint8_t* psm = bsm + SW * a.b_stage_bytes;
    float* scl = reinterpret_cast<float*>(psm + P * kStageBytes);             // up to 512 floats
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(scl) + 2048);
    uint64_t* full_b = bars;                 // [SW] W stage landed (TMA tx)
    uint64_t* b_empty = bars + SW;           // [SW] the MMAs reading the W stage done
    uint64_t* full_a = bars + 2 * SW;        // [S] A slot written to TMEM (4 warps)
    uint64_t* a_empty = full_a + S;          // [S] the MMAs reading the A slot done
    uint64_t* p_full = a_empty + S;          // [P] packed codes landed (TMA tx)
    uint64_t* p_empty = p_full + P;          // [P] packed codes in registers (4 or 8 warps)
    uint64_t* tmem_full = p_empty + P;       // a unit's MMAs done
    uint64_t* d_empty = tmem_full + 1;       // a unit's epilogue has read D (its warps)
    uint64_t* never = d_empty + 1;           // test hook: a barrier nothing arrives at
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(never + 1);

    // warp index through a shuffle: known to be the same in every lane
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const bool ind = a.n_ind != 0;
    auto unit_kb0 = [&](uint32_t u) { return (u / a.gx) * a.kb_per_split; };
    auto unit_nkb = [&](uint32_t u) {
        const uint32_t kb0 = unit_kb0(u), kb1 = min(a.kb_total, kb0 + a.kb_per_split);
        return kb1 > kb0 ? kb1 - kb0 : 0u;
    };
    // K order: the tiles of a launch all read the same W stages, and with
    // every CTA at the same stage the L2 serves one 56 KB stage to ~150 SMs
    // at once.  Each tile starts at its own stage (a rotation of the K loop,
    // fixed by its index in the matrix, so the accumulation order and the
    // bits do not depend on how rows are split into launches).
    auto unit_rot = [&](uint32_t u, uint32_t nkb) {
        return (a.rotate && nkb > 1) ? (uint32_t)(((a.tile0 + u % a.gx) * 37ull) % nkb) : 0u;
    };

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < SW; ++s) {
            mbar_init(full_b + s, 1);
            mbar_init(b_empty + s, a.kcopies == 2 ? 1 : 2);  // every MMA warp that reads the stage
        }
        for (uint32_t s = 0; s < S; ++s) {
            mbar_init(full_a + s, 4);     // one arrival per unpack warp
            mbar_init(a_empty + s, a.kcopies == 2 ? 1 : 2);
        }
        for (uint32_t p = 0; p < P; ++p) {
            mbar_init(p_full + p, 1);
            mbar_init(p_empty + p, 4 * a.parts);  // every unpack warp that reads the slot
        }
        mbar_init(tmem_full, 2);
        mbar_init(d_empty, kEpiWarps);
        mbar_init(never, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                     "r"(a.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (uint32_t e = threadIdx.x; e < a.n_total; e += blockDim.x) scl[e] = a.inv_scale[e];
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_holder;

    // Test hook (slfmm_debug_expire_next_wait): before any copy or MMA is
    // issued, thread 0 waits on a barrier that nothing completes, bounded by
    // expire_cycles; the wait expires, sets the error flag (site 30), and the
    // CTA skips its work and frees its TMEM.  Nothing is in flight, so the
    // context stays usable.
    if (a.expire_cycles > 0) {
        if (threadIdx.x == 0) mbar_wait_for(never, 0, a.err, 30, a.expire_cycles);
    } else if (warp == 0) {
        // packed-code producer: runs up to P stages ahead of the unpackers,
        // across units; each (tile, stage) operand is one contiguous bulk copy.
        // (A slot's first fill waits for the phase before a fresh barrier's
        // first one, which is complete.)
        const uint32_t elected = elect_one();
        Ring pr{0, 0};
        bool ok = true, lapped = false;
        for (uint32_t u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
            const uint32_t nkb = unit_nkb(u);
            const uint8_t* src = a.tiles + (uint64_t)(u % a.gx) * a.tile_bytes + (uint64_t)unit_kb0(u) * kStageBytes;
            uint32_t ks = unit_rot(u, nkb);
            for (uint32_t i = 0; i < nkb; ++i) {
                ok = warp_wait(p_empty + pr.slot, pr.phase ^ 1u, a.err, 21);
                if (!ok) break;
                bulk_g2s_tx(psm + pr.slot * kStageBytes, src + (uint64_t)ks * kStageBytes, kStageBytes,
                            p_full + pr.slot, elected);
                if (++ks == nkb) ks = 0;
                pr.advance(1, P);
                lapped = lapped || pr.slot == 0;
            }
        }
        drain_ring(p_full, pr, lapped, P, a.err, 22);
    } else if (warp == 2) {
        // each spinning role has a warp of its own: lanes of one warp that
        // spin in different loops starve each other
        // W producer: one bulk copy per stage, across units
        const uint32_t elected = elect_one();
        Ring wr{0, 0};
        bool ok = true, lapped = false;
        for (uint32_t u = blockIdx.x; u < a.units && ok; u += gridDim.x) {
            const uint32_t nkb = unit_nkb(u);
            const uint8_t* src = a.wop + (uint64_t)unit_kb0(u) * a.b_stage_bytes;
            uint32_t ks = unit_rot(u, nkb);
            for (uint32_t i = 0; i < nkb; ++i) {
                ok = warp_wait(b_empty + wr.slot, wr.phase ^ 1u, a.err, 23);
                if (!ok) break;
                bulk_g2s_tx(bsm + wr.slot * a.b_stage_bytes, src + (uint64_t)ks * a.b_stage_bytes, a.b_stage_bytes,
                            full_b + wr.slot, elected);
                if (++ks == nkb) ks = 0;
                wr.advance(1, SW);
                lapped = lapped || wr.slot == 0;
            }
        }
        drain_ring(full_b, wr, lapped, SW, a.err, 24);
    } else if (warp == 1 || warp == 3) {
        const uint32_t elected = elect_one();
        const uint32_t second = warp == 3 ? 1u : 0u;
        MmaShare m;
        m.copy = second;
        if (ind) {
            m.idesc = instr_desc_e4m3(second ? a.n_ind : a.n_main);
            m.d = tmem + (second ? a.n_main : 0u);
            m.a_off = second ? a.a_cols / 2 : 0u;
            m.b_off = second && !a.ind_shared ? a.n_main * (128 >> 4) : 0u;
        } else {
            const uint32_t n = a.kcopies == 2 ? a.n_main : a.n_main / 2;
            m.idesc = instr_desc_e4m3(n);
            m.d = tmem + second * (a.kcopies == 2 ? a.d_cols : n);
            m.a_off = 0;
            m.b_off = a.kcopies == 2 ? 0u : second * n * (128 >> 4);
        }
        const uint32_t a0 = tmem + a.a_base;
        const uint64_t bdesc0 = smem_desc(smem_u32(bsm));
        Ring st{0, 0}, sw{0, 0};           // A ring (TMEM), W ring (shared memory)
        uint32_t k = 0;                    // this CTA's units so far
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < a.units && ok; u += gridDim.x, ++k) {
            const uint32_t nkb = unit_nkb(u);
            // D is free once the previous unit's epilogue has read it
            if (k > 0) {
                ok = warp_wait(d_empty, (k - 1) & 1u, a.err, 31);
                fence_after();
            }
            if (ok)
                ok = ind ? tc8_mma_unit<2>(a, m, a0, bdesc0, full_b, full_a, a_empty, b_empty, st, sw, nkb, elected)
                         : tc8_mma_unit<1>(a, m, a0, bdesc0, full_b, full_a, a_empty, b_empty, st, sw, nkb, elected);
            mma_commit(tmem_full, elected);  // both warps arrive per unit (an idle one at once)
        }
    } else if (warp >= kCtlWarps && warp < kCtlWarps + 4 * kUnpackSets) {
        // sets of four unpack warps; warp % 4 is the TMEM lane quarter a warp
        // may access
        const uint32_t set = (uint32_t)(warp - kCtlWarps) >> 2;
        if (set < a.usets) {
            uint32_t stages = 0;  // of the CTA
            for (uint32_t u = blockIdx.x; u < a.units; u += gridDim.x) stages += unit_nkb(u);
            const uint32_t row = ((uint32_t)warp & 3u) * 32 + lane;
            const uint32_t a0 = tmem + ((((uint32_t)warp & 3u) * 32) << 16) + a.a_base;
            if (ind) tc8_unpack<true>(a, a0, psm, row, p_full, p_empty, full_a, a_empty, set, stages);
            else tc8_unpack<false>(a, a0, psm, row, p_full, p_empty, full_a, a_empty, set, stages);
        }
    } else if (warp >= kCtlWarps + 4 * kUnpackSets) {
        // epilogue warps: a unit's accumulators are read as soon as its MMAs
        // are done and handed back (d_empty) before the results are formed and
        // stored, while the unpack and MMA warps go on with the next unit
        const uint32_t row = ((uint32_t)warp & 3u) * 32 + lane;
        const uint32_t d0 = tmem + ((((uint32_t)warp & 3u) * 32) << 16);
        const uint32_t cfirst = ((uint32_t)(warp - kCtlWarps - 4 * kUnpackSets) >> 2) * 16;  // 16-column groups in turn
        uint32_t k = 0;
        for (uint32_t u = blockIdx.x; u < a.units; u += gridDim.x, ++k) {
            const uint32_t nkb = unit_nkb(u);
            const uint32_t grow = (u % a.gx) * kM + row;
            const bool live = grow < a.rows;
            double rm = 0.0, rs = 0.0;
            if (a.mode == 1 && live) {
                rm = a.row_mean[grow];
                rs = a.row_scale[grow];
            }
            float* dst = a.out + (uint64_t)(u / a.gx) * a.split_stride + (uint64_t)grow * a.ldo;
            if (!warp_wait(tmem_full, k & 1u, a.err, 29)) break;
            // the second accumulator copy holds data only if its first group exists
            const bool second_copy = a.kcopies == 2 && nkb > a.group;
            fence_after();
            for (uint32_t c0 = cfirst;; c0 += 4 * kEpiWarps) {
                float pm[16], pi[16];
                if (c0 < a.wpad) read_terms(a, d0, scl, c0, second_copy, pm, pi);
                if (c0 + 4 * kEpiWarps >= a.wpad) {
                    // this warp's last read: D may be overwritten by the next unit's MMAs
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(d_empty);
                }
                if (c0 < a.wpad && live) {
                    float4* d4 = reinterpret_cast<float4*>(dst + c0);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        float o[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int kk = 4 * t + q;
                            if (a.mode == 1)
                                o[q] = (float)(rs * ((double)pm[kk] - rm * (a.cs[c0 + kk] - (double)pi[kk])));
                            else
                                o[q] = pm[kk] + pi[kk];
                        }
                        d4[t] = make_float4(o[0], o[1], o[2], o[3]);
                    }
                }
                if (c0 + 4 * kEpiWarps >= a.wpad) break;
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols)
                     : "memory");
    }
}

// per-column max |x * kscale| as float bits (non-negative floats order as
// ints); one warp per row, lanes over columns (w <= 128), four rows in flight.
// A block's warps are combined before the atomics: with a block per eight rows
// and a warp's own atomics, 20 000 x 72 took 60 us, all of it on 72 addresses.
template <typename T>
__global__ void __launch_bounds__(256) k_colmax_abs(const T* __restrict__ src, int ld, uint64_t K, int w,
                                                    const double* __restrict__ kscale, unsigned* __restrict__ colmax) {
    dependent_start();
    __shared__ unsigned red[128];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 128) red[threadIdx.x] = 0u;
    __syncthreads();
    float m[4] = {0.f, 0.f, 0.f, 0.f};
    const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
#pragma unroll 4
    for (uint64_t k = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); k < K; k += nw) {
        const float ks = kscale ? (float)kscale[k] : 1.f;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int c = lane + 32 * t;
            if (c < w) m[t] = fmaxf(m[t], fabsf((float)src[k * ld + c] * ks));
        }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int c = lane + 32 * t;
        if (c < w) atomicMax(red + c, __float_as_uint(m[t]));
    }
    __syncthreads();
    if ((int)threadIdx.x < w) atomicMax(colmax + threadIdx.x, red[threadIdx.x]);
}

__device__ __forceinline__ int term_e0(unsigned bits) {
    const float cm = __uint_as_float(bits);
    if (!(cm > 0.f)) return 0;
    int E;
    frexpf(cm, &E);
    return 8 - E;  // cm * 2^e0 in [128, 256)
}

// exact 2^ex as a float (ldexpf outside the normal exponent range)
__device__ __forceinline__ float pow2f(int ex) {
    return (ex >= -126 && ex <= 127) ? __int_as_float((127 + ex) << 23) : ldexpf(1.f, ex);
}

// A stage-major W operand with n_rows rows: stage kb = k / 256 is the contiguous
// blob [half][row][128 B] at kb * n_rows * 256, and within each 128-byte row the
// 16-byte chunk j sits at chunk j ^ (row & 7) -- the 128-byte swizzle the MMA
// descriptors expect of a 1024-byte aligned shared-memory stage (n_rows % 8 == 0
// keeps every half's rows aligned to the 8-row swizzle period).

// The E4M3 terms of one scaling of an operand: a transposed pass splits two of
// them (diag(s) Q for the genotypes, diag(mu s) Q for the missing-call
// indicator), a row pass W and, for the indicator, its leading terms again.
struct TermSet {
    const double* kscale;    // per-K-row scale (null: 1)
    int terms;               // E4M3 terms (0: set absent)
    int row_off;             // first B row of the set
    const unsigned* colmax;  // per-column max |x * kscale| (float bits)
};

// Per-column max |x kscale| of both sets in one pass over a narrow operand
// (w <= ld <= 32, ld % 4 == 0, 16-byte aligned rows): a thread keeps one
// 16-byte column quad and walks rows, four rows in flight; lanes with the
// same quad are combined by shuffles before the atomics.
__global__ void __launch_bounds__(256) k_colmax_pair(const float* __restrict__ src, int ld, uint64_t K, int w,
                                                     const double* __restrict__ ksa, const double* __restrict__ ksb,
                                                     unsigned* __restrict__ cma, unsigned* __restrict__ cmb) {
    dependent_start();
    const int q = ld >> 2;  // quads per row: 1, 2, 4 or 8 (divides the thread count)
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthreads = (uint64_t)gridDim.x * blockDim.x;
    const int qp = (int)(tid % q);
    const uint64_t step = nthreads / q;
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float ma[4] = {0.f, 0.f, 0.f, 0.f}, mb[4] = {0.f, 0.f, 0.f, 0.f};
    for (uint64_t j0 = tid / q; j0 < K; j0 += 4 * step) {
        float4 v[4];
        double da[4], db[4];  // all loads before the first conversion's branch
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t j = j0 + u * step;
            const bool ok = j < K;
            v[u] = ok ? s4[j * q + qp] : make_float4(0.f, 0.f, 0.f, 0.f);
            da[u] = ok && ksa ? ksa[j] : 1.0;
            db[u] = ok && ksb ? ksb[j] : 1.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
            const float fa = f32_of_f64(da[u]), fb = f32_of_f64(db[u]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                ma[i] = fmaxf(ma[i], fabsf(x[i] * fa));
                mb[i] = fmaxf(mb[i], fabsf(x[i] * fb));
            }
        }
    }
    // lanes l, l + q, l + 2q, ... of a warp hold the same quad
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (o < q) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ma[i] = fmaxf(ma[i], __shfl_xor_sync(0xffffffffu, ma[i], o));
            mb[i] = fmaxf(mb[i], __shfl_xor_sync(0xffffffffu, mb[i], o));
        }
    }
    // then the block's warps through shared memory: one atomic per column
    // and block (non-negative floats order as their bits)
    __shared__ unsigned red[8][2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane < q) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            red[warp][0][4 * lane + i] = __float_as_uint(ma[i]);
            red[warp][1][4 * lane + i] = __float_as_uint(mb[i]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        const int set = threadIdx.x >> 5, c = threadIdx.x & 31;
        unsigned* dst = set ? cmb : cma;
        if (c < w && c < 4 * q && dst) {
            unsigned m = 0;
            for (int wv = 0; wv < (int)(blockDim.x >> 5); ++wv) m = max(m, red[wv][set][c]);
            atomicMax(dst + c, m);
        }
    }
}

// W (K x w) -> the E4M3 rows of both sets, row_off + t * wpad + c for term t of
// column c, of a stage-major operand with n_rows rows, zero padded
// to whole stages; inv_scale[row] = 2^-(e0 + 4t).  Term t is
// round_e4m3((r - terms_<t) * 2^(e0 + 4t)); the power-of-two scales are exact, so
// each step's residual is rounded once.
//
// A block makes one stage (256 K rows) of 16 columns, a thread 16 K rows of a
// column: those are one 16-byte chunk of every term, the even K indices of its
// halves, then the odd ones (the order the unpackers emit the genotypes of a
// 32-bit code word in), converted in the pairs that the words take.  The chunks
// pass through shared memory so that every term's 16 rows leave as 2 KB in a row.
// With a thread per K pair and the terms through shared memory byte by byte,
// 400 000 x 20 (seven terms) took 87 us and 8 500 x 20 (four) 18 us; so 37
// and 6.
constexpr int kTermCols = 16;
template <typename T>
__global__ void __launch_bounds__(256) k_fp8_terms(const T* __restrict__ src, int ld, uint64_t K, int w, int wpad,
                                                   TermSet sa, TermSet sb, int n_rows, uint8_t* __restrict__ B,
                                                   float* __restrict__ inv_scale) {
    dependent_start();
    constexpr int kT = kMainTerms + kIndTerms;
    __shared__ uint4 tile[kT][2][kTermCols][8];
    __shared__ float ks[2][kStageK];
    __shared__ float up[kT][kTermCols], dn[kT][kTermCols];
    const uint64_t k0 = (uint64_t)blockIdx.x * kStageK;
    const int c0 = blockIdx.y * kTermCols;
    const int nt = sa.terms + sb.terms;
    const int cc = threadIdx.x % kTermCols, g = threadIdx.x / kTermCols;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint64_t k = k0 + 16 * g + i;
        x[i] = k < K && c0 + cc < w ? (float)src[k * ld + c0 + cc] : 0.f;
    }
    {
        const uint64_t k = k0 + threadIdx.x;
        ks[0][threadIdx.x] = sa.kscale && k < K ? f32_of_f64(sa.kscale[k]) : 1.f;
        ks[1][threadIdx.x] = sb.kscale && k < K ? f32_of_f64(sb.kscale[k]) : 1.f;
    }
    for (int e = threadIdx.x; e < nt * kTermCols; e += blockDim.x) {
        const int t = e / kTermCols, c = c0 + e % kTermCols;
        const bool first = t < sa.terms;
        const int tt = first ? t : t - sa.terms;
        const int e0 = c < w ? term_e0((first ? sa.colmax : sb.colmax)[c]) : 0;
        up[t][e % kTermCols] = pow2f(e0 + 4 * tt);
        dn[t][e % kTermCols] = pow2f(-(e0 + 4 * tt));
        if (blockIdx.x == 0)
            inv_scale[(first ? sa.row_off : sb.row_off) + tt * wpad + c] = c < w ? pow2f(-(e0 + 4 * tt)) : 1.f;
    }
    __syncthreads();
#pragma unroll
    for (int set = 0; set < 2; ++set) {
        const int terms = set ? sb.terms : sa.terms, base = set ? sa.terms : 0;
        if (!terms) break;
        float r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = x[i] * ks[set][16 * g + i];
#pragma unroll
        for (int t = 0; t < kMainTerms; ++t) {
            if (t >= terms) break;
            const float u = up[base + t][cc], d = dn[base + t][cc];
            uint32_t word[4];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                // pairs (0, 2), (4, 6), (8, 10), (12, 14), (1, 3) ..: two to a word
                const int i = (q & 3) * 4 + (q >> 2);
                const __nv_fp8x2_storage_t q2 =
                    __nv_cvt_float2_to_fp8x2(make_float2(r[i] * u, r[i + 2] * u), __NV_SATFINITE, __NV_E4M3);
                const float2 f = __half22float2(__half2(__nv_cvt_fp8x2_to_halfraw2(q2, __NV_E4M3)));
                r[i] = fmaf(-f.x, d, r[i]);
                r[i + 2] = fmaf(-f.y, d, r[i + 2]);
                if (q & 1) word[q >> 1] |= (uint32_t)q2 << 16;
                else word[q >> 1] = q2;
            }
            tile[base + t][g >> 3][cc][(g & 7) ^ (cc & 7)] = make_uint4(word[0], word[1], word[2], word[3]);
        }
    }
    __syncthreads();
    uint8_t* stage = B + (uint64_t)blockIdx.x * n_rows * kStageK;
    for (int e = threadIdx.x; e < nt * 2 * kTermCols * 8; e += blockDim.x) {
        const int t = e / (2 * kTermCols * 8), h = e / (kTermCols * 8) % 2, at = e % (kTermCols * 8);
        const int row = (t < sa.terms ? sa.row_off + t * wpad : sb.row_off + (t - sa.terms) * wpad) + c0;
        reinterpret_cast<uint4*>(stage + (uint64_t)(h * n_rows + row) * 128)[at] = tile[t][h][0][at];
    }
}

__global__ void k_sub_colterm(double* __restrict__ S, int lds, uint64_t n, int w, const double* __restrict__ colterm) {
    dependent_start();
    const uint64_t total = n * w;
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = t / w;
        const int c = (int)(t - i * w);
        S[i * lds + c] -= colterm[c];
    }
}

}  // namespace

// Tuning overrides (autotuner / experiments): SLFMM_TC8_STAGES, _PSTAGES, _GROUP.
static int env_int(const char* name, int dflt) {
    const char* v = std::getenv(name);
    return v && *v ? std::atoi(v) : dflt;
}

// The plan with explicit caps on the packed-code ring (pmax), the A ring (smax
// stages), the K blocks per group of an accumulator copy (gmax: 1 or 2) and the
// W ring (wmax); fp8_plan takes them from the environment.
Fp8Plan fp8_plan_knobs(int wpad, bool ind, uint64_t tiles, int pmax_in, int smax, int gmax_in, int wmax,
                       bool ind_shared) {
    Fp8Plan p{};
    p.wpad = (uint32_t)wpad;
    p.n_main = kMainTerms * wpad;
    p.n_ind = ind ? kIndTerms * wpad : 0;
    p.ind_shared = (ind && ind_shared) ? 1u : 0u;
    p.n_total = p.ind_shared ? p.n_main : p.n_main + p.n_ind;      // B rows
    p.d_cols = (uint32_t)round_up(p.n_main + p.n_ind, 32);       // accumulator columns
    const uint32_t a_stage = (ind ? 2 : 1) * (kStageK / 4);  // TMEM columns of one stage's A operand(s)
    p.b_stage_bytes = p.n_total * 128 * kHalves;  // one bulk copy: 16-byte multiple, below the 1 MB tx limit
    p.tmem_cols = 512;  // one CTA per SM: all of TMEM
    const size_t fixed = 1024 + 2048 + 128 * 8 + 64;
    // without the indicator two accumulator copies when TMEM holds them next to
    // at least three A stages; alternate pairs of K blocks go to them
    p.kcopies = (!ind && 2 * p.d_cols + 3 * a_stage <= 512) ? 2 : 1;
    p.group = gmax_in >= 2 ? 2 : 1;
    p.a_base = p.kcopies * p.d_cols;
    // A ring: as deep as TMEM allows (cap smax stages), whole stages or, with
    // the indicator, half stages, an even number of them
    p.parts = ind ? 2 : 1;
    p.a_cols = a_stage / p.parts;
    const uint32_t by_tmem = p.a_base < 512 ? (512 - p.a_base) / a_stage : 0;
    const uint32_t cap = (uint32_t)std::max(1, smax) * p.parts;
    p.slots = p.a_base < 512 ? std::min<uint32_t>((512 - p.a_base) / p.a_cols / p.parts * p.parts, cap) : 0;
    // Shared memory: 4, 3 or 2 W stages (caps wmax, and pmax for the codes), then
    // packed-code stages, up to 8, then more W stages if they fit.  Four of
    // each where they fit: 32 KB W stages and 8 KB code stages stream at 435
    // cycles per stage with 4 + 8 and 507 with 5 + 4 (the MMAs take 512).
    const uint32_t pmax = (uint32_t)std::min(16, std::max(2, pmax_in)) & ~1u;
    const uint32_t wcap = (uint32_t)std::max(p.kcopies == 2 ? 4 : 1, std::min(16, wmax));
    const size_t budget = 225 * 1024 - fixed;
    uint32_t pfit = 0;
    for (p.wstages = std::min(wcap, 4u);; --p.wstages) {
        const size_t wb = (size_t)p.wstages * p.b_stage_bytes;
        pfit = wb < budget ? (uint32_t)((budget - wb) / kStageBytes) & ~1u : 0u;
        if (pfit >= 4 || p.wstages <= 2) break;
    }
    p.pstages = std::max(2u, std::min(pfit, pmax));
    while (p.wstages < wcap &&
           (size_t)(p.wstages + 1) * p.b_stage_bytes + (size_t)p.pstages * kStageBytes <= budget)
        ++p.wstages;
    // A wait by phase parity must know the use before the awaited one to be
    // over.  Two accumulator copies are worked on by two MMA warps that run
    // independently, in turns of group stages: their A and W slots stay with one
    // warp (a multiple of two turns deep; both fit whatever the caps).  With one
    // copy the MMAs complete in item order, and at most one unpack set per A
    // slot suffices.
    if (p.kcopies == 2) {
        p.slots = 4;
        p.wstages &= ~3u;
    }
    p.usets = std::min<uint32_t>(kUnpackSets, std::max(p.slots, 1u));
    p.smem = fixed + (size_t)p.pstages * kStageBytes + (size_t)p.wstages * p.b_stage_bytes;
    (void)tiles;
    p.ok = p.n_total % 8 == 0 && by_tmem >= 2 && p.slots >= 2 * p.parts && p.wstages >= 2 &&
           (size_t)p.wstages * p.b_stage_bytes + (size_t)p.pstages * kStageBytes <= budget &&
           p.n_main <= 512 && p.n_ind <= 256;
    return p;
}

Fp8Plan fp8_plan(int wpad, bool ind, uint64_t tiles, bool ind_shared) {
    return fp8_plan_knobs(wpad, ind, tiles, env_int("SLFMM_TC8_PSTAGES", 8), env_int("SLFMM_TC8_STAGES", 8),
                          env_int("SLFMM_TC8_GROUP", 4), env_int("SLFMM_TC8_WSTAGES", 8),
                          ind_shared && env_int("SLFMM_TC8_SHARED_IND", 1) != 0);
}

// row-major packed rows (rows x stride) -> tile-major copy; one thread per
// 16-byte output chunk, so the writes stream and every read is one full
// 32-byte sector
__global__ void k_tile_rows(const uint8_t* __restrict__ in, uint64_t rows, uint64_t stride, uint64_t kbt,
                            uint64_t chunks, uint8_t* __restrict__ out) {
    dependent_wait();
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < chunks;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t h = e & 1u, r = (e >> 1) & 127u, rest = e >> 8;
        const uint64_t kb = rest % kbt, t = rest / kbt;
        const uint64_t row = t * kM + r, col = kb * 32 + h * 16;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (row < rows && col < stride) v = *reinterpret_cast<const uint4*>(in + row * stride + col);
        reinterpret_cast<uint4*>(out)[e] = v;
    }
}

// 16 x 16 transpose of 2-bit codes, a row per word: swaps of 8, 4, 2 and 1 codes
// between the rows as far apart
__device__ __forceinline__ void transpose16(uint32_t (&w)[16]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t a = w[i], b = w[i + 8];
        w[i] = __byte_perm(a, b, 0x5410);
        w[i + 8] = __byte_perm(a, b, 0x7632);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (i & 4) continue;
        const uint32_t a = w[i], b = w[i + 4];
        w[i] = __byte_perm(a, b, 0x6240);
        w[i + 4] = __byte_perm(a, b, 0x7351);
    }
#pragma unroll
    for (int d = 2; d > 0; d >>= 1) {
        const uint32_t m = d == 2 ? 0x0f0f0f0fu : 0x33333333u;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i & d) continue;
            const uint32_t t = ((w[i] >> (2 * d)) ^ w[i + d]) & m;
            w[i + d] ^= t;
            w[i] ^= t << (2 * d);
        }
    }
}

// Tile-major transpose of the 2-bit matrix.  Block (t, kb) of the output --
// 128 samples of sample tile t x the 128 SNPs of K block kb -- is the 2-bit
// transpose of block (kb, t) of the SNP-row tiles; both are contiguous 4 KiB
// runs.  Four blocks per iteration, 64 threads to a block, a 16 x 16 square of
// codes each, in registers.  Both copies in shared memory keep the eight groups of
// 16 rows at a pitch that puts a warp's words on different banks.  The transpose
// moves 2 bytes per byte of output, and with a byte load, a shift and two logical
// operations per code it was bound by those: 200 000 x 8 500 274 us, 152 us so
// (130 us at the copy rate).
constexpr int kTrPitch = 128 + 8;     // words of 16 input rows
constexpr int kTrPitchOut = 128 + 4;  // words of 16 output rows
__global__ void __launch_bounds__(256) k_transpose_tiles(const uint8_t* __restrict__ src, uint64_t kbt_src,
                                                         uint64_t ntiles_src, uint8_t* __restrict__ dst,
                                                         uint64_t kbt_dst, uint64_t ntiles_dst, uint64_t kb_lo,
                                                         uint64_t kb_hi) {
    dependent_wait();
    __shared__ __align__(16) uint32_t in[4][8 * kTrPitch], out[4][8 * kTrPitchOut];
    const uint64_t nk = kb_hi - kb_lo;  // output K blocks [kb_lo, kb_hi) of every sample tile
    const uint64_t nblocks = ntiles_dst * nk;
    const int q = threadIdx.x >> 6, e = threadIdx.x & 63;
    const int bj = e & 7, bi = e >> 3;  // the square's 16 samples and 16 SNPs
    for (uint64_t b0 = (uint64_t)blockIdx.x * 4; b0 < nblocks; b0 += (uint64_t)gridDim.x * 4) {
        const uint64_t bb = b0 + q;
        const bool mine = bb < nblocks;
        const uint64_t t = mine ? bb / nk : 0, kb = kb_lo + (mine ? bb - t * nk : 0);
        const bool valid = mine && kb < ntiles_src && t < kbt_src;
        const uint4* s4 = reinterpret_cast<const uint4*>(src + (kb * kbt_src + t) * (uint64_t)kTileBytes);
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = valid ? s4[e + 64 * i] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // 32 vectors of four words to a group of rows
            const int at = e + 64 * i;
            *reinterpret_cast<uint4*>(&in[q][(at >> 5) * kTrPitch + 4 * (at & 31)]) = v[i];
        }
        __syncthreads();
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = in[q][bi * kTrPitch + 8 * i + bj];
        transpose16(w);
#pragma unroll
        for (int i = 0; i < 16; ++i) out[q][bj * kTrPitchOut + 8 * i + bi] = w[i];
        __syncthreads();
        if (mine) {
            uint4* d4 = reinterpret_cast<uint4*>(dst + (t * kbt_dst + kb) * (uint64_t)kTileBytes);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = e + 64 * i;
                d4[at] = *reinterpret_cast<const uint4*>(&out[q][(at >> 5) * kTrPitchOut + 4 * (at & 31)]);
            }
        }
    }
}

// Sample-major tiles of a sample subset: row rr of output sample tile ts
// (output sample s = 128 ts + rr) is row i % 128 of source tile i / 128, i =
// keep[s], in every K block; samples past n_keep are zero codes.  One thread
// per 16 bytes (two per 32-byte tile row).
__global__ void k_gather_tile_rows(const uint8_t* __restrict__ src, uint64_t kbt, const uint32_t* __restrict__ keep,
                                   uint64_t n_keep, uint64_t ntiles_dst, uint8_t* __restrict__ dst) {
    dependent_wait();
    const uint64_t total = ntiles_dst * kbt * 256;
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t h = e & 1u, rr = (e >> 1) & 127u, rest = e >> 8;
        const uint64_t kb = rest % kbt, ts = rest / kbt;
        const uint64_t sidx = ts * kM + rr;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (sidx < n_keep) {
            const uint64_t i = keep[sidx];
            v = s4[((i / kM) * kbt + kb) * 256 + (i % kM) * 2 + h];
        }
        d4[e] = v;
    }
}

// Allele and missing counts of every SNP from the SNP-major tiles (the
// codes of samples past n are 00 there): one warp per SNP, lanes over the
// K blocks of its tile row; counts as k_snp_counts (c0 = n - c1 - c2 - cm).
__global__ void k_snp_counts_tiles(const uint8_t* __restrict__ tiles, uint64_t kbt, uint64_t p, uint64_t n,
                                   int32_t* __restrict__ counts) {
    dependent_wait();
    constexpr uint32_t kLo2 = 0x55555555u;
    const uint64_t j = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (j >= p) return;
    const uint64_t t = j / kM, r = j % kM;
    uint32_t c1 = 0, c2 = 0, cm = 0;
    for (uint64_t kb = lane; kb < kbt; kb += 32) {
        const uint4* q = reinterpret_cast<const uint4*>(tiles + (t * kbt + kb) * kTileBytes + r * 32);
        const uint4 a = q[0], b = q[1];
        const uint32_t ws[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t lo = ws[k] & kLo2, hi = (ws[k] >> 1) & kLo2;
            c1 += __popc(hi & ~lo);
            c2 += __popc(hi & lo);
            cm += __popc(~hi & lo);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c1 += __shfl_xor_sync(0xffffffffu, c1, o);
        c2 += __shfl_xor_sync(0xffffffffu, c2, o);
        cm += __shfl_xor_sync(0xffffffffu, cm, o);
    }
    if (lane == 0) {
        counts[j * 4 + 0] = (int32_t)(n - c1 - c2 - cm);
        counts[j * 4 + 1] = (int32_t)c1;
        counts[j * 4 + 2] = (int32_t)c2;
        counts[j * 4 + 3] = (int32_t)cm;
    }
}

// Missing-call lists (CSR by SNP, ascending sample indices) of a matrix held
// only as SNP-major tiles: one warp per SNP, lanes over 32 K blocks at a
// time; a lane's missing calls (code 01) are placed after those of the lower
// lanes by a warp scan of the per-lane counts.
__global__ void k_miss_fill_tiles(const uint8_t* __restrict__ tiles, uint64_t kbt, uint64_t p,
                                  const uint64_t* __restrict__ ptr, uint32_t* __restrict__ idx) {
    dependent_wait();
    constexpr uint32_t kLo2 = 0x55555555u;
    const uint64_t j = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (j >= p) return;
    const uint64_t t = j / kM, r = j % kM;
    uint64_t base = ptr[j];
    for (uint64_t kb0 = 0; kb0 < kbt; kb0 += 32) {
        const uint64_t kb = kb0 + lane;
        uint32_t m[8];
        int cnt = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) m[k] = 0u;
        if (kb < kbt) {
            const uint4* q = reinterpret_cast<const uint4*>(tiles + (t * kbt + kb) * kTileBytes + r * 32);
            const uint4 a = q[0], b = q[1];
            const uint32_t ws[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                m[k] = ws[k] & kLo2 & ~((ws[k] >> 1) & kLo2);
                cnt += __popc(m[k]);
            }
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        uint64_t pos = base + (uint64_t)(incl - cnt);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint32_t mm = m[k];
            while (mm) {
                const int bit = __ffs(mm) - 1;
                idx[pos++] = (uint32_t)(kb * 128 + k * 16 + bit / 2);
                mm &= mm - 1;
            }
        }
        base += (uint64_t)__shfl_sync(0xffffffffu, incl, 31);
    }
}

__global__ void k_miss_counts_of(const int32_t* __restrict__ counts, uint64_t p, uint64_t* __restrict__ mc) {
    dependent_wait();
    for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < p; j += (uint64_t)gridDim.x * blockDim.x)
        mc[j] = (uint64_t)counts[j * 4 + 3];
}

void launch_miss_counts_of(Ctx& c, const Geno& g, uint64_t* mc) {
    if (!g.p) return;
    launch_next(c, k_miss_counts_of, grid_for(c, g.p, 256), 256, 0, g.counts.get(), g.p, mc);
    SLFMM_LAUNCHED(c, "k_miss_counts_of");
}

void launch_miss_fill_tiles(Ctx& c, const Geno& g) {
    SLFMM_REQUIRE(g.have_tiles, SLFMM_ERR_BAD_ARG, "this matrix has neither a row-major copy nor SNP-major tiles");
    if (!g.p) return;
    launch_next(c, k_miss_fill_tiles, (unsigned)ceil_div(g.p * 32, 256), 256, 0, g.tiles.get(), g.kbt, g.p,
                                                                               g.miss_ptr.get(), g.miss_idx.get());
    SLFMM_LAUNCHED(c, "k_miss_fill_tiles");
}

static void tile_rows(Ctx& c, const uint8_t* in, uint64_t rows, uint64_t stride, DBuf<uint8_t>& out, uint64_t& kbt,
                      uint64_t& ntiles) {
    SLFMM_REQUIRE(stride % 32 == 0, SLFMM_ERR_BAD_ARG, "packed stride must be a multiple of 32 bytes");
    kbt = stride / 32;
    ntiles = round_up(std::max<uint64_t>(ceil_div(rows, kM), 1), 8);
    const uint64_t bytes = ntiles * kbt * kTileBytes;
    out.alloc(bytes, c.stream);
    const uint64_t chunks = bytes / 16;
    launch_next(c, k_tile_rows, grid_for(c, chunks, 256), 256, 0, in, rows, stride, kbt, chunks, out.get());
    SLFMM_LAUNCHED(c, "k_tile_rows");
}

// four 4 KiB blocks to a CTA, as many CTAs as are resident (34 KB each)
static unsigned transpose_grid(const Ctx& c, uint64_t blocks) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(blocks, 4), (uint64_t)c.sm_count * 6));
}

// Tile-major copies built chunk by chunk while a matrix is uploaded: rows
// [r0, r1) of the SNP-major matrix (r0 a multiple of 128) are tiled and
// transposed as soon as they land.  `last` also writes the padding tiles.
void tile_chunk(Ctx& c, const Geno& g, uint64_t r0, uint64_t r1, bool last) {
    SLFMM_REQUIRE(r0 % kM == 0, SLFMM_ERR_BAD_ARG, "upload chunks must start on a 128-row tile");
    if (r0 == 0) {
        SLFMM_REQUIRE(g.stride % 32 == 0, SLFMM_ERR_BAD_ARG, "packed stride must be a multiple of 32 bytes");
        g.kbt = g.stride / 32;
        g.ntiles = round_up(std::max<uint64_t>(ceil_div(g.p, kM), 1), 8);
        g.tiles.alloc(g.ntiles * g.kbt * kTileBytes, c.stream);
        g.kbtT = round_up(std::max<uint64_t>(ceil_div(g.p, kM), 1), kHalves);
        g.ntilesT = round_up(std::max<uint64_t>(ceil_div(g.n, kM), 1), 8);
        g.tilesT.alloc(g.ntilesT * g.kbtT * kTileBytes, c.stream);
    }
    const uint64_t t0 = r0 / kM, t1 = last ? g.ntiles : ceil_div(r1, kM);
    const uint64_t chunks = (t1 - t0) * g.kbt * (kTileBytes / 16);
    launch_next(c, k_tile_rows, grid_for(c, chunks, 256), 256, 0, packed_rows(g) + r0 * g.stride, r1 - r0, g.stride,
                                                                 g.kbt, chunks,
                                                                 g.tiles.get() + t0 * g.kbt * kTileBytes);
    SLFMM_LAUNCHED(c, "k_tile_rows");
    const uint64_t k1 = last ? g.kbtT : std::min(g.kbtT, ceil_div(r1, kM));
    if (k1 > t0) {
        const unsigned blocks = transpose_grid(c, g.ntilesT * (k1 - t0));
        launch_next(c, k_transpose_tiles, blocks, 256, 0, g.tiles.get(), g.kbt, g.ntiles, g.tilesT.get(),
                                                                   g.kbtT, g.ntilesT, t0, k1);
        SLFMM_LAUNCHED(c, "k_transpose_tiles");
    }
    if (last) g.have_tiles = g.have_tilesT = true;
}

void tiles_subset_samples(Ctx& c, const Geno& full, const uint32_t* keep_dev, uint64_t n_keep, Geno& sub) {
    SLFMM_REQUIRE(n_keep > 0 && n_keep <= full.n, SLFMM_ERR_BAD_ARG, "bad sample subset");
    build_tiles(c, full, true);
    sub.n = n_keep;
    sub.p = full.p;
    sub.stride = round_up(ceil_div(n_keep, 4), 128);
    // sample-major: the kept samples' rows of the full matrix's tiles
    sub.kbtT = full.kbtT;
    sub.ntilesT = round_up(std::max<uint64_t>(ceil_div(n_keep, kM), 1), 8);
    sub.tilesT.alloc(sub.ntilesT * sub.kbtT * kTileBytes, c.stream);
    const uint64_t rows16 = sub.ntilesT * sub.kbtT * 256;
    launch_next(c, k_gather_tile_rows, grid_for(c, rows16, 256), 256, 0, full.tilesT.get(), full.kbtT, keep_dev, n_keep,
                                                                       sub.ntilesT, sub.tilesT.get());
    SLFMM_LAUNCHED(c, "k_gather_tile_rows");
    // SNP-major: the 2-bit transpose of those blocks
    sub.kbt = sub.stride / 32;
    sub.ntiles = round_up(std::max<uint64_t>(ceil_div(sub.p, kM), 1), 8);
    sub.tiles.alloc(sub.ntiles * sub.kbt * kTileBytes, c.stream);
    const unsigned blocks = transpose_grid(c, sub.ntiles * sub.kbt);
    launch_next(c, k_transpose_tiles, blocks, 256, 0, sub.tilesT.get(), sub.kbtT, sub.ntilesT,
                sub.tiles.get(),
                                                               sub.kbt, sub.ntiles, 0, sub.kbt);
    SLFMM_LAUNCHED(c, "k_transpose_tiles");
    sub.have_tiles = sub.have_tilesT = true;
    sub.counts.alloc(std::max<uint64_t>(sub.p, 1) * 4, c.stream);
    if (sub.p) {
        launch_next(c, k_snp_counts_tiles, (unsigned)ceil_div(sub.p * 32, 256), 256, 0, sub.tiles.get(), sub.kbt, sub.p,
                                                                                      sub.n, sub.counts.get());
        SLFMM_LAUNCHED(c, "k_snp_counts_tiles");
    }
}

TileView build_tiles(Ctx& c, const Geno& g, bool transposed) {
    if (!transposed) {
        if (!g.have_tiles) {
            tile_rows(c, packed_rows(g), g.p, g.stride, g.tiles, g.kbt, g.ntiles);
            g.have_tiles = true;
        }
        return TileView{g.tiles.get(), g.kbt, g.ntiles};
    }
    if (!g.have_tilesT) {
        // straight from the SNP-row tiles: sample tiles x K blocks of 128 SNPs
        build_tiles(c, g, false);
        g.kbtT = round_up(std::max<uint64_t>(ceil_div(g.p, kM), 1), kHalves);  // whole stages
        g.ntilesT = round_up(std::max<uint64_t>(ceil_div(g.n, kM), 1), 8);
        g.tilesT.alloc(g.ntilesT * g.kbtT * kTileBytes, c.stream);
        const unsigned blocks = transpose_grid(c, g.ntilesT * g.kbtT);
        launch_next(c, k_transpose_tiles, blocks, 256, 0, g.tiles.get(), g.kbt, g.ntiles, g.tilesT.get(),
                                                                   g.kbtT, g.ntilesT, 0, g.kbtT);
        SLFMM_LAUNCHED(c, "k_transpose_tiles");
        g.have_tilesT = true;
    }
    return TileView{g.tilesT.get(), g.kbtT, g.ntilesT};
}

// blocks of k_colmax_abs: few enough for their atomics, eight warps with four
// rows in flight each
static unsigned colmax_blocks(const Ctx& c, uint64_t K) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(K, 32), (uint64_t)c.sm_count * 4));
}

void launch_fp8_terms_f64(Ctx& c, const double* src, int ld, uint64_t K, int w, int wpad, uint64_t K_pad,
                          int ind_row_off, int n_rows, uint8_t* B, float* inv_scale) {
    DBuf<unsigned> cm(wpad, c.stream);
    cm.zero();
    SLFMM_REQUIRE(w >= 1 && w <= 128 && wpad <= 128, SLFMM_ERR_BAD_ARG, "operand wider than 128 columns");
    SLFMM_REQUIRE(n_rows % 8 == 0 && kMainTerms * wpad <= n_rows && ind_row_off % 8 == 0 &&
                      (!ind_row_off || ind_row_off + kIndTerms * wpad <= n_rows) && wpad % kTermCols == 0 &&
                      K_pad % kStageK == 0,
                  SLFMM_ERR_BAD_ARG, "bad stage-major operand shape");
    launch_next(c, k_colmax_abs<double>, colmax_blocks(c, K), 256, 0, src, ld, K, w, nullptr, cm.get());
    SLFMM_LAUNCHED(c, "k_colmax_abs");
    const TermSet sa{nullptr, kMainTerms, 0, cm.get()};
    const TermSet sb{nullptr, ind_row_off ? kIndTerms : 0, ind_row_off, cm.get()};
    dim3 grid((unsigned)(K_pad / kStageK), (unsigned)(wpad / kTermCols));
    launch_next(c, k_fp8_terms<double>, grid, 256, 0, src, ld, K, w, wpad, sa, sb, n_rows, B, inv_scale);
    SLFMM_LAUNCHED(c, "k_fp8_terms");
}

void launch_fp8_terms_f32_pair(Ctx& c, const float* src, int ld, uint64_t K, int w, int wpad, uint64_t K_pad,
                               const double* ks_main, const double* ks_ind, int ind_row_off, int n_rows, uint8_t* B,
                               float* inv_scale) {
    SLFMM_REQUIRE(w >= 1 && w <= 128 && wpad <= 128, SLFMM_ERR_BAD_ARG, "operand wider than 128 columns");
    SLFMM_REQUIRE(n_rows % 8 == 0 && kMainTerms * wpad <= n_rows &&
                      (!ks_ind || (ind_row_off % 8 == 0 && ind_row_off + kIndTerms * wpad <= n_rows)) &&
                      wpad % kTermCols == 0 && K_pad % kStageK == 0,
                  SLFMM_ERR_BAD_ARG, "bad stage-major operand shape");
    DBuf<unsigned> cm(2 * (uint64_t)wpad, c.stream);
    cm.zero();
    unsigned* cma = cm.get();
    unsigned* cmb = ks_ind ? cm.get() + wpad : nullptr;
    const bool quads = ld % 4 == 0 && ld <= 32 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
    if (quads) {
        const unsigned blocks = (unsigned)std::max<uint64_t>(
            1, std::min<uint64_t>(ceil_div(K * (uint64_t)(ld / 4), 1024), (uint64_t)c.sm_count * 4));
        launch_next(c, k_colmax_pair, blocks, 256, 0, src, ld, K, w, ks_main, ks_ind, cma, cmb);
        SLFMM_LAUNCHED(c, "k_colmax_pair");
    } else {
        launch_next(c, k_colmax_abs<float>, colmax_blocks(c, K), 256, 0, src, ld, K, w, ks_main, cma);
        SLFMM_LAUNCHED(c, "k_colmax_abs");
        if (ks_ind) {
            launch_next(c, k_colmax_abs<float>, colmax_blocks(c, K), 256, 0, src, ld, K, w, ks_ind, cmb);
            SLFMM_LAUNCHED(c, "k_colmax_abs");
        }
    }
    const TermSet sa{ks_main, kMainTerms, 0, cma};
    const TermSet sb{ks_ind, ks_ind ? kIndTerms : 0, ind_row_off, cmb};
    dim3 grid((unsigned)(K_pad / kStageK), (unsigned)(wpad / kTermCols));
    launch_next(c, k_fp8_terms<float>, grid, 256, 0, src, ld, K, w, wpad, sa, sb, n_rows, B, inv_scale);
    SLFMM_LAUNCHED(c, "k_fp8_terms");
}

int Tc8Errors::read() {
    int h = 0;
    SLFMM_CUDA(cudaMemcpyAsync(&h, flag.get(), sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    SLFMM_CUDA(cudaStreamSynchronize(c.stream));
    return h;
}

void throw_tc8_timeout(int site) {
    throw Error(SLFMM_ERR_DEVICE_TIMEOUT,
                "split-FP8 contraction: a bounded device wait expired (site " + std::to_string(site) + ")");
}

static int tc8_launch(Ctx& c, const Fp8Plan& pl, const TileView& tv, uint64_t rows, uint64_t K, const uint8_t* B,
                      const float* inv_scale, uint64_t K_pad, int mode, const double* row_mean,
                      const double* row_scale, const double* cs, float* out, int ldo, int splits,
                      uint64_t split_stride, int* err_dev);

// Autotuner: the ring depths (packed codes, W stages) of a plan, timed on
// two waves of the real pass and cached per context and shape.  Only knobs
// that leave the arithmetic alone are tuned: the candidates keep the default
// plan's MMA wait group and accumulator layout, so every choice gives the
// same bits.
static Fp8Plan tc8_tuned_plan(Ctx& c, const Fp8Plan& pl, const TileView& tv, uint64_t rows, uint64_t K,
                              const uint8_t* B, const float* inv_scale, uint64_t K_pad, int mode,
                              const double* row_mean, const double* row_scale, const double* cs, int ldo, int splits,
                              uint64_t split_stride) {
    const std::string key = std::to_string(pl.wpad) + "/" + std::to_string(pl.n_ind) + "/" + std::to_string(K) +
                            "/" + std::to_string(splits) + "/" + std::to_string(mode) + "/" +
                            std::to_string(pl.ind_shared);
    auto rebuild = [&](int pmax, int smax) {
        return fp8_plan_knobs((int)pl.wpad, pl.n_ind != 0, ceil_div(rows, (uint64_t)kM), pmax, smax, (int)pl.group,
                              env_int("SLFMM_TC8_WSTAGES", 8), pl.ind_shared != 0);
    };
    auto it = c.tuned.find(key);
    if (it != c.tuned.end()) return rebuild(it->second.first, it->second.second);
    const uint64_t trial_rows = std::min<uint64_t>(rows, (uint64_t)c.sm_count * 2 * kM);
    DBuf<float> scratch(std::max<uint64_t>(trial_rows, 1) * (uint64_t)ldo * std::max(splits, 1), c.stream);
    cudaEvent_t e0, e1;
    SLFMM_CUDA(cudaEventCreate(&e0));
    SLFMM_CUDA(cudaEventCreate(&e1));
    struct EvGuard {
        cudaEvent_t a, b;
        ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); }
    } guard{e0, e1};
    DBuf<int> err(1, c.stream);
    err.zero();
    float best = 1e30f;
    std::pair<int, int> pick{8, 8};
    for (int pmax : {2, 4, 8, 16})
        for (int smax : {2, 3, 4, 8}) {
            const Fp8Plan q = rebuild(pmax, smax);
            if (!q.ok || q.group != pl.group || q.kcopies != pl.kcopies) continue;
            float ms = 1e30f;
            for (int rep = 0; rep < 2; ++rep) {
                SLFMM_CUDA(cudaEventRecord(e0, c.stream));
                tc8_launch(c, q, tv, trial_rows, K, B, inv_scale, K_pad, mode, row_mean, row_scale, cs,
                           scratch.get(), ldo, splits, trial_rows * (uint64_t)ldo, err.get());
                SLFMM_CUDA(cudaEventRecord(e1, c.stream));
                SLFMM_CUDA(cudaEventSynchronize(e1));
                float t = 0.f;
                SLFMM_CUDA(cudaEventElapsedTime(&t, e0, e1));
                ms = std::min(ms, t);
            }
            if (ms < best) {
                best = ms;
                pick = {pmax, smax};
            }
        }
    int h = 0;
    SLFMM_CUDA(cudaMemcpyAsync(&h, err.get(), sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    SLFMM_CUDA(cudaStreamSynchronize(c.stream));
    if (h != 0) throw_tc8_timeout(h);
    c.tuned[key] = pick;
    if (c.verbose)
        fprintf(stderr, "[schnelgpu] autotune %s: packed ring cap %d, W ring cap %d (%.3f ms on %llu rows)\n",
                key.c_str(), pick.first, pick.second, best, (unsigned long long)trial_rows);
    return rebuild(pick.first, pick.second);
}

int launch_tc8_rows(Ctx& c, const Fp8Plan& pl, const TileView& tv, uint64_t rows, uint64_t K,
                    const uint8_t* B, const float* inv_scale, uint64_t K_pad, int mode, const double* row_mean,
                    const double* row_scale, const double* cs, float* out, int ldo, int splits,
                    uint64_t split_stride, int* err_dev) {
    if (c.autotune && pl.ok && rows > 0) {
        const Fp8Plan tp = tc8_tuned_plan(c, pl, tv, rows, K, B, inv_scale, K_pad, mode, row_mean, row_scale, cs, ldo,
                                          splits, split_stride);
        if (tp.ok) return tc8_launch(c, tp, tv, rows, K, B, inv_scale, K_pad, mode, row_mean, row_scale, cs, out, ldo,
                                     splits, split_stride, err_dev);
    }
    return tc8_launch(c, pl, tv, rows, K, B, inv_scale, K_pad, mode, row_mean, row_scale, cs, out, ldo, splits,
                      split_stride, err_dev);
}

static int tc8_launch(Ctx& c, const Fp8Plan& pl, const TileView& tv, uint64_t rows, uint64_t K, const uint8_t* B,
                      const float* inv_scale, uint64_t K_pad, int mode, const double* row_mean,
                      const double* row_scale, const double* cs, float* out, int ldo, int splits,
                      uint64_t split_stride, int* err_dev) {
    SLFMM_REQUIRE(pl.ok, SLFMM_ERR_BAD_ARG, "no feasible split-FP8 tile plan for this width");
    SLFMM_REQUIRE(K_pad % kStageK == 0 && K_pad >= ceil_div(K, kStageK) * kStageK, SLFMM_ERR_BAD_ARG,
                  "bad K padding");
    SLFMM_REQUIRE(tv.base && tv.kbt % kHalves == 0 && tv.kbt >= ceil_div(K, kStageK) * kHalves, SLFMM_ERR_BAD_ARG,
                  "tile-major operand too short in K");
    SLFMM_REQUIRE(tv.ntiles >= ceil_div(rows, kM), SLFMM_ERR_BAD_ARG,
                  "tile-major operand has too few tiles");
    SLFMM_REQUIRE(mode == 0 || pl.n_ind != 0, SLFMM_ERR_BAD_ARG, "row correction needs the indicator operand");
    SLFMM_REQUIRE(reinterpret_cast<uintptr_t>(B) % 16 == 0 && pl.b_stage_bytes % 16 == 0, SLFMM_ERR_BAD_ARG,
                  "W operand not 16-byte aligned");
    raise_dynamic_smem((const void*)k_tc8_rows, pl.smem);
    DBuf<int> err;
    if (!err_dev) err_dev = c.tc8_err;
    if (!err_dev) {
        err.alloc(1, c.stream);
        err.zero();
    }
    Tc8Args a{};
    a.rows = (uint32_t)rows;
    a.kb_total = (uint32_t)ceil_div(K, kStageK);
    a.kb_per_split = (uint32_t)ceil_div(a.kb_total, (uint64_t)std::max(splits, 1));
    a.wpad = pl.wpad;
    a.n_main = pl.n_main;
    a.n_ind = pl.n_ind;
    a.n_total = pl.n_total;
    a.ind_shared = pl.ind_shared;
    a.d_cols = pl.d_cols;
    a.a_cols = pl.a_cols;
    a.parts = pl.parts;
    a.slots = pl.slots;
    a.wstages = pl.wstages;
    a.pstages = pl.pstages;
    a.group = pl.group;
    a.kcopies = pl.kcopies;
    a.a_base = pl.a_base;
    a.usets = pl.usets;
    a.none = 0;
    a.tmem_cols = pl.tmem_cols;
    a.b_stage_bytes = pl.b_stage_bytes;
    a.inv_scale = inv_scale;
    a.wop = B;
    a.expire_cycles = c.expire_next_wait;
    a.tile0 = (uint32_t)tv.tile0;
    a.rotate = (uint32_t)env_int("SLFMM_TC8_ROTATE", 1);  // tuning override
    c.expire_next_wait = 0;
    a.mode = mode;
    a.row_mean = row_mean;
    a.row_scale = row_scale;
    a.cs = cs;
    a.out = out;
    a.ldo = (uint32_t)ldo;
    a.split_stride = split_stride;
    a.tiles = tv.base;
    a.tile_bytes = tv.kbt * (uint64_t)kTileBytes;
    a.err = err_dev ? err_dev : err.get();
    const unsigned gy = (unsigned)ceil_div(a.kb_total, a.kb_per_split);
    const unsigned gx = (unsigned)ceil_div(rows, kM);
    a.gx = gx;
    a.units = gx * gy;
    // one CTA per SM working through the units (SLFMM_TC8_PERSIST=0: one CTA
    // per unit; the same code and bits either way)
    const unsigned ctas = env_int("SLFMM_TC8_PERSIST", 1) != 0
                              ? std::min<unsigned>(a.units, (unsigned)std::max(c.sm_count, 1))
                              : a.units;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(std::max(ctas, 1u), 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = c.stream;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, k_tc8_rows, a);
    if (le != cudaSuccess) {
        cudaGetLastError();
        char buf[320];
        snprintf(buf, sizeof buf,
                 "split-FP8 contraction launch failed (%s): units %u x %u, smem %zu, slots %u, stages %u, pstages %u, "
                 "group %u, n_total %u, rows %llu, K %llu",
                 cudaGetErrorString(le), gx, gy, pl.smem, pl.slots, pl.wstages, pl.pstages, pl.group, pl.n_total,
                 (unsigned long long)rows, (unsigned long long)K);
        throw Error(SLFMM_ERR_CUDA, buf);
    }
    SLFMM_LAUNCHED(c, "k_tc8_rows");
    if (err_dev) return (int)gy;
    int h = 0;
    SLFMM_CUDA(cudaMemcpyAsync(&h, err.get(), sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    SLFMM_CUDA(cudaStreamSynchronize(c.stream));
    if (h != 0) throw_tc8_timeout(h);
    return (int)gy;
}

void launch_sub_colterm(Ctx& c, double* S, int lds, uint64_t n, int w, const double* colterm) {
    if (!n || !w) return;
    launch_next(c, k_sub_colterm, grid_for(c, n * w, 256), 256, 0, S, lds, n, w, colterm);
    SLFMM_LAUNCHED(c, "k_sub_colterm");
}

}  // namespace slfmm
