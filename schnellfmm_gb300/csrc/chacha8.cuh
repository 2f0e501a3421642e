// ChaCha8Rng::seed_from_u64(seed) on the device: output `ctr` is keystream
// words 2 ctr and 2 ctr + 1 (block ctr / 8: 64-bit block counter in state words
// 12-13, stream id 0), the key 8 PCG32 XSH-RR outputs of the seed -- the stream
// host_rng.cpp describes.  The last block stays in registers, so consecutive
// counters reuse it.
#pragma once
#include <cstdint>

namespace slfmm {

__device__ __forceinline__ void chacha_quarter(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
    a += b; d ^= a; d = __funnelshift_l(d, d, 16);
    c += d; b ^= c; b = __funnelshift_l(b, b, 12);
    a += b; d ^= a; d = __funnelshift_l(d, d, 8);
    c += d; b ^= c; b = __funnelshift_l(b, b, 7);
}

struct ChaCha8Draws {
    uint32_t key[8];
    uint32_t x[16];
    uint64_t blk;
    __device__ explicit ChaCha8Draws(uint64_t seed) : blk(~0ull) {
        uint64_t s = seed;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            s = s * 6364136223846793005ull + 11634580027462260723ull;
            const uint32_t xs = (uint32_t)(((s >> 18) ^ s) >> 27);
            key[j] = __funnelshift_r(xs, xs, (uint32_t)(s >> 59));
        }
    }
    __device__ void refill() {
        const uint32_t in[16] = {0x61707865u, 0x3320646eu, 0x79622d32u, 0x6b206574u, key[0], key[1], key[2], key[3],
                                 key[4], key[5], key[6], key[7], (uint32_t)blk, (uint32_t)(blk >> 32), 0u, 0u};
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = in[i];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            chacha_quarter(x[0], x[4], x[8], x[12]);
            chacha_quarter(x[1], x[5], x[9], x[13]);
            chacha_quarter(x[2], x[6], x[10], x[14]);
            chacha_quarter(x[3], x[7], x[11], x[15]);
            chacha_quarter(x[0], x[5], x[10], x[15]);
            chacha_quarter(x[1], x[6], x[11], x[12]);
            chacha_quarter(x[2], x[7], x[8], x[13]);
            chacha_quarter(x[3], x[4], x[9], x[14]);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] += in[i];
    }
    __device__ uint64_t at(uint64_t ctr) {
        if ((ctr >> 3) != blk) {
            blk = ctr >> 3;
            refill();
        }
        return word((int)(ctr & 7));
    }
    // output j (0..7) of the block in registers
    __device__ uint64_t word(int j) const {
        uint32_t lo = x[0], hi = x[1];
#pragma unroll
        for (int w = 1; w < 8; ++w)
            if (w == j) {
                lo = x[2 * w];
                hi = x[2 * w + 1];
            }
        return (uint64_t)lo | ((uint64_t)hi << 32);
    }
};

}  // namespace slfmm
