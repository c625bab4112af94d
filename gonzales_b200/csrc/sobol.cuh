// sobol.cuh - Z-Sobol sampler on the device (Sources/libgonzales/Sampler/
// ZSobolSampler.swift:6-280).  The integer path (Morton index, base-4 digit
// permutation, matrix product, Owen scramble) is bit-exact with the
// reference; the final value is (float)bits * 2^-32 clamped to 1 - 1e-6.
#pragma once

#include <stdint.h>

namespace gzg {

constexpr int kSobolDims = 1024;
constexpr int kSobolColumns = 52;
// Per dimension: the xor of the first 32 matrix columns over each 4-bit group
// of index bits, [8 groups][16 values] (512 KB for all dimensions).
constexpr int kSobolNibbleWords = 8 * 16;

struct ZSobol {
        uint64_t morton;  // (Morton(px, py) << log2spp) | sample index
        int32_t dim;      // next dimension
};

struct ZSobolConfig {
        const uint32_t *matrices;  // kSobolDims x kSobolColumns
        const uint32_t *nibbles;   // kSobolDims x kSobolNibbleWords
        uint64_t seed;             // sampler seed (1234, Sampler/Random.swift:66)
        int32_t log2spp;
        int32_t n_base4_digits;
};

__device__ __forceinline__ uint32_t zs_reverse_bits(uint32_t v) { return __brev(v); }

// mixBits (ZSobolSampler.swift:90-101): the 64-bit argument folded to 32
// bits by xor, then the 32-bit finaliser.
__device__ __forceinline__ uint32_t zs_mix_bits32(uint32_t x) {
        x ^= x >> 16;
        x *= 0x85ebca77u;
        x ^= x >> 13;
        x *= 0xc2b2ae35u;
        x ^= x >> 16;
        return x;
}
__device__ __forceinline__ uint32_t zs_mix_bits(uint64_t v) {
        return zs_mix_bits32((uint32_t)(v & 0xFFFFFFFFull) ^ (uint32_t)(v >> 32));
}

// FastOwenScrambler (ZSobolSampler.swift:43-67).
__device__ __forceinline__ uint32_t zs_owen(uint32_t v, uint32_t seed) {
        v = __brev(v);
        v ^= v * 0x3d20adeau;
        v += seed;
        v *= (seed >> 16) | 1u;
        v ^= v * 0x05526c56u;
        v ^= v * 0x53a22864u;
        return __brev(v);
}

// encodeMorton2 (ZSobolSampler.swift:70-88).
__device__ __forceinline__ uint64_t zs_morton2(uint32_t x, uint32_t y) {
        uint64_t a = x, b = y;
        a = (a | (a << 16)) & 0x0000FFFF0000FFFFull;
        a = (a | (a << 8)) & 0x00FF00FF00FF00FFull;
        a = (a | (a << 4)) & 0x0F0F0F0F0F0F0F0Full;
        a = (a | (a << 2)) & 0x3333333333333333ull;
        a = (a | (a << 1)) & 0x5555555555555555ull;
        b = (b | (b << 16)) & 0x0000FFFF0000FFFFull;
        b = (b | (b << 8)) & 0x00FF00FF00FF00FFull;
        b = (b | (b << 4)) & 0x0F0F0F0F0F0F0F0Full;
        b = (b | (b << 2)) & 0x3333333333333333ull;
        b = (b | (b << 1)) & 0x5555555555555555ull;
        return a | (b << 1);
}

__device__ __forceinline__ uint64_t zs_shr(uint64_t v, int s) { return s >= 64 ? 0ull : (v >> s); }
__device__ __forceinline__ uint32_t zs_shr32(uint32_t v, int s) { return s >= 32 ? 0u : (v >> s); }

// The 24 permutations of ZSobolSampler.swift:105-112, two bits per entry, one
// byte per permutation (entry d of permutation p = (byte p >> (2 * d)) & 3),
// laid out for a 256-byte shared table indexed by the top byte b of a hash:
// entry b is permutation b % 24, so the table repeats these six words.
__constant__ const uint32_t kZsPermWords[6] = {0x78d8b4e4u, 0xb1e19c6cu, 0x8d2d39c9u,
                                               0x72d236c6u, 0x87271e4eu, 0x93634b1bu};

// One table per block.  64 words in 32 banks: any access pattern of a warp
// takes at most two wavefronts.
__device__ __forceinline__ uint32_t *zs_perm_table() {
        __shared__ uint32_t table[64];
        return table;
}

// Fills the block's permutation table; every thread of the block calls it
// before any of them draws a sample or returns.
__device__ __forceinline__ void zs_block_init() {
        uint32_t *t = zs_perm_table();
        for (unsigned i = threadIdx.x; i < 64u; i += blockDim.x) t[i] = kZsPermWords[i % 6u];
        __syncthreads();
}

// A draw's dimensions: the one its hashes use, and the first matrix dimension
// (they part only where the sampler wraps around past its last dimension).
struct ZSlot {
        int32_t hash, base;
};
// Takes the next n dimensions (get1D / get2D / get3D, ZSobolSampler.swift:
// 203-280, advance the sampler this way).  A draw whose values are not needed
// takes its dimensions and nothing else.
__device__ __forceinline__ ZSlot zs_take(ZSobol &s, int n) {
        ZSlot r;
        r.hash = s.dim;
        if (s.dim + (n - 1) >= kSobolDims) s.dim = 2;
        r.base = s.dim;
        s.dim += n;
        return r;
}

// Whether every index of this path fits 32 bits (2048 x 2048 pixels at up to
// 1024 spp, say): the index permutation then runs in 32-bit arithmetic and the
// matrix products come from the nibble tables.
__device__ __forceinline__ bool zs_fits32(const ZSobolConfig &c, const ZSobol &s) {
        return (s.morton >> 32) == 0 && c.n_base4_digits <= 16;
}

// getSampleIndex in 64-bit arithmetic (ZSobolSampler.swift:138-166) for the
// frames that need it, out of line: the draws' code stays small (the shade
// kernels wait on instruction fetches as it is).
__device__ __noinline__ uint64_t zs_index64(int log2spp, int n_base4_digits, uint64_t morton, int dim) {
        uint64_t idx = 0;
        const bool pow2 = (log2spp & 1) == 1;
        const int last = pow2 ? 1 : 0;
        const uint64_t dmul = 0x55555555ull * (uint64_t)(int64_t)dim;
        for (int di = n_base4_digits - 1; di >= last; --di) {
                const int shift = 2 * di - (pow2 ? 1 : 0);
                const int digit = (int)(zs_shr(morton, shift) & 3u);
                const uint64_t higher = zs_shr(morton, shift + 2);
                const uint32_t e = reinterpret_cast<const uint8_t *>(zs_perm_table())[zs_mix_bits(higher ^ dmul) >> 24];
                idx |= (uint64_t)((e >> (2 * digit)) & 3u) << shift;
        }
        if (pow2) {
                int digit = (int)(morton & 1u);
                const uint32_t h = zs_mix_bits((morton >> 1) ^ dmul);
                digit ^= (int)(h & 1u);
                idx |= (uint64_t)digit;
        }
        return idx;
}

// sobolSample's matrix product (ZSobolSampler.swift:6-31) by scanning the
// index bits, for indices above 32 bits.
__device__ __noinline__ uint32_t zs_sobol64(const uint32_t *m, uint64_t index) {
        uint32_t acc = 0;
        while (index != 0) {
                const int bit = __ffsll((long long)index) - 1;
                if (bit >= kSobolColumns) break;
                acc ^= __ldg(m + bit);
                index &= index - 1;
        }
        return acc;
}

// getSampleIndex of a draw in 32-bit arithmetic.  Every base-4 digit of the
// Morton index is permuted by a hash of the digits above it and the draw's
// dimension.  mixBits folds its argument to 32 bits by xor, so the argument is
// (digits above) ^ fold(dim x 0x55555555), and its first step x ^= x >> 16
// distributes over that xor: the dimension's half leaves the loop.  Only the top
// byte of the hash is used (its last step leaves that byte alone), and it picks
// the permutation from the block's table.  About 10 instructions per digit, where
// h % 24 and register-selected permutations took 28.  The shade kernels are bound
// by integer issue, mostly the sampler's: with this, the nibble tables below and
// no values drawn that nothing reads, the box-scene frame (256 x 256, 16 spp,
// depth 5) went 1,387 -> 1,108 us, the adjoint step 4.64 -> 3.75 ms, the two-level
// frame with layered materials 30.9 -> 29.3 ms.
__device__ __forceinline__ uint32_t zs_index32(const ZSobolConfig &c, uint32_t morton, int dim) {
        const uint8_t *perm = reinterpret_cast<const uint8_t *>(zs_perm_table());
        const uint64_t dmul = 0x55555555ull * (uint64_t)(int64_t)dim;
        const uint32_t fold = (uint32_t)(dmul & 0xFFFFFFFFull) ^ (uint32_t)(dmul >> 32);
        const uint32_t mixed = fold ^ (fold >> 16);
        const int odd = c.log2spp & 1;
        uint32_t idx = 0;
#pragma unroll 1
        for (int shift = 2 * (c.n_base4_digits - 1) - odd; shift >= odd; shift -= 2) {
                uint32_t above = zs_shr32(morton, shift + 2);
                above ^= above >> 16;
                uint32_t x = (above ^ mixed) * 0x85ebca77u;
                x ^= x >> 13;
                x *= 0xc2b2ae35u;
                const uint32_t e = perm[x >> 24];
                idx = idx * 4u + ((e >> (((morton >> shift) & 3u) * 2u)) & 3u);
        }
        if (odd) idx = idx * 2u + ((morton ^ zs_mix_bits32((morton >> 1) ^ fold)) & 1u);
        return idx;
}

// sobolSample's matrix products of `dims` consecutive dimensions from base for
// a 32-bit index: one table entry per four index bits and dimension (table
// [dim][nibble][16], the xor of the matrix columns of the nibble's set bits),
// where scanning the index took one column per set bit in a loop as long as
// the warp's largest bit count.
template <int DIMS>
__device__ __forceinline__ void zs_sobol32(const ZSobolConfig &c, uint32_t index, int base, uint32_t (&acc)[DIMS]) {
        const uint32_t *t = c.nibbles + (size_t)base * kSobolNibbleWords;
#pragma unroll
        for (int k = 0; k < DIMS; ++k) acc[k] = 0u;
        const int bits = 2 * c.n_base4_digits - (c.log2spp & 1);
#pragma unroll 1
        for (int b = 0; b < bits; b += 4, t += 16) {
                const uint32_t v = (index >> b) & 15u;
#pragma unroll
                for (int k = 0; k < DIMS; ++k) acc[k] ^= __ldg(t + k * kSobolNibbleWords + v);
        }
}

// Owen scramble, times 2^-32, clamped below 1 (the tail of sobolSample).
__device__ __forceinline__ float zs_finish(uint32_t acc, uint32_t scramble) {
        const uint32_t r = zs_owen(acc, scramble);
        const float f = __fmul_rn(__uint2float_rn(r), 2.32830643653869628906e-10f);
        const float one_minus_eps = 1.0f - 1e-6f;
        return one_minus_eps < f ? one_minus_eps : f;
}

// getSampleHash (ZSobolSampler.swift:188-199); the second hash is 0 because
// mixBits returns 32 bits.
__device__ __forceinline__ uint32_t zs_hash(const ZSobolConfig &c, int dim) {
        return zs_mix_bits((uint64_t)(int64_t)dim ^ c.seed);
}

// The DIMS values of a draw whose 32-bit index is known, or (wide) of one
// whose index needs 64 bits.
template <int DIMS>
__device__ __forceinline__ void zs_values(const ZSobolConfig &c, const ZSobol &s, const ZSlot &slot, bool wide,
                                          uint32_t index, float (&out)[DIMS]) {
        uint32_t acc[DIMS];
        if (wide) {
                const uint64_t idx = zs_index64(c.log2spp, c.n_base4_digits, s.morton, slot.hash);
#pragma unroll 1
                for (int k = 0; k < DIMS; ++k) {
                        const uint32_t a = zs_sobol64(c.matrices + (size_t)(slot.base + k) * kSobolColumns, idx);
#pragma unroll
                        for (int j = 0; j < DIMS; ++j)
                                if (j == k) acc[j] = a;
                }
        } else {
                zs_sobol32<DIMS>(c, index, slot.base, acc);
        }
        out[0] = zs_finish(acc[0], zs_hash(c, slot.hash));
        if (DIMS > 1) out[DIMS > 1 ? 1 : 0] = zs_finish(acc[DIMS > 1 ? 1 : 0], 0u);
        if (DIMS > 2) out[DIMS > 2 ? 2 : 0] = zs_finish(acc[DIMS > 2 ? 2 : 0], zs_hash(c, slot.hash + 2));
}

// The first DIMS values of a draw.
template <int DIMS>
__device__ __forceinline__ void zs_draw(const ZSobolConfig &c, const ZSobol &s, const ZSlot &slot, float (&out)[DIMS]) {
        const bool wide = !zs_fits32(c, s);
        zs_values<DIMS>(c, s, slot, wide, wide ? 0u : zs_index32(c, (uint32_t)s.morton, slot.hash), out);
}

// startPixelSample (ZSobolSampler.swift:130-136).
__device__ __forceinline__ void zs_start(const ZSobolConfig &c, ZSobol &s, uint32_t px, uint32_t py, uint32_t index) {
        s.dim = 0;
        s.morton = (zs_morton2(px, py) << c.log2spp) | (uint64_t)index;
}

// get1D (ZSobolSampler.swift:203-219).
__device__ __forceinline__ float zs_get1d(const ZSobolConfig &c, ZSobol &s) {
        const ZSlot slot = zs_take(s, 1);
        float v[1];
        zs_draw<1>(c, s, slot, v);
        return v[0];
}

// get2D (ZSobolSampler.swift:221-244).
__device__ __forceinline__ void zs_get2d(const ZSobolConfig &c, ZSobol &s, float &a, float &b) {
        const ZSlot slot = zs_take(s, 2);
        float v[2];
        zs_draw<2>(c, s, slot, v);
        a = v[0];
        b = v[1];
}

// get3D (ZSobolSampler.swift:249-280).
__device__ __forceinline__ void zs_get3d(const ZSobolConfig &c, ZSobol &s, float &a, float &b, float &d) {
        const ZSlot slot = zs_take(s, 3);
        float v[3];
        zs_draw<3>(c, s, slot, v);
        a = v[0];
        b = v[1];
        d = v[2];
}

}  // namespace gzg
