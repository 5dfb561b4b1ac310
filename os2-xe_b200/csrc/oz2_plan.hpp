// oz2_plan.hpp - host planning for the Ozaki Scheme II path: modulus sets, the exact
// product M, the bits per scaled element tk, CRT weights, and the per-modulus constants the
// split, GEMM-epilogue and CRT kernels read.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define OZ2_HD __host__ __device__
#else
#define OZ2_HD
#endif

namespace oz2 {

constexpr int kMaxModuli = 24;     // the reference's range of s (Ozaki2::gemm / zgemm)
// The adaptive path (no counterpart in the reference) may go further, to s = 32, with moduli sets
// of its own: tiles whose certified error bound needs more than the 91 bits per element of 24
// moduli run emulated instead of in native FP64.
constexpr int kMaxModuliExt = 32;
constexpr int kBigWords = 8;       // 256-bit host integers
constexpr int kMaxLimbs = 8;       // 32-bit limbs of M for s <= 32
constexpr int kMaxScaleBits = 100;     // tk cap of the reference's plans (s <= 24)
constexpr int kMaxScaleBitsExt = 124;  // tk cap of the extended plans (s = 25..32)
constexpr int kNarrowScaleBits = 62;
// the split's wide offset (2^93 in three 32-bit words) holds |x| <= 2^92; every plan with
// s <= 24 has tk <= 91
constexpr int kWideScaleBits = 92;
// the widest offset (2^125 in four 32-bit words) holds |x| <= 2^124 (extended plans)
constexpr int kNonFinite = -2147483647 - 1;

// 32-bit limbs of M per s: max(2, floor(log2 M / 32) + 1) (ref src/ozaki2_gpu.hpp:55-59, :168)
// a = q b + r for the block and unit indices of a launch (below 2^31, which the host checks for
// every grid): 32-bit division, several times cheaper than the 64-bit one
OZ2_HD inline void divmod_index(int64_t a, int64_t b, int64_t& q, int64_t& r) {
    const uint32_t qq = static_cast<uint32_t>(a) / static_cast<uint32_t>(b);
    q = qq;
    r = a - static_cast<int64_t>(qq) * b;
}

OZ2_HD constexpr int limbs_for(int s) {
    constexpr int t[kMaxModuliExt + 1] = {0, 0, 2, 2, 2, 2, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 4,
                                          5, 5, 5, 5, 6, 6, 6, 6, 6, 7, 7, 7, 7, 8, 8, 8};
    return t[s];
}

// 16-bit limbs of M per s: floor(log2 M / 16) + 1
OZ2_HD constexpr int limbs16_for(int s) {
    constexpr int t[kMaxModuliExt + 1] = {0, 0, 1,  2,  2,  3,  3,  4,  4,  5,  5,  6,  6,  7,  7,  8, 8,
                                          9, 9, 10, 10, 11, 11, 12, 12, 12, 13, 13, 14, 14, 15, 15, 16};
    return t[s];
}

// Constants of one modulus as the kernels use them.
// GEMM sums of at most kExactKB k-blocks of 128 products of int8 residues are bounded by
// kExactSum = 511 * 128 * 128^2 < 2^30, so c + kbias30 < 2^31 and the epilogue's quotient is exact
constexpr int kExactKB = 511;
constexpr uint32_t kExactSum = 511u * 128u * 16384u;

struct ModConst {
    uint32_t m;      // modulus
    uint32_t mu;     // floor(2^32 / m), Barrett
    uint32_t kbias;  // m ceil(2^31 / m): c + kbias is in [0, 2^32) for every int32 GEMM sum c
                     // (|c| < 2^31 - 2^21) and congruent to c modulo m
    uint32_t kbias30;  // m ceil(kExactSum / m): c + kbias30 is in [0, 2^31) for every int32 GEMM sum
                       // c of at most kExactKB k-blocks (|c| <= kExactSum) and congruent to c
    uint32_t mx31;     // ceil(2^(32 + mxs) / m): floor(v / m) = umulhi(v, mx31) >> mxs exactly for v < 2^31
    uint32_t mxs;      // 7, or 6 for m < 128 (the moduli of the extended sets from s = 29), where
                       // ceil(2^39 / m) would not fit 32 bits
};

// Constants of one modulus as the split uses them, for the number of words of the plan's offset
// integers (split_words). The byte dot product v = start + sum_l byte_l (2^(8 l) mod m) of an offset
// integer x + 2^62 (2^93, 2^125) is the bit pattern of the float K m + v', with v' = off + sum_l ...
// congruent to x and K m the first multiple of m from 2^23 on; one FMA by finv and 1.5 2^23 then
// leaves K + rint(v' / m) in the low mantissa bits (oz2_split.cu: sym_residue).
struct alignas(16) SplitMod {
    uint32_t cb[4];  // bytes 2^(8 l) mod m, l = 0..15, four per word (byte-limb weights)
    uint32_t m;
    float finv;      // fl(1 / m)
    uint32_t start;  // 0x4B000000 + (K m - 2^23) + off
    uint32_t off;    // -2^62 (-2^93, -2^125) mod m
};
// 32-bit words of the offset integer of |x| <= 2^tk
OZ2_HD constexpr int split_words(int tk) { return tk <= kNarrowScaleBits ? 2 : (tk <= kWideScaleBits ? 3 : 4); }

struct Plan {
    int s = 0;
    int nl = 0;
    int tk = 0;
    double log2M = 0;
    uint32_t m[kMaxModuliExt] = {};
    uint32_t y[kMaxModuliExt] = {};             // (M/m_t)^-1 mod m_t
    uint32_t W[kMaxModuliExt][kBigWords] = {};  // CRT weights (M/m_t) y_t
    uint32_t M[kBigWords] = {};
    ModConst mc[kMaxModuliExt] = {};            // the GEMM's per-modulus constants (mod_constants)
    SplitMod sm[kMaxModuliExt] = {};            // the split's (split_constants, for the words of this tk)
};

// Returns 0, or 1 (invalid: s out of [2, 24], k < 1, s too small for k), or 5 (overflow).
// ref src/ozaki2_gpu.hpp:159-200
int make_plan(int s, int64_t k, Plan& p);
// Whether the GEMM reduces this plan's sums over kb k-blocks in FP32, to signed residues (otherwise
// in integers, to residues in [0, m)). |c| <= 128 * 128^2 kb must be exact in FP32: 8 k-blocks; m = 255, whose
// signed residue must not reach +128, stays exact up to 4. B200, 4096^2, s = 16: the GEMM stage 196 ->
// 159 us at k = 256, 163 -> 149 at 512, 224 -> 218 at 1024.
bool f32_residues(const Plan& p, int64_t kb);
// the same for s in [2, 32]: the reference's plans for s <= 24, the extended sets above
int make_plan_ext(int s, int64_t k, Plan& p);
// tk of make_plan_ext(s, k), or 0 where that plan is invalid (s too small for k)
int plan_tk(int s, int64_t k);
const char* plan_error_text(int s, int64_t k, int status, char* buf, int len);

void mod_constants(const Plan& p, ModConst* out);
// for offset integers of `words` 32-bit words (split_words)
void split_constants(const Plan& p, int words, SplitMod* out);

// CRT table: Sum_t r_t W_t - q M on 16-bit limbs, q from the sum's top two limbs in FP32 (the
// reference estimates q from the residues in FP32, src/ozaki2_gpu.hpp:526-588)
constexpr int kQuads = (kMaxModuliExt + 3) / 4;  // moduli in groups of four (one residue byte each)
constexpr int kLimbs16 = 2 * kMaxLimbs;

struct CrtConst {
    // W_t = (M / m_t) y_t in 16-bit limbs, paired for two-way byte dot products: for the moduli
    // 4g..4g+3 and limb l, Wq[g][l][0] = W16[4g][l] | W16[4g+1][l] << 16 and Wq[g][l][1] the same
    // for 4g+2, 4g+3 (zero past s)
    uint32_t Wq[kQuads][kLimbs16][2];
    uint32_t M16[kLimbs16];  // limbs of M
    float qf[kLimbs16];      // 2^(16 l) / M (zero where it underflows)
};
void crt_constants(const Plan& p, CrtConst& out);

}  // namespace oz2
