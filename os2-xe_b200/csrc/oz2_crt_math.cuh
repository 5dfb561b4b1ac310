// oz2_crt_math.cuh - the exact CRT reconstruction of one C entry, shared by the CRT kernels
// (oz2_crt.cu) and the GEMM whose epilogue runs the CRT for small s (oz2_gemm.cu).
//
// x = Sum_t r_t W_t - q M with q the nearest integer to Sum_t r_t W_t / M (|x| <= M/4), rounded once
// to double. Everything runs on 16-bit limbs: a_l = Sum_t r_t W_t[l] (|r_t| <= 255, so
// below 32 * 255 * 2^16 < 2^29), then
//   q      from the top two limbs of the sum in FP32: the limbs below add at most 0.05 to Sum / M
//          (0.03 for complex operands' combined sums; the plan's build checks both), so the estimate errs by less than 1/4;
//   limbs  c_l = a_l - q M_l + (c_{l-1} >> 16), one multiply-add and one shifted add each: the low 16
//          bits of c_0 .. c_{L-2} and all of c_{L-1} are x in two's complement;
//   RNE    the three top 32-bit words h, m, l as doubles (l with a sticky bit for the words below):
//          h 2^32 + m rounds with an exact error term, and the last FMA rounds the exact sum once,
//          signed numbers included. A top word that only repeats the sign is folded into the next.
// The FP64 pipe takes over the sign, normalisation and rounding, which cost about 100 integer
// instructions per entry as 64-bit words.
#pragma once

#include <cstdint>

#include "oz2_plan.hpp"

namespace oz2 {

__device__ __forceinline__ int exponent_of(unsigned long long b, int tk) {
    if (b >= 0x7FF0000000000000ull) return kNonFinite;
    if (b == 0) return 0;
    const int be = static_cast<int>(b >> 52);
    const int e2 = be ? be - 1022 : -1010 - __clzll(static_cast<long long>(b));
    return tk - e2;
}

// The exponent for the unscaling, with kFarExponent for a non-finite row or column: a sum of two
// exponents (each within +-1200) at or above kFarExponent / 2 then means NaN.
constexpr int kFarExponent = 1 << 20;
__device__ __forceinline__ int unscale_exponent(unsigned long long b, int tk) {
    const int e = exponent_of(b, tk);
    return e == kNonFinite ? kFarExponent : e;
}

// 32-bit words as doubles (exact)
__device__ __forceinline__ double u32_double(uint32_t w) {
    return __hiloint2double(0x43300000, static_cast<int>(w)) - 4503599627370496.0;  // 2^52
}
__device__ __forceinline__ double i32_double(int32_t w) {
    return __hiloint2double(0x43300000, static_cast<int>(static_cast<uint32_t>(w) ^ 0x80000000u)) - 4503601774854144.0;  // 2^52 + 2^31
}

// Limb l of the sums of EG entries: R[e][g] holds the residues (any byte congruent to r_t) of the
// moduli 4g..4g+3 as bytes (zero past s); every weight word is read once for all entries.
template <int Q, int EG>
__device__ __forceinline__ void crt_limb(const uint32_t (&R)[EG][Q], const CrtConst& cc, int l, uint32_t (&a)[EG]) {
#pragma unroll
    for (int e = 0; e < EG; ++e) a[e] = 0;
#pragma unroll
    for (int g = 0; g < Q; ++g) {
        const uint32_t w0 = cc.Wq[g][l][0], w1 = cc.Wq[g][l][1];
#pragma unroll
        for (int e = 0; e < EG; ++e) a[e] = __dp2a_hi(w1, R[e][g], __dp2a_lo(w0, R[e][g], a[e]));
    }
}

// The 32-bit words of EG entries' x from the top: word k is the limbs L - 2 - 2k and L - 1 - 2k.
// sum(l, a) gives limb l of the EG sums (signed for SIGNED); the top two come first, for the
// quotient (the nearest integer to their part of the sum over M), the others as they are used.
template <int L, int EG, bool SIGNED, class Sum>
__device__ __forceinline__ void crt_words(Sum sum, const uint32_t* M16, const float* qf, uint32_t (&w)[EG][(L + 1) / 2]) {
    uint32_t a1[EG], a0[EG], q[EG], c[EG];
    sum(L - 1, a1);
    if (L > 1) sum(L > 1 ? L - 2 : 0, a0);
#pragma unroll
    for (int e = 0; e < EG; ++e) {
        auto f = [](uint32_t v) { return SIGNED ? __int2float_rn(static_cast<int>(v)) : __uint2float_rn(v); };
        float x = f(a1[e]) * qf[L - 1];
        if (L > 1) x = __fmaf_rn(f(a0[e]), qf[L > 1 ? L - 2 : 0], x);
        q[e] = __float_as_uint(__fadd_rn(x, 12582912.0f)) - 0x4B400000u;  // + 1.5 2^23
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
        uint32_t a[EG];
        if (l < L - 2) sum(l, a);
#pragma unroll
        for (int e = 0; e < EG; ++e) {
            const uint32_t b = (l < L - 2 ? a[e] : (l == L - 2 ? a0[e] : a1[e])) - q[e] * M16[l];
            const uint32_t prev = l ? c[e] : 0u;
            c[e] = static_cast<uint32_t>(__dp2a_lo(static_cast<int>(prev), 0x100, static_cast<int>(b)));  // b + (prev >> 16)
            if ((L - 1 - l) % 2 == 0) w[e][(L - 1 - l) / 2] = __byte_perm(prev, c[e], 0x5410);
        }
    }
}

// x 2^-shift from x's words, rounded once (twice only into the subnormal range, as ldexp of the
// rounded value); NaN when shift marks a non-finite row or column
template <int L>
__device__ __forceinline__ double crt_round(const uint32_t (&w)[(L + 1) / 2], int shift) {
    constexpr int NW = (L + 1) / 2;
    auto word = [&](int k) { return k < NW ? w[k < NW ? k : 0] : 0u; };
    auto low = [&](int k) {  // word k with a sticky bit for the words below it
        uint32_t rest = 0;
#pragma unroll
        for (int i = 0; i < NW; ++i) rest |= i > k ? w[i] : 0u;
        return word(k) | (rest != 0 ? 1u : 0u);
    };
    double dt = i32_double(static_cast<int32_t>(w[0]));
    uint32_t m = word(1), l = low(2);
    int E = 16 * L - 96 - shift;
    if (w[0] + 1u <= 1u) {  // h is 0 or -1: x is small beside M
        if constexpr (NW > 1) {
            // past the words that only repeat the sign, by selects, as lanes differ in how many they have (a branch and
            // a double per word before: 6144^2 wide entries, s = 20, 560 -> 537 us; 4096^2, s = 24, 236 -> 227)
            uint32_t v[NW];
#pragma unroll
            for (int i = 0; i < NW; ++i) v[i] = word(i + 1);
            E -= 32;
#pragma unroll
            for (int k = 2; k < NW; ++k) {
                const bool skip = v[0] == w[0];
#pragma unroll
                for (int i = 0; i + 1 < NW; ++i) v[i] = skip ? v[i + 1] : v[i];
                E -= skip ? 32 : 0;
            }
            uint32_t rest = 0;
#pragma unroll
            for (int i = 3; i < NW; ++i) rest |= v[i];
            dt = __fma_rn(dt, 4294967296.0, u32_double(v[0]));
            m = v[1];
            l = (NW > 2 ? v[NW > 2 ? 2 : 0] : 0u) | (rest != 0 ? 1u : 0u);
        }
        if (dt == 0.0) return shift >= kFarExponent / 2 ? __longlong_as_double(0x7FF8000000000000ll) : 0.0;
    }
    // |dt| 2^32 > m, so the first sum's error is exact; (e 2^32 + l) is below 2^45 and exact; the
    // sticky bit lies below half an ulp of the result, which is at least 2^64
    const double s = __fma_rn(dt, 4294967296.0, u32_double(m));
    const double e = u32_double(m) - __fma_rn(dt, -4294967296.0, s);
    const double r = __fma_rn(s, 4294967296.0, __fma_rn(e, 4294967296.0, u32_double(l)));
    // 2^64 <= |r| <= 2^98
    if (static_cast<uint32_t>(E + 1086) <= 1086u + 924u)
        return __hiloint2double(__double2hiint(r) + (E << 20), __double2loint(r));
    if (shift >= kFarExponent / 2) return __longlong_as_double(0x7FF8000000000000ll);
    return ldexp(r, E);
}

// 4 x 4 byte transpose: word t of `in` holds entries e = 0..3 of modulus 4g + t; word e of `out`
// holds moduli 4g..4g+3 of entry e
__device__ __forceinline__ void transpose4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&out)[4]) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
    const uint32_t t2 = __byte_perm(c, d, 0x5140), t3 = __byte_perm(c, d, 0x7362);
    out[0] = __byte_perm(t0, t2, 0x5410);
    out[1] = __byte_perm(t0, t2, 0x7632);
    out[2] = __byte_perm(t1, t3, 0x5410);
    out[3] = __byte_perm(t1, t3, 0x7632);
}

}  // namespace oz2
