// oz2_split.cu - scale and split phases of the Ozaki-II path.
//
// scale: max |x| per plane row as raw FP64 bits (ref src/ozaki2_gpu.hpp:309-358); the bit
//        pattern of a non-negative double orders like the value, and Inf/NaN land above
//        0x7FF0000000000000 so one integer max also detects non-finite rows.
// split: for every element x of plane row r, the integer RNE(x * 2^e_r) with
//        e_r = tk - frexp_exp(max_r) (ref :360-377, :251-289) and its symmetric residue
//        modulo each m_t in [-h_t, m_t-1-h_t] (ref :407-455, complex 3M form :457-520),
//        stored as int8 in the pre-tiled plane layout of oz2_kernels.cuh.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "oz2_kernels.cuh"
#include "oz2_ptx.cuh"

namespace oz2 {
namespace {

constexpr uint64_t kAbsMask = 0x7FFFFFFFFFFFFFFFull;

__device__ __forceinline__ int exponent_of(unsigned long long b, int tk) {
    if (b >= 0x7FF0000000000000ull) return kNonFinite;
    if (b == 0) return 0;
    const int be = static_cast<int>(b >> 52);
    const int e2 = be ? be - 1022 : -1010 - __clzll(static_cast<long long>(b));  // frexp exponent
    return tk - e2;
}

// ------------------------------------------------------------------ item lookup
// index of the item whose [block0, next block0) range holds `b` (items sorted by block0)
template <class Item>
__device__ __forceinline__ int find_item(const Item* items, int count, int64_t b) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].block0 <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ------------------------------------------------------------------ scale
// ROWC: plane rows contiguous in memory, one thread per row and a k range per block.
// Otherwise: inner index contiguous, one warp per row and a k range per block.
// The layout is the item's, so both operands share one launch.
template <bool CPLX>
__global__ void __launch_bounds__(256) scale_kernel(const ScaleItem* items, int count) {
    dev::chain_wait();
    dev::chain_next();
    const ScaleItem* I = items + find_item(items, count, blockIdx.x);
    const int64_t local = static_cast<int64_t>(blockIdx.x) - I->block0;
    int64_t rb, kc;
    divmod_index(local, I->rblocks, kc, rb);
    const unsigned long long* X = reinterpret_cast<const unsigned long long*>(I->X);
    const int64_t rows = I->rows, k = I->k, ldx = I->ldx, kchunk = I->kchunk;
    if (I->row_contig) {
        // 32 consecutive rows per block (one per lane); the 8 warps interleave the k range
        const int64_t r = rb * 32 + (threadIdx.x & 31);
        if (r >= rows) return;
        const int64_t p0 = kc * kchunk, p1 = min(k, p0 + kchunk);
        unsigned long long best = 0;
        for (int64_t p = p0 + (threadIdx.x >> 5); p < p1; p += 8) {
            const int64_t idx = r + p * ldx;
            if (CPLX) {
                best = max(best, __ldg(X + 2 * idx) & kAbsMask);
                best = max(best, __ldg(X + 2 * idx + 1) & kAbsMask);
            } else {
                best = max(best, __ldg(X + idx) & kAbsMask);
            }
        }
        if (best) atomicMax(I->out + r, best);
    } else {
        const int64_t r = rb * 8 + (threadIdx.x >> 5);
        const int lane = threadIdx.x & 31;
        if (r >= rows) return;
        const int w = CPLX ? 2 : 1;
        const int64_t p0 = kc * kchunk * w, p1 = min(k * w, p0 + kchunk * w);
        const unsigned long long* row = X + r * ldx * w;
        unsigned long long best = 0;
        for (int64_t p = p0 + lane; p < p1; p += 32) best = max(best, __ldg(row + p) & kAbsMask);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, o));
        if (lane == 0 && best) atomicMax(I->out + r, best);
    }
}

// The same maxima as the first launch of a small product: the descriptors come as the kernel's parameter, the last
// block writes them for the kernels that follow, and a block owns 32 whole rows (rows contiguous: a lane per row, 32
// warps interleave k; otherwise a warp per row), so its stores need no zeroed maxima. For k <= kScaleFirstMaxK, where
// a thread reads at most 16 entries, eight in flight: 256^3 24.0 -> 20.4 us per call back to back, 1024 x 1024 x 512
// 41.2 -> 37.3; at k = 1024 the few blocks take longer than the launch saved (1024^3 57 -> 64 us), splitting k wins.
template <int N, bool CPLX>
__global__ void __launch_bounds__(1024) scale_first_kernel(const __grid_constant__ BlobParam<N> b, unsigned char* dst,
                                                           uint32_t off, int count) {
    __shared__ unsigned long long part[32][33];
    dev::chain_next();
    if (blockIdx.x == gridDim.x - 1) {
        for (uint32_t i = threadIdx.x * 16; i < b.bytes; i += 1024 * 16)
            *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(b.data + i);
        return;
    }
    const ScaleItem* items = reinterpret_cast<const ScaleItem*>(b.data + off);
    const ScaleItem* I = items + find_item(items, count, blockIdx.x);
    const int64_t r0 = (static_cast<int64_t>(blockIdx.x) - I->block0) * 32;
    const int warp = static_cast<int>(threadIdx.x >> 5), lane = static_cast<int>(threadIdx.x & 31);
    constexpr int W = CPLX ? 2 : 1;
    const unsigned long long* X = reinterpret_cast<const unsigned long long*>(I->X);
    const int k = static_cast<int>(I->k);
    unsigned long long best = 0;
    if (I->row_contig) {
        const int64_t r = r0 + lane, ldx = I->ldx;
        if (r < I->rows) {
#pragma unroll 8
            for (int p = warp; p < k; p += 32) {
                const unsigned long long* x = X + W * (r + p * ldx);
                best = max(best, __ldg(x) & kAbsMask);
                if (CPLX) best = max(best, __ldg(x + 1) & kAbsMask);
            }
        }
        part[lane][warp] = best;
        __syncthreads();
        best = part[warp][lane];
    } else if (r0 + warp < I->rows) {
        const unsigned long long* x = X + W * (r0 + warp) * I->ldx;
#pragma unroll 8
        for (int p = lane; p < W * k; p += 32) best = max(best, __ldg(x + p) & kAbsMask);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, o));
    if (lane == 0 && r0 + warp < I->rows) I->out[r0 + warp] = best;
}

template <int N>
void scale_first_n(const void* blob, size_t bytes, unsigned char* dst, uint32_t off, int count, unsigned grid, bool cplx,
                   cudaStream_t st) {
    static thread_local BlobParam<N> bp;
    std::memcpy(bp.data, blob, bytes);
    bp.bytes = static_cast<uint32_t>((bytes + 15) & ~size_t{15});
    if (cplx) scale_first_kernel<N, true><<<grid, 1024, 0, st>>>(bp, dst, off, count);
    else scale_first_kernel<N, false><<<grid, 1024, 0, st>>>(bp, dst, off, count);
}

// ------------------------------------------------------------------ split
// 2^k as a double for k in [-1022, 1023]
__device__ __forceinline__ double pow2(int k) {
    return __longlong_as_double(static_cast<long long>(k + 1023) << 52);
}

// x = RNE(v 2^e) as the reference derives it from the double's bits (src/ozaki2_gpu.hpp:251-289),
// computed in floating point: y = v 2^e as two exact power-of-two products (e = e1 + e2 keeps
// both factors normal for every e the split sees; a product that underflows means
// |y| < 2^-1022, which rounds to 0 like the exact value), then one round-to-nearest-even
// conversion. The offset integer 2^62 + x (narrow path, tk <= 62: x fits int64) as two 32-bit
// words.
__device__ __forceinline__ void offset_words_fp(double y, uint32_t (&W)[2]) {
    const long long x = __double2ll_rn(y);
    const uint64_t xo = static_cast<uint64_t>(x + (1ll << 62));
    W[0] = static_cast<uint32_t>(xo);
    W[1] = static_cast<uint32_t>(xo >> 32);
}

// Wide path (62 < tk <= 92; the largest tk of any plan is 91): y = v 2^e as above, a = |rint(y)|
// <= 2^92 split exactly into hi = trunc(a 2^-64) and lo = a - hi 2^64 (both exact: power-of-two
// scaling, and lo keeps a subset of a's 53 significant bits), then 2^93 +- (hi:lo), which lies in
// (0, 2^94), as three 32-bit words.
__device__ __forceinline__ void offset_words_fp_wide(double y0, uint32_t (&W)[3]) {
    const double y = rint(y0);
    const double a = fabs(y);
    const double hd = trunc(a * 5.421010862427522e-20);     // 2^-64
    const double ld = fma(hd, -18446744073709551616.0, a);  // a - hd 2^64, exact
    const uint64_t hi = __double2ull_rz(hd), lo = __double2ull_rz(ld);
    uint64_t ol, oh;
    if (y < 0.0) {
        ol = 0 - lo;
        oh = (1ull << 29) - hi - (lo != 0 ? 1 : 0);
    } else {
        ol = lo;
        oh = (1ull << 29) + hi;
    }
    W[0] = static_cast<uint32_t>(ol);
    W[1] = static_cast<uint32_t>(ol >> 32);
    W[2] = static_cast<uint32_t>(oh);
}

// Widest path (92 < tk <= 124, the extended moduli sets of the adaptive path): as the wide path
// with a = |rint(y)| <= 2^124, hi = trunc(a 2^-64) < 2^60, and the offset 2^125 +- (hi:lo), which
// lies in (0, 2^126), as four 32-bit words.
__device__ __forceinline__ void offset_words_fp_widest(double y0, uint32_t (&W)[4]) {
    const double y = rint(y0);
    const double a = fabs(y);
    const double hd = trunc(a * 5.421010862427522e-20);     // 2^-64
    const double ld = fma(hd, -18446744073709551616.0, a);  // a - hd 2^64, exact
    const uint64_t hi = __double2ull_rz(hd), lo = __double2ull_rz(ld);
    uint64_t ol, oh;
    if (y < 0.0) {
        ol = 0 - lo;
        oh = (1ull << 61) - hi - (lo != 0 ? 1 : 0);
    } else {
        ol = lo;
        oh = (1ull << 61) + hi;
    }
    W[0] = static_cast<uint32_t>(ol);
    W[1] = static_cast<uint32_t>(ol >> 32);
    W[2] = static_cast<uint32_t>(oh);
    W[3] = static_cast<uint32_t>(oh >> 32);
}

// The symmetric residue v' - q m, q = rint(v' / m), in the low byte of the result (the upper bytes
// hold anything), from the bits v of the float K m + v' (SplitMod). One FMA gives 1.5 2^23 + K + q
// with a single rounding to an integer (ulp 1): the product errs by (K m + v') |fl(1/m) - 1/m| <
// 0.63 / m, against a distance of at least 1 / (2 m) of v' / m from a half-integer (m odd), so q is
// the nearest integer or, next to a tie, its neighbour: |residue| <= (m + 1) / 2 <= 127 for m <=
// 253; fl(1/255) > 1/255, so m = 255 errs only upwards, to -128. Either way the byte is
// congruent to x, which is all the INT8 products need (m = 256: any q gives the low byte of v').
// v - bits m is v' - q m modulo 256: 0x4B000000, 2^22 and K m - K m are. Two instructions per residue.
__device__ __forceinline__ uint32_t sym_residue(uint32_t v, float finv, uint32_t mneg) {
    uint32_t r;  // in one piece: left to itself the compiler narrows the arithmetic to the byte it sees
                 // used, which costs an instruction more per residue
    asm("{\n\t.reg .f32 x, y;\n\t.reg .b32 t;\n\t"
        "mov.b32 x, %1;\n\t"
        "fma.rn.f32 y, x, %2, 0f4B400000;\n\t"  // + 1.5 2^23
        "mov.b32 t, y;\n\t"
        "mad.lo.u32 %0, t, %3, %1;\n\t}"
        : "=r"(r)
        : "r"(v), "f"(finv), "r"(mneg));
    return r;
}

// low bytes of a, b, c, d as one little-endian word
__device__ __forceinline__ uint32_t pack_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// D = C + A B: 16 x 32 by 32 x 8 unsigned bytes, int32 sums
__device__ __forceinline__ void mma_u8(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                                       const uint4& c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%10, %11, %12, %13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w));
}
__device__ __forceinline__ void mma_u8_add(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int NW>
__device__ __forceinline__ void offset_words(double y, uint32_t (&W)[NW]) {
    if constexpr (NW == 2) offset_words_fp(y, W);
    else if constexpr (NW == 3) offset_words_fp_wide(y, W);
    else offset_words_fp_widest(y, W);
}

// The split's byte dot products run as mma.sync u8 x u8 -> s32 with the weights in A and the
// offset integers in B, in a shape where no element leaves the lane that holds it: lane 4 n + q
// gives column n of B the words of its own element in K positions q (bytes 4 q .. and 16 + 4 q ..),
// and row (modulus t, q) of A (t < 4) holds modulus t's weights in K positions q and zeros
// elsewhere, so entry ((t, q), n) of the product is the dot product of lane 4 n + q's element with
// modulus t. One instruction gives 32 elements' residues for four moduli (two words; a second
// instruction adds words 2 and 3), and lane (g, c) = (lane / 4, lane % 4) receives, for modulus
// g % 4, those of the four lanes 4 n + q with n / 2 = c and q % 2 = g / 4. Every lane holds four
// elements (j = 0..3) of a plane row's 128, lane 4 n + q the inner indices 16 ch + 4 j + sub with ch =
// 2 (n / 2) + q % 2 and sub = n % 2 + 2 (q / 2): the sixteen residues that a lane receives from four
// instructions are then the 16 bytes of one chunk of one plane, and a warp stores whole 128-byte
// plane rows of four planes.
//
// Bound: instruction issue, then DRAM. A residue costs one FMA, one multiply-add, 3/4 of a byte
// permute and 1/128 mma per lane (8.6 cycles of the scheduler per mma, measured) where dp4a took
// two to four quarter-of-the-lanes dot products and a two-step quotient. The operand comes through
// cp.async double buffering (rows contiguous: whole lines, transposed on the way out of shared
// memory). Two blocks per SM of up to 128 registers on the narrow and complex paths (three or four, with
// spilled or serialised accumulators, measured slower), three of 80 on the wider ones, which spill 24 (three
// words) and 72 bytes (four): against two blocks without spills 582 and 601 us at 6144^3 s = 20, 1574 and 1624
// on 512 grouped problems, 269 and 275 at 4096^3 s = 24, but 149 and 130 at 4096^2 x 2048 s = 20 and 2.93
// and 2.80 ms on 64 adaptive problems. Stage times, start -> now, alternating in one process: 8192^3 s = 16 1044 -> 682 us (498 us of DRAM time at the
// measured copy rate), 6144^3 s = 20 (three words) 849 -> 575, 1024^2 x 262144 s = 16 3790 -> 2490,
// ZGEMM 4096^3 s = 16 781 -> 424.
constexpr int kSplitThreads = 256;
constexpr int kSplitTileBytes = 16384;  // the operand's elements of one block tile
// rows of a block tile (two per warp, one for complex operands), by 128 inner indices
template <bool CPLX>
__host__ __device__ constexpr int split_rows() { return CPLX ? 8 : 16; }

// Shared memory of a block: two operand tiles, and the plan's constants per group of four moduli:
// every lane's A fragments, the accumulators an mma starts from, and {-m, 1 / m, start - off} of the
// lane's modulus (a group past s repeats modulus 0 and stores nothing).
template <int NW>
struct SplitShared {
    alignas(128) unsigned char tile[2][kSplitTileBytes];
    uint4 a[kMaxModuliExt / 4][NW > 2 ? 2 : 1][32];
    uint4 start[kMaxModuliExt / 4][4];
    uint4 c[kMaxModuliExt / 4][4];
};
template <int NW>
__device__ __forceinline__ void split_consts(const SplitItem* I, SplitShared<NW>& S) {
    const int lane = static_cast<int>(threadIdx.x & 31), g = lane >> 2, c = lane & 3, nmod = I->s;
    for (int grp = static_cast<int>(threadIdx.x >> 5); 4 * grp < nmod; grp += kSplitThreads / 32) {
        const int t = 4 * grp + (g & 3);
        const SplitMod& sm = I->mc[t < nmod ? t : 0];
        const uint32_t m0 = c == (g >> 2) ? 0xFFFFFFFFu : 0u, m1 = c == 2 + (g >> 2) ? 0xFFFFFFFFu : 0u;
        S.a[grp][0][lane] = make_uint4(sm.cb[0] & m0, sm.cb[0] & m1, sm.cb[1] & m0, sm.cb[1] & m1);
        if constexpr (NW > 2) S.a[grp][1][lane] = make_uint4(sm.cb[2] & m0, sm.cb[2] & m1, sm.cb[3] & m0, sm.cb[3] & m1);
        if (lane < 16 && c == 0) {
            S.start[grp][g] = make_uint4(sm.start, sm.start, sm.start, sm.start);
            S.c[grp][g] = make_uint4(0u - sm.m, __float_as_uint(sm.finv), sm.start - sm.off, 0u);
        }
    }
}

// asynchronous copy of `bytes` (0: zeros) of 8 / 16 bytes to shared memory
__device__ __forceinline__ void copy8(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Where element (row r, inner index k) of a tile lies in shared memory, in elements. k contiguous:
// [r][128]; rows contiguous: [k][rows]. The exclusive-or spreads the elements that the lanes of a
// warp read together (inner indices 16 ch + 4 j + sub of one row, ch and sub by lane) over all banks
// and keeps pairs of neighbours together.
template <bool CPLX, bool ROWC>
__device__ __forceinline__ int split_slot(int r, int k) {
    if (ROWC) return k * split_rows<CPLX>() + (r ^ ((k & 3) | ((k >> 2) & (CPLX ? 4 : 12))));
    return r * kTileK + (k ^ ((k >> 2) & (CPLX ? 4 : 12)));
}

// A thread's share of the copies of the block's tiles. k contiguous: warp w copies its own rows;
// rows contiguous: the block copies whole lines. Tiles inside the operand take fixed strides from
// one source and one shared-memory address; edge tiles check every element and read zeros outside.
template <bool CPLX, bool ROWC>
struct SplitFetch {
    static constexpr int RB = split_rows<CPLX>(), E = CPLX ? 16 : 8;  // rows, bytes per element
    static constexpr int R = RB / 8;
    const char* src;  // of this thread's first element in the next tile
    uint32_t dst;     // its shared-memory address in tile 0
    int64_t step;     // source bytes between the thread's rows (k contiguous) or inner indices

    __device__ __forceinline__ SplitFetch(const SplitItem* I, uint32_t tile0, int64_t r0, int kb0) {
        const int tid = static_cast<int>(threadIdx.x), lane = tid & 31;
        const int64_t ldx = I->ldx, k0 = static_cast<int64_t>(kb0) * kTileK;
        int r, p;
        if (ROWC) {
            r = tid % RB, p = tid / RB;
            step = ldx * (E * (kSplitThreads / RB));
        } else {
            r = R * (tid >> 5), p = lane * (I->vec ? 16 / E : 1);
            step = ldx * E;
        }
        src = reinterpret_cast<const char*>(I->X) + (ROWC ? r0 + r + (k0 + p) * ldx : (r0 + r) * ldx + k0 + p) * E;
        dst = tile0 + split_slot<CPLX, ROWC>(r, p) * E;
    }

    __device__ __forceinline__ void fast(uint32_t buf, bool vec) const {
        const uint32_t d = dst + buf;
        if (ROWC) {
            const char* x = src;
#pragma unroll
            for (int i = 0; i < kTileK * RB / kSplitThreads; ++i, x += step) {
                if (CPLX) {  // inner indices 32 apart: the same place in the swizzle
                    const uint32_t to = d + i * (32 * RB * E);
                    if (vec) {
                        copy16(to, x, 16);
                    } else {
                        copy8(to, x, 8);
                        copy8(to + 8, x + 8, 8);
                    }
                } else {  // inner indices 16 apart: swizzle bits 2, 3 of the row count them
                    copy8((d ^ ((i & 3) << 5)) + i * (16 * RB * E), x, 8);
                }
            }
        } else if (vec) {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const char* x = u ? src + step : src;
#pragma unroll
                for (int i = 0; i < kTileK * E / 512; ++i) copy16(d + u * (kTileK * E) + 512 * i, x + 512 * i, 16);
            }
        } else {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const char* x = u ? src + step : src;
#pragma unroll
                for (int i = 0; i < kTileK / 32; ++i) {
                    if (CPLX) {
                        copy8(d + 32 * E * i, x + 32 * E * i, 8);
                        copy8(d + 32 * E * i + 8, x + 32 * E * i + 8, 8);
                    } else {  // inner indices 32 apart: swizzle bit 3 alternates
                        copy8((d ^ ((i & 1) << 6)) + u * (kTileK * E) + 32 * E * i, x + 32 * E * i, 8);
                    }
                }
            }
        }
    }

    // the tile at k0, with every access checked
    __device__ __noinline__ static void edge(const SplitItem* I, uint32_t tile, int64_t r0, int k0) {
        const int64_t rows = I->rows - r0, ldx = I->ldx;
        const int k = static_cast<int>(I->k) - k0;
        const char* X = reinterpret_cast<const char*>(I->X);
        for (int f = static_cast<int>(threadIdx.x); f < kTileK * RB; f += kSplitThreads) {
            // k contiguous: warp w takes its rows' elements, so that it alone waits for them
            const int r = ROWC ? f % RB : R * static_cast<int>(threadIdx.x >> 5) + (f / kSplitThreads) * 32 / kTileK;
            const int q = ROWC ? f / RB : (f / kSplitThreads * 32 + static_cast<int>(threadIdx.x & 31)) % kTileK;
            const bool in = r < rows && q < k;
            const char* x = in ? X + (ROWC ? r0 + r + (k0 + q) * ldx : (r0 + r) * ldx + k0 + q) * E : X;
            const uint32_t to = tile + split_slot<CPLX, ROWC>(r, q) * E;
            copy8(to, x, in ? 8 : 0);
            if (CPLX) copy8(to + 8, x + 8, in ? 8 : 0);
        }
    }
};

// The block's rows r0 .. r0 + split_rows - 1 at the k blocks kb0 .. kb1 - 1: residues of the rows
// below I->rows (the GEMM never uses a padding row's products) and of all inner indices (zero past
// k). mx[r - mbase]: the rows' maximum bits. The next tile's copies run under this one's work.
template <int NW, bool CPLX, bool ROWC>
__device__ __forceinline__ void split_tiles(const SplitItem* I, SplitShared<NW>& S, int64_t r0, int kb0,
                                            int kb1, const unsigned long long* mx, int64_t mbase) {
    constexpr int R = split_rows<CPLX>() / 8, NG = CPLX ? 2 : 1, NP = CPLX ? 3 : 1, E = CPLX ? 16 : 8;
    const int lane = static_cast<int>(threadIdx.x & 31), w8 = static_cast<int>(threadIdx.x >> 5);
    const uint32_t tile0 = dev::smem_addr(S.tile[0]);
    SplitFetch<CPLX, ROWC> F(I, tile0, r0, kb0);
    const int64_t adv = ROWC ? I->ldx * (E * kTileK) : E * kTileK;
    const bool vec = I->vec;
    const int kfull = r0 + split_rows<CPLX>() <= I->rows ? static_cast<int>(I->k / kTileK) : 0;  // k blocks without edges
    auto fetch = [&](int kb, uint32_t buf) {
        if (kb < kfull) F.fast(buf, vec);
        else SplitFetch<CPLX, ROWC>::edge(I, tile0 + buf, r0, kb * kTileK);
        F.src += adv;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(kb0, 0);
    const int n = lane >> 2, q = lane & 3;
    const int ch = 2 * (n >> 1) + (q & 1), sub = (n & 1) + 2 * (q >> 1);  // as a source of elements
    const int64_t rw = r0 + R * w8;                                       // the warp's first row
    const int64_t left = I->rows - rw;
    const int nrows = left < R ? static_cast<int>(left) : R;
    // scaling: 2^e in one exact factor; rows far up or down the exponent range take a second one,
    // and a non-finite row's residues are zero (both rare, and the same for the whole warp)
    double s1[R];
    uint32_t odd = 0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int e = u < nrows ? exponent_of(mx[rw + u - mbase], I->tk) : 0;
        const int e1 = max(-1000, min(1000, e));
        s1[u] = pow2(e == kNonFinite ? 0 : e1);
        if (e != e1) odd |= 1u << u;
    }
    const double im_sign = CPLX && I->conj ? -1.0 : 1.0;  // residues of -y are the negated residues of y
    const unsigned char* tiles = reinterpret_cast<const unsigned char*>(&S.tile);
    // byte in a tile of the lane's element j = 0 of the warp's first row
    const uint32_t el0 = split_slot<CPLX, ROWC>(R * w8, 16 * ch + sub) * E;
    // as a receiver: modulus g % 4 of each group of four, 16-byte chunk 2 c + g / 4 of the row
    const int g = n, c = q, tl = g & 3, nmod = I->s;
    const int64_t plane_bytes = I->plane_bytes, gstride = nmod * plane_bytes, tstep = 4 * plane_bytes;
    const int rr = static_cast<int>(rw & 127), place = (2 * c + (g >> 2)) ^ (rr & 7);
    int8_t* out0 = I->planes + ((rw >> 7) * I->kb_total + kb0) * kTileBytes + rr * kTileK + tl * plane_bytes + (place << 4);
    const int next_row = kTileK + ((place & 1) ? -16 : 16);  // rr is even when a warp has two rows
    for (int kb = kb0; kb < kb1; ++kb, out0 += kTileBytes) {
        const uint32_t buf = ((kb - kb0) & 1) * kSplitTileBytes;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (ROWC) __syncthreads();  // the whole block's copies; the other buffer's readers are done
        else __syncwarp();
        if (kb + 1 < kb1) fetch(kb + 1, buf ^ kSplitTileBytes);
        if (nrows <= 0) continue;
        uint32_t W[R][NG][4][NW];
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                // k contiguous: 4 j is bits 2, 3 of the inner index, which the swizzle flips
                const uint32_t at = buf + (ROWC ? (el0 ^ (u * E)) + j * (4 * split_rows<CPLX>() * E)
                                                : (CPLX ? (el0 ^ ((j & 1) << 6)) + ((j & 2) << 6) : (el0 ^ (j << 5))) +
                                                      u * (kTileK * E));
                double y[NG];
                if constexpr (CPLX) {  // ordinary loads: the copies' waits above order them
                    const double2 v = *reinterpret_cast<const double2*>(tiles + at);
                    y[0] = v.x, y[1] = v.y;
                } else {
                    y[0] = *reinterpret_cast<const double*>(tiles + at);
                }
#pragma unroll
                for (int h = 0; h < NG; ++h) {
                    double x = y[h] * s1[u];
                    if (CPLX && h) x *= im_sign;
                    if (odd >> u & 1) {
                        const int e = exponent_of(mx[rw + u - mbase], I->tk);
                        x = e == kNonFinite ? 0.0 : x * pow2(e - max(-1000, min(1000, e)));
                    }
                    offset_words<NW>(x, W[u][h][j]);
                }
            }
        int8_t* out = out0;
#pragma unroll 1
        for (int grp = 0; 4 * grp < nmod; ++grp, out += tstep) {
            const uint4 av = S.a[grp][0][lane], mc = S.c[grp][tl], start = S.start[grp][tl];
            const uint32_t a[4] = {av.x, av.y, av.z, av.w};
            uint32_t a2[4] = {};
            if constexpr (NW > 2) {
                const uint4 bv = S.a[grp][1][lane];
                a2[0] = bv.x, a2[1] = bv.y, a2[2] = bv.z, a2[3] = bv.w;
            }
            const float finv = __uint_as_float(mc.y);
            const bool valid = 4 * grp + tl < nmod;
#pragma unroll
            for (int u = 0; u < R; ++u) {
                uint32_t w[NP][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t d[NG][4];
#pragma unroll
                    for (int h = 0; h < NG; ++h) {
                        mma_u8(d[h], a, W[u][h][j][0], W[u][h][j][1], start);
                        if constexpr (NW > 2) mma_u8_add(d[h], a2, W[u][h][j][2], NW > 3 ? W[u][h][j][NW - 1] : 0u);
                    }
#pragma unroll
                    for (int h = 0; h < NP; ++h) {
                        uint32_t r4[4];
#pragma unroll
                        for (int x = 0; x < 4; ++x)  // re + im: K m + (v0' + v1'), v0' + v1' < 2^21
                            r4[x] = sym_residue(CPLX && h == 2 ? d[0][x] + d[NG - 1][x] - mc.z : d[h % NG][x], finv, mc.x);
                        w[h][j] = pack_bytes(r4[0], r4[1], r4[2], r4[3]);
                    }
                }
                if (valid && u < nrows) {
                    int8_t* dst = out + u * next_row;
#pragma unroll
                    for (int h = 0; h < NP; ++h)
                        *reinterpret_cast<uint4*>(dst + h * gstride) = make_uint4(w[h][0], w[h][1], w[h][2], w[h][3]);
                }
            }
        }
    }
}

// A block: split_rows rows by I->kspan k blocks; block index -> (row block, k span). The layout is the item's
// (one branch per block), so both operands share one launch.
template <int NW, bool CPLX>
__global__ void __launch_bounds__(kSplitThreads, CPLX || NW == 2 ? 2 : 3)
    split_kernel(const SplitItem* items, int count) {
    __shared__ SplitShared<NW> S;
    // no chain_next: GEMM blocks placed while these drain land on the SMs in the order they fall free, and tiles
    // that share operands drift apart (8192^3, s = 14: 7.75 ms, 8.3 ms so placed)
    dev::chain_wait();
    const SplitItem* I = items + find_item(items, count, blockIdx.x);
    const int64_t local = static_cast<int64_t>(blockIdx.x) - I->block0;
    int64_t bx, by;
    divmod_index(local, I->rblocks, by, bx);
    split_consts<NW>(I, S);
    __syncthreads();
    const int kb0 = static_cast<int>(by) * I->kspan, kb1 = min(kb0 + I->kspan, static_cast<int>(I->kb_total));
    if (I->row_contig) split_tiles<NW, CPLX, true>(I, S, bx * split_rows<CPLX>(), kb0, kb1, I->maxbits, 0);
    else split_tiles<NW, CPLX, false>(I, S, bx * split_rows<CPLX>(), kb0, kb1, I->maxbits, 0);
}

// ------------------------------------------------------------------ scale fused into the split
// One launch for both phases of a real operand (ref src/ozaki2_gpu.hpp:974-989 then :1004-1022
// run them as two passes over A and B): a block owns RB whole plane rows, takes their maxima over
// all of k (and writes them for the CRT), then splits the same rows. The second read of the rows
// follows the first within the block, so it is served by L2 while the rows that all resident
// blocks have in flight fit there (the launcher uses it for k up to kFuseMaxK: at most 8 rows of
// 16 KiB, or 16 rows of 4 KiB, per block). k contiguous: a warp per row, lanes over k. Rows
// contiguous: a line per inner index, the 256 / RB thread groups over k.
template <int NW, bool ROWC>
__global__ void __launch_bounds__(kSplitThreads) scale_split_kernel(const SplitItem* __restrict__ items, int count) {
    constexpr int RB = split_rows<false>();  // rows per block
    __shared__ unsigned long long smax[RB];
    __shared__ SplitShared<NW> S;
    const SplitItem* __restrict__ I = items + find_item(items, count, blockIdx.x);
    split_consts<NW>(I, S);
    const int64_t r0 = (static_cast<int64_t>(blockIdx.x) - I->block0) * RB;
    const unsigned long long* X = reinterpret_cast<const unsigned long long*>(I->X);
    const int64_t rows = I->rows, k = I->k, ldx = I->ldx;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < RB) smax[tid] = 0;
    __syncthreads();
    if (ROWC) {
        const int64_t r = r0 + tid % RB;
        unsigned long long best = 0;
        if (r < rows) {
#pragma unroll 4
            for (int64_t p = tid / RB; p < k; p += 256 / RB) best = max(best, __ldg(X + r + p * ldx) & kAbsMask);
        }
        if (best) atomicMax(&smax[tid % RB], best);
    } else {
        for (int u = 0; u < RB / 8; ++u) {
            const int64_t r = r0 + (RB / 8) * warp + u;
            unsigned long long best = 0;
            if (r < rows) {
#pragma unroll 4
                for (int64_t p = lane; p < k; p += 32) best = max(best, __ldg(X + p + r * ldx) & kAbsMask);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xFFFFFFFFu, best, o));
            if (lane == 0) smax[(RB / 8) * warp + u] = best;
        }
    }
    __syncthreads();
    if (tid < RB && r0 + tid < rows) const_cast<unsigned long long*>(I->maxbits)[r0 + tid] = smax[tid];  // for the CRT
    split_tiles<NW, false, ROWC>(I, S, r0, 0, static_cast<int>(I->kb_total), smax, r0);
}

// ------------------------------------------------------------------ tensor-core split
// The byte dot products v_t = Sum_l byte_l (2^(8 l) mod m_t) form a small
// matrix product: (moduli x bytes) times (bytes x elements). One tcgen05.mma kind::i8 (unsigned
// A and B, M = 128, N = 256, K = 32, int32 in TMEM) computes them for a unit of 512 elements:
//   B (N x K, K-major): column n holds two elements, segment g = 0, 1 in bytes 16 g .. 16 g + 15
//     (the offset integer's 8 / 12 / 16 bytes, zero-filled);
//   A (M x K, K-major): row 32 q + l is the slot sigma = 32 (q % Qa) + l, sigma < 2 s: segment
//     sigma / s, modulus sigma % s, the weights 2^(8 l) mod m in that segment's bytes. With
//     Qa = 1 (s <= 16) all four TMEM lane quarters hold the same 32 slots, with Qa = 2 (s <= 32)
//     quarters 0, 1 hold the 2 s slots and 2, 3 repeat them, so every epilogue warp reads its own
//     lane quarter (a hardware rule) and the quarters split the 256 columns between them.
// The epilogue turns v + koff into the residue (x + h) mod m by the exact multiply-high quotient
// (v < 2^20), subtracts h modulo 256 and stores the 32 residues of one slot's 32 consecutive
// inner indices as one 32-byte piece of its plane. The integer pipe keeps one multiply-high and
// one multiply-subtract per residue.
// Persistent, one CTA per SM with 16 warps, software-pipelined over the CTA's units: while the
// MMA of unit k runs, the threads finish unit k - 1 from the other accumulator (two A and two B
// tiles, 2 x 256 TMEM columns); a unit's FP64 loads are issued kTcAhead units ahead, into
// registers.
constexpr int kTcThreads = 512;
constexpr int kTcAhead = 3;
constexpr int kTcSmem = 1024 + 2 * 16384 + 2 * 32768 + 64;  // two A tiles, two B tiles, barriers + TMEM slot
constexpr int kTcSmemLaunch = 160 * 1024;                   // one CTA per SM (TMEM: 2 x 256 columns)
constexpr uint32_t kTcIdesc = (2u << 4)                     // D: s32; A, B: unsigned 8-bit, K-major
                              | (static_cast<uint32_t>(256 >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);

template <bool ROWC>
struct TcGeom {
    static constexpr int UR = ROWC ? 16 : 4;    // rows per unit
    static constexpr int UK = ROWC ? 32 : 128;  // inner indices per unit
    // element f = 0..511 of a unit -> row offset, inner offset (loads: coalesced along the
    // contiguous index), segment and column
    __device__ static void element(int f, int& ro, int& po, int& seg, int& n) {
        if (ROWC) {
            ro = f & 15;
            po = f >> 4;
            seg = ro >> 3;
            n = ((ro & 7) << 5) | po;
        } else {
            ro = f >> 7;
            po = f & 127;
            seg = ro >> 1;
            n = ((ro & 1) << 7) | po;
        }
    }
    // the 32 columns n0 .. n0 + 31 of segment seg -> row offset and first inner offset
    __device__ static void chunk(int seg, int n0, int& ro, int& po) {
        if (ROWC) {
            ro = 8 * seg + (n0 >> 5);
            po = 0;
        } else {
            ro = 2 * seg + (n0 >> 7);
            po = n0 & 127;
        }
    }
};

template <int NW>
__device__ __forceinline__ void offset_words_padded(double y, uint32_t (&W)[4]) {
    if constexpr (NW == 2) {
        uint32_t w[2];
        offset_words_fp(y, w);
        W[0] = w[0], W[1] = w[1], W[2] = 0, W[3] = 0;
    } else if constexpr (NW == 3) {
        uint32_t w[3];
        offset_words_fp_wide(y, w);
        W[0] = w[0], W[1] = w[1], W[2] = w[2], W[3] = 0;
    } else {
        offset_words_fp_widest(y, W);
    }
}

template <int NW, bool ROWC>
__global__ void __launch_bounds__(kTcThreads, 1) split_tc_kernel(const SplitItem* __restrict__ items, int count,
                                                                int64_t units, int* err) {
    using G = TcGeom<ROWC>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t{1023});
    uint8_t* sA0 = smem;              // two 128 rows x 128 bytes (swizzled; the first two chunks used)
    uint8_t* sB0 = smem + 2 * 16384;  // two 256 rows x 128 bytes
    uint64_t* bar_p = reinterpret_cast<uint64_t*>(smem + 2 * 16384 + 2 * 32768);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_p + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        dev::mbar_init(dev::smem_addr(bar_p), 1);
        dev::mbar_init(dev::smem_addr(bar_p + 1), 1);
        *abort_flag = 0;
        dev::fence_barrier_init();
    }
    if (warp == 0) {
        dev::tmem_alloc(dev::smem_addr(tmem_slot), 512);
        dev::tmem_relinquish();
    }
    dev::tc_fence_before();
    __syncthreads();
    dev::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int64_t stride = gridDim.x;
    const int64_t nmine = units > blockIdx.x ? (units - 1 - blockIdx.x) / stride + 1 : 0;
    int ro_l, po_l, seg_l, n_l;  // this thread's element of every unit
    G::element(tid, ro_l, po_l, seg_l, n_l);

    int first = 0;
    {  // the item of this CTA's first unit; later units only move forward
        int hi = count - 1;
        const int64_t u = blockIdx.x;
        while (first < hi) {
            const int mid = (first + hi + 1) >> 1;
            if (items[mid].block0 <= u) first = mid;
            else hi = mid - 1;
        }
    }
    auto advance = [&](int& cur, int64_t u) {
        while (cur + 1 < count && items[cur + 1].block0 <= u) ++cur;
    };
    // the element's value (0 outside the item's rows and k, and for non-finite rows, whose
    // residues are then zero like the padding's) and its row's maximum bits
    int cur_l = first;
    auto load_elem = [&](int64_t kk, double& v, unsigned long long& mb) {
        v = 0.0;
        mb = 0;
        if (kk >= nmine) return;
        const int64_t u = blockIdx.x + kk * stride;
        advance(cur_l, u);
        const SplitItem* I = items + cur_l;
        const int64_t local = u - I->block0;
        int64_t qd, rm;
        divmod_index(local, I->rblocks, qd, rm);
        const int64_t r = rm * G::UR + ro_l, p = qd * G::UK + po_l;
        if (r < I->rows && p < I->k) {
            mb = __ldg(I->maxbits + r);
            if (mb < 0x7FF0000000000000ull) v = __ldg(I->X + (ROWC ? r + p * I->ldx : p + r * I->ldx));
        }
    };
    double pv[kTcAhead];
    unsigned long long pm[kTcAhead];
#pragma unroll
    for (int a = 0; a < kTcAhead; ++a) load_elem(a, pv[a], pm[a]);

    int cur_w = first, cur_e = first;  // items of the unit being written and of the one being finished
    int a_item0 = -1, a_item1 = -1;    // item whose weights are in A tile 0 / 1
    int e_item = -1;                   // item of the epilogue lane constants
    bool valid = false;
    int seg = 0, qa = 1;
    uint32_t m = 1, m32 = 0, koff = 0, c256h = 0;
    int8_t* plane = nullptr;
    bool ok = true;
    uint32_t committed = 0, last_par = 0;  // (thread 0) per accumulator: a commit issued, its parity
    for (int64_t kb = 0; ok && kb <= nmine; kb += kTcAhead) {
#pragma unroll
        for (int a = 0; a < kTcAhead; ++a) {
            const int64_t kk = kb + a;  // unit kk is written, unit kk - 1 finished
            if (!ok || kk > nmine) break;
            const int buf = static_cast<int>(kk & 1);
            if (kk < nmine) {
                const int64_t u = blockIdx.x + kk * stride;
                advance(cur_w, u);
                const SplitItem* __restrict__ I = items + cur_w;
                if ((buf ? a_item1 : a_item0) != cur_w) {  // unit kk - 2's MMA, this tile's last reader, is complete
                    if (buf) a_item1 = cur_w;
                    else a_item0 = cur_w;
                    if (tid < 128) {
                        const int s = I->s, q2 = s <= 16 ? 1 : 2;
                        const int sigma = 32 * ((tid >> 5) % q2) + (tid & 31);
                        uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0;
                        if (sigma < 2 * s) {
                            const SplitMod& c = I->mc[sigma % s];
                            const uint4 cw = make_uint4(c.cb[0], c.cb[1], NW > 2 ? c.cb[2] : 0u, NW > 3 ? c.cb[3] : 0u);
                            if (sigma < s) w0 = cw;
                            else w1 = cw;
                        }
                        uint8_t* row = sA0 + buf * 16384 + tid * 128;
                        *reinterpret_cast<uint4*>(row + ((0 ^ (tid & 7)) << 4)) = w0;
                        *reinterpret_cast<uint4*>(row + ((1 ^ (tid & 7)) << 4)) = w1;
                    }
                }
                const int e = exponent_of(pm[a], I->tk);
                const bool live = e != kNonFinite;
                const int e1 = e >> 1;
                const double s1 = pow2(live ? e1 : 0), s2 = pow2(live ? e - e1 : 0);
                uint32_t W[4];
                offset_words_padded<NW>((pv[a] * s1) * s2, W);
                *reinterpret_cast<uint4*>(sB0 + buf * 32768 + n_l * 128 + ((seg_l ^ (n_l & 7)) << 4)) =
                    make_uint4(W[0], W[1], W[2], W[3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            dev::tc_fence_before();
            __syncthreads();
            if (kk < nmine && tid == 0) {
                dev::tc_fence_after();
                dev::mma_i8(tmem + static_cast<uint32_t>(buf * 256), dev::sw128_kmajor_desc(dev::smem_addr(sA0 + buf * 16384)),
                            dev::sw128_kmajor_desc(dev::smem_addr(sB0 + buf * 32768)), kTcIdesc, 0u);
                dev::tc_commit(dev::smem_addr(bar_p + buf));
                committed |= 1u << buf;
                last_par = (last_par & ~(1u << buf)) | (static_cast<uint32_t>((kk >> 1) & 1) << buf);
            }
            if (kk < nmine) load_elem(kk + kTcAhead, pv[a], pm[a]);
            if (kk > 0) {  // finish unit kk - 1
                const int pb = buf ^ 1;
                const uint32_t parity = static_cast<uint32_t>(((kk - 1) >> 1) & 1);
                int got = 1;  // one thread waits; the others sleep in the block barrier
                if (tid == 0)
                    got = dev::mbar_wait(dev::smem_addr(bar_p + pb), parity, abort_flag, err, dev::kErrTimeoutAccFull,
                                         dev::kWaitLimitNs) ? 1 : 0;
                if (!__syncthreads_and(got)) {
                    ok = false;
                    break;
                }
                dev::tc_fence_after();
                const int64_t u = blockIdx.x + (kk - 1) * stride;
                advance(cur_e, u);
                const SplitItem* __restrict__ I = items + cur_e;
                if (cur_e != e_item) {
                    e_item = cur_e;
                    const int s = I->s;
                    qa = s <= 16 ? 1 : 2;
                    const int sigma = 32 * ((warp & 3) % qa) + lane;
                    valid = sigma < 2 * s;
                    if (valid) {
                        const int t = sigma % s;
                        const SplitMod& c = I->mc[t];
                        const uint32_t h = (c.m - 1) / 2;  // residues symmetric in [-h, m - 1 - h]
                        seg = sigma / s;
                        m = c.m;
                        // ceil(2^32 / m): floor(v / m) = umulhi(v, m32) exactly for v < 2^24 (Granlund
                        // and Montgomery, 1994)
                        m32 = 0xFFFFFFFFu / m + 1u;
                        koff = (h + c.off) % m;
                        c256h = 256u - h;
                        plane = I->planes + t * I->plane_bytes;
                    }
                }
                const int64_t local = u - I->block0;
                int64_t qd, rm;
                divmod_index(local, I->rblocks, qd, rm);
                const int64_t r0 = rm * G::UR, p0 = qd * G::UK;
                // warp (quarter q, part pt) reads lane quarter q: with qa = 1 (four copies of the
                // slots) 16 columns, with qa = 2 (two copies) 32 columns
                const int q = warp & 3, pt = warp >> 2;
                const uint32_t taddr = tmem + (static_cast<uint32_t>(32 * q) << 16) + static_cast<uint32_t>(pb * 256);
                if (qa == 1) {
                    const int n0 = 16 * (4 * q + pt);
                    uint32_t d[16];
                    dev::tmem_load_32x16(taddr + n0, d);
                    dev::tmem_load_wait();
                    if (valid) {
                        int ro, po;
                        G::chunk(seg, n0 & ~31, ro, po);
                        const int64_t r = r0 + ro, pk = p0 + po + (n0 & 31);
                        const int rr = static_cast<int>(r & 127);
                        const int c = static_cast<int>((pk & 127) >> 4);
                        int8_t* tile = plane + ((r >> 7) * I->kb_total + (pk >> 7)) * kTileBytes + rr * kTileK;
                        uint32_t w[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint32_t r4[4];
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const uint32_t v = d[4 * j + b] + koff;     // < 2^20 + 2^8
                                r4[b] = v - __umulhi(v, m32) * m + c256h;  // low byte: (x mod m, symmetric)
                            }
                            w[j] = pack_bytes(r4[0], r4[1], r4[2], r4[3]);
                        }
                        *reinterpret_cast<uint4*>(tile + ((c ^ (rr & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                } else {
                    const int n0 = 32 * (4 * (q >> 1) + pt);
                    uint32_t d[32];
                    dev::tmem_load_32x32(taddr + n0, d);
                    dev::tmem_load_wait();
                    if (valid) {
                        int ro, po;
                        G::chunk(seg, n0, ro, po);
                        const int64_t r = r0 + ro, pk = p0 + po;
                        const int rr = static_cast<int>(r & 127);
                        const int c = static_cast<int>((pk & 127) >> 4);
                        int8_t* tile = plane + ((r >> 7) * I->kb_total + (pk >> 7)) * kTileBytes + rr * kTileK;
                        uint32_t w[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint32_t r4[4];
#pragma unroll
                            for (int b = 0; b < 4; ++b) {
                                const uint32_t v = d[4 * j + b] + koff;
                                r4[b] = v - __umulhi(v, m32) * m + c256h;
                            }
                            w[j] = pack_bytes(r4[0], r4[1], r4[2], r4[3]);
                        }
                        *reinterpret_cast<uint4*>(tile + ((c ^ (rr & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
                        *reinterpret_cast<uint4*>(tile + (((c + 1) ^ (rr & 7)) << 4)) = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
            }
        }
    }
    if (!ok && tid == 0) {  // the last MMA of each accumulator completes before TMEM is freed
        for (int b = 0; b < 2; ++b)
            if (committed & (1u << b)) dev::mbar_wait_drain(dev::smem_addr(bar_p + b), (last_par >> b) & 1u);
    }
    dev::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        dev::tc_fence_after();
        dev::tmem_dealloc(tmem, 512);
    }
}

// Ozaki Scheme I digits (the reference's comparison baseline, benchmarks/ozaki1_gpu.hpp:31-40):
// x = RNE(v 2^e) as on the narrow split path (tk = 7L - 2 <= 61), then L balanced base-128
// digits in [-64, 63], most significant in plane 0, written in the same plane layout and with
// 16 elements of one row per thread. Rows contiguous: a warp is 16 rows by 2 pieces of 16 inner
// indices, a block 16 rows by kSliceRowcK; otherwise a warp is one row by 32 pieces, a block 8 rows.
constexpr int kSliceEpt = 16, kSliceRowcK = 256;
template <bool ROWC>
__global__ void __launch_bounds__(256) slice_kernel(const SplitItem* __restrict__ items, int count) {
    constexpr int EPT = kSliceEpt;
    const SplitItem* __restrict__ I = items + find_item(items, count, blockIdx.x);
    const int64_t local = static_cast<int64_t>(blockIdx.x) - I->block0;
    int64_t bx, by;
    divmod_index(local, I->rblocks, by, bx);
    const int lane = static_cast<int>(threadIdx.x & 31), warp = static_cast<int>(threadIdx.x >> 5);
    const int64_t r = ROWC ? bx * EPT + lane % EPT : bx * 8 + warp;
    const int64_t k0 = ROWC ? by * kSliceRowcK + (warp * (32 / EPT) + lane / EPT) * EPT : by * (32 * EPT) + lane * EPT;
    const int64_t kb_total = I->kb_total, plane_bytes = I->plane_bytes, ldx = I->ldx, k = I->k;
    if (r >= I->rows_pad || k0 >= kb_total * kTileK) return;
    const int ndig = I->s;
    const int64_t rb = r >> 7;
    const int rr = static_cast<int>(r & 127);
    const int c = static_cast<int>((k0 >> 4) & 7);
    int8_t* out = I->planes + (rb * kb_total + (k0 >> 7)) * kTileBytes + rr * kTileK + ((c ^ (rr & 7)) << 4);
    long long x[EPT];
#pragma unroll
    for (int q = 0; q < EPT; ++q) x[q] = 0;
    if (r < I->rows && k0 < k) {
        const int e = exponent_of(I->maxbits[r], I->tk);
        if (e != kNonFinite) {
            const int e1 = e >> 1;
            const double s1 = pow2(e1), s2 = pow2(e - e1);
#pragma unroll
            for (int q = 0; q < EPT; ++q) {
                const int64_t p = k0 + q;
                if (p < k) x[q] = __double2ll_rn((__ldg(I->X + (ROWC ? r + p * ldx : p + r * ldx)) * s1) * s2);
            }
        }
    }
    // least significant digit first, into planes ndig - 1 .. 0
    for (int i = ndig - 1; i >= 0; --i) {
        uint32_t b[EPT];
#pragma unroll
        for (int q = 0; q < EPT; ++q) {
            const long long d = ((x[q] + 64) & 127) - 64;
            x[q] = (x[q] - d) >> 7;
            b[q] = static_cast<uint32_t>(d);
        }
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = pack_bytes(b[4 * q], b[4 * q + 1], b[4 * q + 2], b[4 * q + 3]);
        *reinterpret_cast<uint4*>(out + i * plane_bytes) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

template <int NW>
void split_tc_dispatch(const SplitItem* d, int count, int64_t units, bool rowc, int* err, cudaStream_t st) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(units, static_cast<int64_t>(sms)));
    if (rowc) split_tc_kernel<NW, true><<<grid, kTcThreads, kTcSmemLaunch, st>>>(d, count, units, err);
    else split_tc_kernel<NW, false><<<grid, kTcThreads, kTcSmemLaunch, st>>>(d, count, units, err);
}

std::atomic<int> g_split_tc{0};
std::atomic<int> g_scale_fusion{0};

template <int NW>
void scale_split_dispatch(const SplitItem* d, int count, int64_t blocks, bool rowc, cudaStream_t st) {
    const unsigned g = static_cast<unsigned>(blocks);
    if (rowc) scale_split_kernel<NW, true><<<g, kSplitThreads, 0, st>>>(d, count);
    else scale_split_kernel<NW, false><<<g, kSplitThreads, 0, st>>>(d, count);
}

template <int NW, bool CPLX>
void split_dispatch(const SplitItem* d, int count, int64_t blocks, cudaStream_t st) {
    launch_chained(split_kernel<NW, CPLX>, static_cast<unsigned>(blocks), kSplitThreads, 0, st, d, count);
}

}  // namespace

int64_t scale_item_blocks(ScaleItem& it, int num_sms, int64_t block0) {
    it.block0 = block0;
    if (it.rows <= 0 || it.k <= 0) {
        it.rblocks = 1;
        it.kchunk = 1;
        return 0;
    }
    const int64_t target = static_cast<int64_t>(num_sms) * 2048 * 2;  // threads in flight
    if (it.row_contig) {
        it.rblocks = ceil_div(it.rows, 32);
        // at least 64 inner indices per block (8 per warp)
        const int64_t chunks =
            std::max<int64_t>(1, std::min<int64_t>(ceil_div(it.k, 64), target / (it.rblocks * 256)));
        it.kchunk = ceil_div(it.k, chunks);
    } else {
        it.rblocks = ceil_div(it.rows, 8);
        const int64_t chunks = std::max<int64_t>(1, std::min<int64_t>(ceil_div(it.k, 256), target / (it.rows * 32)));
        it.kchunk = ceil_div(it.k, chunks);
    }
    return it.rblocks * ceil_div(it.k, it.kchunk);
}

int64_t slice_item_blocks(SplitItem& it, int64_t block0) {
    it.block0 = block0;
    const int64_t kpad = it.kb_total * kTileK;  // inner indices of the plane, padding included
    if (it.row_contig) {
        it.rblocks = ceil_div(it.rows_pad, kSliceEpt);
        it.kblocks = ceil_div(kpad, kSliceRowcK);
    } else {
        it.rblocks = ceil_div(it.rows_pad, 8);
        it.kblocks = ceil_div(kpad, 32 * kSliceEpt);
    }
    return it.rblocks * it.kblocks;
}

void split_launch_shape(SplitItem* items, int count, int num_sms) {
    // up to 16 k blocks per block (a block's start costs about a tile's time: 8192^3 split 779, 697 and
    // 682 us with at most 3, 8 and 16) while about four blocks per SM remain in the launch
    int64_t tiles = 0;
    for (int q = 0; q < count; ++q)
        tiles += ceil_div(items[q].rows, items[q].cplx ? split_rows<true>() : split_rows<false>()) * items[q].kb_total;
    const int span = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(16, tiles / (4 * num_sms))));
    for (int q = 0; q < count; ++q) items[q].kspan = span;
}

int64_t split_geometry(SplitItem& it, int64_t block0) {
    it.block0 = block0;
    const int rb = it.cplx ? split_rows<true>() : split_rows<false>();
    // 16-byte copies where every row (every element of complex rows) is 16-byte aligned
    it.vec = (reinterpret_cast<uintptr_t>(it.X) & 15) == 0 && (it.cplx || it.ldx % 2 == 0);
    if (it.fuse) {  // whole rows per block
        it.tc = 0;
        it.rblocks = ceil_div(it.rows, rb);
        it.kblocks = 1;
        return it.rblocks;
    }
    it.tc = !it.cplx && g_split_tc.load() ? 1 : 0;
    if (it.tc) {
        const int ur = it.row_contig ? TcGeom<true>::UR : TcGeom<false>::UR;
        const int uk = it.row_contig ? TcGeom<true>::UK : TcGeom<false>::UK;
        it.rblocks = it.rows_pad / ur;  // rows_pad is a multiple of 128
        it.kblocks = it.kb_total * (kTileK / uk);
        return it.rblocks * it.kblocks;
    }
    it.rblocks = ceil_div(it.rows, rb);
    it.kblocks = ceil_div(it.kb_total, it.kspan);
    return it.rblocks * it.kblocks;
}

void set_split_path(int tc) { g_split_tc.store(tc ? 1 : 0); }
void set_scale_fusion(int on) { g_scale_fusion.store(on ? 1 : 0); }
bool fuse_scale(bool cplx, bool row_contig, int64_t k) {
    return g_scale_fusion.load() && !cplx && k > 0 && k <= (row_contig ? kFuseMaxKRowc : kFuseMaxK);
}
int split_path() { return g_split_tc.load(); }

cudaError_t prepare_split_kernels() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* f) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmemLaunch);
    };
    set(reinterpret_cast<const void*>(split_tc_kernel<2, false>));
    set(reinterpret_cast<const void*>(split_tc_kernel<2, true>));
    set(reinterpret_cast<const void*>(split_tc_kernel<3, false>));
    set(reinterpret_cast<const void*>(split_tc_kernel<3, true>));
    set(reinterpret_cast<const void*>(split_tc_kernel<4, false>));
    set(reinterpret_cast<const void*>(split_tc_kernel<4, true>));
    return e;
}

void launch_scale(const ScaleItem* d, const ScaleItem* h, int count, int64_t blocks, cudaStream_t st) {
    if (count <= 0 || blocks <= 0) return;
    const unsigned g = static_cast<unsigned>(blocks);
    if (h[0].cplx) launch_chained(scale_kernel<true>, g, 256, 0, st, d, count);
    else launch_chained(scale_kernel<false>, g, 256, 0, st, d, count);
}

int64_t scale_rows_blocks(ScaleItem& it, int64_t block0) {
    it.block0 = block0;
    it.rblocks = ceil_div(it.rows, 32);
    it.kchunk = it.k;
    return it.rblocks;
}

void launch_scale_first(const void* blob, size_t bytes, void* dst, size_t off, int count, int64_t blocks, bool cplx,
                        cudaStream_t st) {
    unsigned char* d = static_cast<unsigned char*>(dst);
    const unsigned grid = static_cast<unsigned>(blocks) + 1;
    const uint32_t o = static_cast<uint32_t>(off);
    if (bytes <= 4608) scale_first_n<4608>(blob, bytes, d, o, count, grid, cplx, st);  // two operands: 4248
    else scale_first_n<kScaleFirstBytes>(blob, bytes, d, o, count, grid, cplx, st);
}

void launch_slice(const SplitItem* d, const SplitItem* h, int count, int64_t blocks, cudaStream_t st) {
    if (count <= 0 || blocks <= 0) return;
    if (h[0].row_contig) slice_kernel<true><<<static_cast<unsigned>(blocks), 256, 0, st>>>(d, count);
    else slice_kernel<false><<<static_cast<unsigned>(blocks), 256, 0, st>>>(d, count);
}

void launch_split(const SplitItem* d, const SplitItem* h, int count, int64_t blocks, int* err, cudaStream_t st) {
    if (count <= 0 || blocks <= 0) return;
    const int words = split_words(h[0].tk);
    const bool rowc = h[0].row_contig != 0;
    if (h[0].fuse) {
        if (words == 4) scale_split_dispatch<4>(d, count, blocks, rowc, st);
        else if (words == 3) scale_split_dispatch<3>(d, count, blocks, rowc, st);
        else scale_split_dispatch<2>(d, count, blocks, rowc, st);
    } else if (h[0].tc) {
        if (words == 4) split_tc_dispatch<4>(d, count, blocks, rowc, err, st);
        else if (words == 3) split_tc_dispatch<3>(d, count, blocks, rowc, err, st);
        else split_tc_dispatch<2>(d, count, blocks, rowc, err, st);
    } else if (h[0].cplx) {  // s <= 24: at most three words
        if (words == 3) split_dispatch<3, true>(d, count, blocks, st);
        else split_dispatch<2, true>(d, count, blocks, st);
    } else {
        if (words == 4) split_dispatch<4, false>(d, count, blocks, st);
        else if (words == 3) split_dispatch<3, false>(d, count, blocks, st);
        else split_dispatch<2, false>(d, count, blocks, st);
    }
}

}  // namespace oz2
