// oz2_crt.cu - CRT reconstruction of the Ozaki-II path: per C entry, s residues r_t
// (bytes) -> the exact integer x = Sum_t r_t W_t - q M (|x| <= M/4) -> one round-to-nearest-even to
// a double -> * 2^-(D_i + E_j) -> alpha/beta update (oz2_crt_math.cuh). Ref
// src/ozaki2_gpu.hpp:526-588 (CrtAcc), :603-626 (launch_crt), :628-664 (launch_crt_cplx, 3M
// recombination Re = P0 - P1, Im = P2 - P0 - P1).
//
// s bytes of residues per entry in (3s for complex), 8 (16) bytes of C out, plus 8 (16) in when
// beta != 0.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "oz2_kernels.cuh"
#include "oz2_crt_math.cuh"
#include "oz2_ptx.cuh"

namespace oz2 {
namespace {

// ---------------------------------------------------------------- CRT on mma.sync
// The limb sums are a small integer matrix product, entries by moduli times moduli by weight bytes:
// mma.sync u8 (signed residues: s8) x u8 -> s32 with 16 entries in the rows of A, the moduli along K (16, or 32 for s > 16)
// and 8 bytes of W_t in the columns of B. A warp takes the 32 rows of a row block in one column at a
// time: lane (g, c) = (lane / 4, lane % 4) reads the residue words (rows g, g + 8, g + 16, g + 24) of
// the moduli 4 c .. 4 c + 3, and a 4 x 4 byte transpose makes them the A fragments of the four rows;
// the B fragments stay in registers for the whole launch. A lane's two columns of the product are
// the two bytes of one 16-bit limb, so it holds limb 4 T + c (tile T of 8 bytes) of four rows, which
// go through shared memory to the lane of their row: lane l finishes row l (crt_words, crt_round)
// and a warp reads and writes 32 consecutive entries of C. Complex: the three products' limb sums
// are combined (Re = P0 - P1, Im = P2 - P0 - P1) before the quotient.
// Residues arrive through cp.async, four columns (one 128-byte line per plane) ahead.
// Bound: instruction issue (166 warp instructions per 32 entries at s = 16, 34 cycles of them the four
// mma at 8.6 each; the dp2a form it replaces took 304, 72 of them two-cycle dot products whose weights
// had to be moved to registers), then DRAM. Four blocks per SM up to 8 limbs (64 registers), three
// above, two for complex operands (of 24 residue planes above 8 limbs). CRT stage, start -> now, alternating in one process: 8192^2, s = 16,
// beta != 0 1019 -> 595 us (332 us of DRAM time at the measured copy rate); 6144^2, s = 20 757 -> 566;
// 4096^2, s = 24 315 -> 193, s = 32 (a tcgen05 form before) 451 -> 221; ZGEMM 4096^2, s = 16 720 -> 429, s = 18
// 890 -> 482 (736 with one block per SM, before complex plans kept 24 planes only), 1000^2, s = 18 60 -> 56 (87);
// 512 grouped problems 1506 -> 1111.
// columns of a warp tile: a 128-byte line per plane, or half of one where shared memory would cost blocks
constexpr int crt_cols(int L, bool cplx) { return cplx || L > 8 ? 2 : 4; }
constexpr int crt_pitch(int L) { return L <= 4 ? 4 : (L <= 12 ? 12 : 20); }  // words per row, 4 x odd: no bank conflicts
template <int L, bool CPLX>
struct alignas(128) CrtWarp {  // a warp's shared memory
    static constexpr int KH = L <= 8 ? 1 : 2, G = CPLX ? 3 : 1, W = CPLX ? 2 : 1;
    static constexpr int kCols = crt_cols(L, CPLX);
    // residue planes kept: complex plans stop at 24 moduli, and with 32 planes a second block would not fit the SM
    static constexpr int kPlanes = KH == 1 ? 16 : (CPLX ? kMaxModuli : kMaxModuliExt);
    uint8_t res[2][G][kPlanes][32 * kCols];
    uint32_t limb[W][32][crt_pitch(L)];
};
struct CrtParams {
    const CrtItem* items;
    int count, s;
    uint32_t M16[kLimbs16];
    float qf[kLimbs16];
    alignas(16) uint8_t wb[2 * kLimbs16][32];  // byte b of W_t for t = 0..31 (zero past s)
};

// residues as signed or unsigned bytes times unsigned weight bytes
template <bool SGN>
__device__ __forceinline__ void mma_res_k16(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    if constexpr (SGN)
        asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(b), "r"(0));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(b), "r"(0));
}
template <bool SGN>
__device__ __forceinline__ void mma_res_k32(uint32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1) {
    if constexpr (SGN)
        asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
    else
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
            : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

constexpr int crt_blocks(int L, bool cplx) { return cplx ? 2 : (L <= 8 ? 4 : 3); }  // per SM
template <int L, bool CPLX>
__global__ void __launch_bounds__(256, crt_blocks(L, CPLX)) crt_kernel(const __grid_constant__ CrtParams P) {
    using Warp = CrtWarp<L, CPLX>;
    constexpr int KH = Warp::KH, G = Warp::G, NT = (L + 3) / 4, PL = Warp::kPlanes, COLS = Warp::kCols, W2 = Warp::W;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    const int warp = static_cast<int>(threadIdx.x >> 5), lane = static_cast<int>(threadIdx.x & 31);
    Warp& S = reinterpret_cast<Warp*>(smem_raw)[warp];
    const int g = lane >> 2, c = lane & 3;
    uint32_t B[NT][KH];
#pragma unroll
    for (int T = 0; T < NT; ++T)
#pragma unroll
        for (int h = 0; h < KH; ++h) B[T][h] = *reinterpret_cast<const uint32_t*>(&P.wb[8 * T + g][16 * h + 4 * c]);
    dev::chain_wait();  // no chain_next: what follows is another program's, or the caller's
    int lo = 0, hi = P.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.items[mid].block0 <= static_cast<int64_t>(blockIdx.x)) lo = mid;
        else hi = mid - 1;
    }
    const CrtItem* I = P.items + lo;
    int64_t jblk, ib;
    divmod_index(static_cast<int64_t>(blockIdx.x) - I->block0, I->iblocks, jblk, ib);
    const int tk = I->tk, s = P.s;
    const int64_t m = I->m, n = I->n, ldc = I->ldc, i = ib * 32 + lane;
    const double ar = I->ar, ai = I->ai, br = I->br, bi = I->bi;
    const bool beta = br != 0.0 || (CPLX && bi != 0.0), in = i < m, sgn = I->sgn;
    const int De = in ? unscale_exponent(I->maxA[i], tk) : 0;
    const int64_t rstride = I->rstride, gstride = I->gstride;
    // the block's warps take neighbouring groups of COLS columns, I->jc times
    const int64_t jstep = 8 * COLS, span = jstep * I->jc;
    int64_t j0 = jblk * span + warp * COLS;
    const int64_t jend = min(n, (jblk + 1) * span);
    constexpr int CH = 2 * COLS, PI = 32 / CH;  // 16-byte chunks per plane, planes per copy instruction
    const int p0 = lane / CH, col0 = (lane % CH) >> 1;
    const uint8_t* src = I->resid + ib * (32 * n) + 16 * (lane % CH) + p0 * rstride;
    const unsigned long long* maxB = I->maxB;
    const int64_t cstep = W2 * ldc;
    double* cp = I->C + W2 * i + j0 * cstep;
    // Column k of plane p lies at 32-byte slot (p COLS + k) ^ (p / 4 % 4), so that the lanes' reads (moduli
    // 4 c + u of one column) meet no bank conflict.
    auto fetch = [&](int buf, int64_t j) {
        const bool ok = j + col0 < n;
        const uint32_t dst = dev::smem_addr(&S.res[buf][0][0][0]) + ((lane & 1) << 4);
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const uint8_t* p = src + h * gstride + j * 32;
#pragma unroll
            for (int x = 0; x < PL / PI; ++x, p += PI * rstride) {
                const int pl = PI * x + p0;
                const bool in_p = ok && pl < s;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                 dst + h * (PL * 32 * COLS) + (((pl * COLS + col0) ^ (pl >> 2 & 3)) << 5)),
                             "l"(in_p ? p : I->resid), "r"(in_p ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto column_max = [&](int64_t j) { return j + (lane & (COLS - 1)) < n ? maxB[j + (lane & (COLS - 1))] : 0ull; };
    unsigned long long mb = 0;
    if (j0 < jend) {
        fetch(0, j0);
        mb = column_max(j0);
    }
    // the lane's words of a column: moduli 4 c + u, and 16 + 4 c + u (past the kept planes any word will do: its
    // weights are zero), rows g + 8 e
    const uint32_t upper = 16 + 4 * c < PL ? 16 * (32 * COLS) : 0;
    const uint32_t at = dev::smem_addr(&S.res[0][0][0][0]) + 4 * c * (32 * COLS) + 4 * g;
    for (int buf = 0; j0 < jend; j0 += jstep, buf ^= 1) {
        const int Ec = unscale_exponent(mb, tk);  // of column j0 + lane % COLS
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (j0 + jstep < jend) {
            fetch(buf ^ 1, j0 + jstep);
            mb = column_max(j0 + jstep);
        }
        const int cols = static_cast<int>(min(n - j0, int64_t{COLS}));
#pragma unroll 1
        for (int k = 0; k < cols; ++k, cp += cstep) {
            double c0 = 0.0, c1 = 0.0;
            if (beta && in) {
                c0 = cp[0];
                if (CPLX) c1 = cp[W2 - 1];
            }
            const uint32_t slot = at + buf * static_cast<uint32_t>(sizeof S.res[0]) + ((k ^ (COLS == 4 ? c : 0)) << 5);
            uint32_t o[G][KH][4];  // A fragments: entry rows g + 8 e
#pragma unroll
            for (int h = 0; h < G; ++h)
#pragma unroll
                for (int x = 0; x < KH; ++x) {
                    uint32_t w[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        asm volatile("ld.shared.u32 %0, [%1];"
                                     : "=r"(w[u])
                                     : "r"((COLS == 4 ? slot : slot ^ ((((u & 1) << 1) ^ c) << 5)) + h * PL * (32 * COLS) +
                                           x * upper + (COLS == 4 ? u * 128 : (u >> 1) * 128))
                                     : "memory");
                    transpose4(w[0], w[1], w[2], w[3], o[h][x]);
                }
            auto limbs = [&](auto sg) {
                constexpr bool SGN = decltype(sg)::value;
#pragma unroll
                for (int T = 0; T < NT; ++T)
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        uint32_t v[G][2];
#pragma unroll
                        for (int h = 0; h < G; ++h) {
                            uint32_t d[4];
                            if constexpr (KH == 1) mma_res_k16<SGN>(d, o[h][0][2 * mt], o[h][0][2 * mt + 1], B[T][0]);
                            else
                                mma_res_k32<SGN>(d, o[h][0][2 * mt], o[h][0][2 * mt + 1], o[h][KH - 1][2 * mt],
                                           o[h][KH - 1][2 * mt + 1], B[T][0], B[T][KH - 1]);
                            v[h][0] = d[0] + (d[1] << 8);
                            v[h][1] = d[2] + (d[3] << 8);
                        }
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            const int row = 8 * (2 * mt + y) + g;
                            if constexpr (CPLX) {  // below 2^31 in magnitude
                                S.limb[0][row][4 * T + c] = v[0][y] - v[1][y];
                                S.limb[CPLX][row][4 * T + c] = v[2 % G][y] - v[0][y] - v[1][y];
                            } else {
                                S.limb[0][row][4 * T + c] = v[0][y];
                            }
                        }
                    }
            };
            if (sgn) limbs(std::true_type{});
            else limbs(std::false_type{});
            __syncwarp();
            uint32_t a[CPLX ? 2 : 1][4 * NT];
#pragma unroll
            for (int h = 0; h < (CPLX ? 2 : 1); ++h)
#pragma unroll
                for (int T = 0; T < NT; ++T)
                    *reinterpret_cast<uint4*>(&a[h][4 * T]) = *reinterpret_cast<const uint4*>(&S.limb[h][lane][4 * T]);
            __syncwarp();
            const int shift = De + __shfl_sync(0xFFFFFFFFu, Ec, k);
            uint32_t w[CPLX ? 2 : 1][(L + 1) / 2];
            crt_words<L, CPLX ? 2 : 1, true>(
                [&](int l, uint32_t(&x)[CPLX ? 2 : 1]) {
                    x[0] = a[0][l];
                    if (CPLX) x[CPLX] = a[CPLX][l];
                },
                P.M16, P.qf, w);
            if constexpr (!CPLX) {
                const double v = crt_round<L>(w[0], shift);
                // the reference's unfused alpha*v + beta*c, one rounding per operation
                const double av = __dmul_rn(ar, v);
                if (in) cp[0] = beta ? __dadd_rn(av, __dmul_rn(br, c0)) : av;
            } else {
                const double vr = crt_round<L>(w[0], shift), vi = crt_round<L>(w[CPLX], shift);
                double orr = __dsub_rn(__dmul_rn(ar, vr), __dmul_rn(ai, vi));
                double oi = __dadd_rn(__dmul_rn(ar, vi), __dmul_rn(ai, vr));
                if (beta) {
                    orr = __dadd_rn(orr, __dsub_rn(__dmul_rn(br, c0), __dmul_rn(bi, c1)));
                    oi = __dadd_rn(oi, __dadd_rn(__dmul_rn(br, c1), __dmul_rn(bi, c0)));
                }
                if (in) {
                    cp[0] = orr;
                    cp[1] = oi;
                }
            }
        }
        cp += (jstep - COLS) * cstep;
    }
}

template <int L, bool CPLX>
constexpr int crt_smem() {
    constexpr int bytes = 8 * static_cast<int>(sizeof(CrtWarp<L, CPLX>));
    // the blocks that the registers are cut for have room in an SM's 228 KB (1 KB of it reserved per block)
    static_assert(crt_blocks(L, CPLX) * (bytes + 1024) <= 228 * 1024, "CRT blocks per SM");
    return bytes;
}

// by the plan's limbs; complex CRTs stop at s = 24 (zgemm is the reference's call): 12 limbs
template <int L>
void crt_dispatch(int limbs, const CrtParams& P, int64_t blocks, bool cplx, cudaStream_t st) {
    if constexpr (L <= kLimbs16) {
        if (limbs != L) return crt_dispatch<L + 1>(limbs, P, blocks, cplx, st);
        const unsigned grid = static_cast<unsigned>(blocks);
        if constexpr (L <= limbs16_for(kMaxModuli))
            if (cplx) {
                launch_chained(crt_kernel<L, true>, grid, 256, crt_smem<L, true>(), st, P);
                return;
            }
        launch_chained(crt_kernel<L, false>, grid, 256, crt_smem<L, false>(), st, P);
    }
}
template <int L>
cudaError_t crt_prepare() {
    if constexpr (L > kLimbs16) {
        return cudaSuccess;
    } else {
        cudaError_t e = cudaFuncSetAttribute(crt_kernel<L, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, crt_smem<L, false>());
        if constexpr (L <= limbs16_for(kMaxModuli))
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(crt_kernel<L, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, crt_smem<L, true>());
        return e == cudaSuccess ? crt_prepare<L + 1>() : e;
    }
}

// block 0 writes the blob, the others zero their share of [zero, zero + 16 nzero)
template <int N>
__global__ void write_blob_kernel(const __grid_constant__ BlobParam<N> b, unsigned char* dst, uint4* zero, size_t nzero) {
    dev::chain_next();
    if (blockIdx.x) {
        const size_t stride = static_cast<size_t>(gridDim.x - 1) * blockDim.x;
        for (size_t i = static_cast<size_t>(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < nzero; i += stride)
            zero[i] = make_uint4(0, 0, 0, 0);
        return;
    }
    for (uint32_t i = threadIdx.x * 16; i < b.bytes; i += blockDim.x * 16)
        *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(b.data + i);
}
template <int N>
void write_blob_n(const unsigned char* src, size_t n, unsigned char* dst, cudaStream_t st, void* zero, size_t zero_bytes) {
    static thread_local BlobParam<N> bp;
    std::memcpy(bp.data, src, n);
    bp.bytes = static_cast<uint32_t>((n + 15) & ~size_t{15});
    const unsigned fill = static_cast<unsigned>(std::min<size_t>((zero_bytes / 16 + 255) / 256, 4 * 148));
    write_blob_kernel<N><<<1 + fill, 256, 0, st>>>(bp, dst, static_cast<uint4*>(zero), zero_bytes / 16);
}

// VEC: both pointers 16-byte aligned, 16-byte words first
template <bool VEC>
__global__ void sm_copy_kernel(const unsigned char* __restrict__ src, unsigned char* __restrict__ dst, size_t bytes) {
    const size_t tid = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t tail = 0;
    if (VEC) {
        const size_t n16 = bytes / 16;
        for (size_t i = tid; i < n16; i += stride)
            reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
        tail = n16 * 16;
    }
    for (size_t i = tail + tid; i < bytes; i += stride) dst[i] = src[i];
}

template <bool VEC>
__global__ void fill_kernel(unsigned char* __restrict__ dst, uint32_t word, size_t bytes) {
    dev::chain_next();
    const size_t tid = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    size_t tail = 0;
    if (VEC) {
        const size_t n16 = bytes / 16;
        for (size_t i = tid; i < n16; i += stride) reinterpret_cast<uint4*>(dst)[i] = make_uint4(word, word, word, word);
        tail = n16 * 16;
    }
    for (size_t i = tail + tid; i < bytes; i += stride) dst[i] = static_cast<unsigned char>(word);
}

// blocks of 256 threads for `units` units of work, at most 4 per SM of a B200
unsigned copy_blocks(size_t units) {
    return static_cast<unsigned>(std::min<size_t>((units + 255) / 256 + 1, 4 * 148));
}

__global__ void scale_c_kernel(double* C, int64_t ldc, int64_t m, int64_t n, double br, double bi, int cplx) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= m) return;
    for (int64_t j = blockIdx.y; j < n; j += gridDim.y) {
        if (!cplx) {
            double* cp = C + i + j * ldc;
            *cp = br == 0.0 ? 0.0 : __dmul_rn(br, *cp);
        } else {
            double* cp = C + 2 * (i + j * ldc);
            if (br == 0.0 && bi == 0.0) {
                cp[0] = 0.0;
                cp[1] = 0.0;
            } else {
                const double r = cp[0], im = cp[1];
                cp[0] = __dsub_rn(__dmul_rn(br, r), __dmul_rn(bi, im));
                cp[1] = __dadd_rn(__dmul_rn(br, im), __dmul_rn(bi, r));
            }
        }
    }
}

// Ozaki Scheme I (the reference's comparison baseline, benchmarks/ozaki1_gpu.hpp:50-75): the
// exact diagonal sums S_d, most significant first, in double-double Horner steps T = 128 T + S_d
// (scaling by 128 is exact, so a contracted multiply-add rounds as the separate operations do),
// then one ldexp by 7 (L - 1) - D_i - E_j, NaN for non-finite rows / columns. The sums are
// stored row-major (acc[d][i n + j]); a block takes a 32 x 32 tile, reads it along j and writes
// C along i through shared memory. Block (32, 8), grid (ceil(n / 32), rows of tiles strided).
__global__ void __launch_bounds__(256) oz1_horner_kernel(const int64_t* __restrict__ acc, int64_t m, int64_t n, int L,
                                                         const unsigned long long* __restrict__ maxA,
                                                         const unsigned long long* __restrict__ maxB, int tk,
                                                         double* __restrict__ C, int64_t ldc) {
    __shared__ double tile[32][33];
    const int64_t j0 = static_cast<int64_t>(blockIdx.x) * 32, plane = m * n;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t j = j0 + tx;
    const int Ej = j < n ? exponent_of(maxB[j], tk) : 0;
    for (int64_t i0 = static_cast<int64_t>(blockIdx.y) * 32; i0 < m; i0 += static_cast<int64_t>(gridDim.y) * 32) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t i = i0 + ty + 8 * r;
            if (i >= m || j >= n) continue;
            const int Di = exponent_of(maxA[i], tk);
            double hi = 0.0, lo = 0.0;
            for (int d = 0; d < L; ++d) {
                const double sd = static_cast<double>(acc[d * plane + i * n + j]);
                if (d > 0) {
                    hi *= 128.0;
                    lo *= 128.0;
                }
                const double sm = hi + sd, bb = sm - hi;
                const double err = (hi - (sm - bb)) + (sd - bb) + lo;
                hi = sm + err;
                lo = err - (hi - sm);
            }
            double v = ldexp(hi + lo, 7 * (L - 1) - Di - Ej);
            if (Di == kNonFinite || Ej == kNonFinite) v = __longlong_as_double(0x7FF8000000000000ll);
            tile[ty + 8 * r][tx] = v;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int64_t jj = j0 + ty + 8 * r, ii = i0 + tx;
            if (ii < m && jj < n) C[ii + jj * ldc] = tile[tx][ty + 8 * r];
        }
        __syncthreads();
    }
}

}  // namespace

void crt_launch_shape(CrtItem* items, int count, const Plan& plan, bool cplx, int num_sms) {
    // a block and turn: 32 rows by 8 warps' columns; up to 8 turns per block while about eight blocks per
    // SM remain in the launch
    const int L = limbs16_for(plan.s), cols = 8 * crt_cols(L, cplx);
    int64_t turns = 0;
    for (int q = 0; q < count; ++q) turns += ceil_div(items[q].m, 32) * ceil_div(items[q].n, cols);
    const int jc = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(8, turns / (8 * num_sms))));
    for (int q = 0; q < count; ++q) {
        items[q].cols = cols;
        items[q].jc = jc;
    }
}

int64_t crt_item_blocks(CrtItem& it, int64_t block0) {
    it.block0 = block0;
    it.iblocks = ceil_div(it.m, 32);
    const int64_t turns = ceil_div(it.n, it.cols);
    return it.m > 0 ? ceil_div(turns, it.jc) * it.iblocks : 0;
}

cudaError_t prepare_crt_kernels() { return crt_prepare<1>(); }

namespace {
void crt_tables(const Plan& plan, uint32_t* M16, float* qf, uint8_t (*wb)[32]) {
    CrtConst cc;
    crt_constants(plan, cc);
    std::memcpy(M16, cc.M16, sizeof cc.M16);
    std::memcpy(qf, cc.qf, sizeof cc.qf);
    for (int t = 0; t < plan.s; ++t)
        for (int b = 0; b < 4 * plan.nl; ++b) wb[b][t] = static_cast<uint8_t>(plan.W[t][b / 4] >> (8 * (b % 4)));
}
}  // namespace

void launch_crt(const CrtItem* d_items, int count, int64_t blocks, const Plan& plan, bool cplx, cudaStream_t st) {
    if (count <= 0 || blocks <= 0) return;
    CrtParams P{};
    P.items = d_items;
    P.count = count;
    P.s = plan.s;
    crt_tables(plan, P.M16, P.qf, P.wb);
    crt_dispatch<1>(limbs16_for(plan.s), P, blocks, cplx, st);
}

void launch_oz1_horner(const int64_t* acc, int64_t m, int64_t n, int L, const unsigned long long* maxA,
                       const unsigned long long* maxB, int tk, double* C, int64_t ldc, cudaStream_t st) {
    if (m <= 0 || n <= 0) return;
    dim3 grid(static_cast<unsigned>(ceil_div(n, 32)), static_cast<unsigned>(std::min<int64_t>(ceil_div(m, 32), 65535)));
    oz1_horner_kernel<<<grid, dim3(32, 8), 0, st>>>(acc, m, n, L, maxA, maxB, tk, C, ldc);
}

void launch_write_blob(const void* src, size_t bytes, void* dst, cudaStream_t st, void* zero, size_t zero_bytes) {
    const unsigned char* p = static_cast<const unsigned char*>(src);
    for (size_t off = 0; off < bytes; off += kParamBlobBytes) {
        const size_t n = std::min(kParamBlobBytes, bytes - off);
        unsigned char* d = static_cast<unsigned char*>(dst) + off;
        if (n <= 1024) write_blob_n<1024>(p + off, n, d, st, zero, zero_bytes);
        else if (n <= 4096) write_blob_n<4096>(p + off, n, d, st, zero, zero_bytes);
        else if (n <= 12288) write_blob_n<12288>(p + off, n, d, st, zero, zero_bytes);
        else write_blob_n<kParamBlobBytes>(p + off, n, d, st, zero, zero_bytes);
        zero_bytes = 0;
    }
}

void launch_sm_copy(const void* src, void* dst, size_t bytes, cudaStream_t st) {
    if (bytes == 0) return;
    const auto* s = static_cast<const unsigned char*>(src);
    auto* d = static_cast<unsigned char*>(dst);
    if (((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(d)) & 15) == 0)
        sm_copy_kernel<true><<<copy_blocks(bytes / 16), 256, 0, st>>>(s, d, bytes);
    else
        sm_copy_kernel<false><<<copy_blocks(bytes), 256, 0, st>>>(s, d, bytes);
}

void launch_fill(void* dst, unsigned char value, size_t bytes, cudaStream_t st) {
    if (bytes == 0) return;
    auto* d = static_cast<unsigned char*>(dst);
    const uint32_t word = value * 0x01010101u;
    if ((reinterpret_cast<uintptr_t>(d) & 15) == 0) fill_kernel<true><<<copy_blocks(bytes / 16), 256, 0, st>>>(d, word, bytes);
    else fill_kernel<false><<<copy_blocks(bytes), 256, 0, st>>>(d, word, bytes);
}

void launch_scale_c(double* C, int64_t ldc, int64_t m, int64_t n, const double* beta, bool cplx, cudaStream_t st) {
    if (m <= 0 || n <= 0) return;
    dim3 grid(static_cast<unsigned>(ceil_div(m, 256)), static_cast<unsigned>(std::min<int64_t>(n, 65535)));
    scale_c_kernel<<<grid, 256, 0, st>>>(C, ldc, m, n, beta[0], cplx ? beta[1] : 0.0, cplx ? 1 : 0);
}

}  // namespace oz2
