// Batched FP64 (real / complex) GEMM over a flat tile list.
//
// One launch covers many independent products of uneven shapes (symmetry
// blocks of different sizes, frequency batches): the host builds a list of
// (problem, tile_m, tile_n) entries and the grid walks it, so no CTA idles
// on an empty tile of a small block.  Operands are addressed through
// arbitrary (row, column) strides, so transposes cost nothing, and the
// reduction index k may be gathered through index arrays with a per-k scale
// (the signed row gather of a fermionic operator).
#pragma once

#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "pgx_common.cuh"
#include "pgx_internal.h"

namespace pgx {

// An operand declared Dressed<T> is stored as the operator block X (type T,
// rows a, columns b in the block's own orientation) and enters the product as
// the complex matrix X[a][b] / (z - (Eb[b] - Ea[a])): the frequency dressing of
// a Lehmann factor, computed as the tile is loaded instead of materialised.
template <typename T> struct Dressed {};
template <typename T> struct is_dressed : std::false_type {};
template <typename T> struct is_dressed<Dressed<T>> : std::true_type {};
template <typename T> struct src_t { using type = T; };
template <typename T> struct src_t<Dressed<T>> { using type = T; };
template <typename T> struct val_t { using type = T; };
template <typename T> struct val_t<Dressed<T>> { using type = cd; };

template <typename TA, typename TB, typename TC> struct GemmProblem {
    const typename src_t<TA>::type* A;
    const typename src_t<TB>::type* B;
    TC* C;
    int M, N, K;
    long sa_i, sa_k;   // A(i,k) = A[i*sa_i + k'*sa_k], k' = a_kidx ? a_kidx[k] : k
    long sb_k, sb_j;   // B(k,j) = B[k''*sb_k + j*sb_j], k'' = b_kidx ? b_kidx[k] : k
    long sc_i, sc_j;
    const int* a_kidx;
    const int* b_kidx;
    const double* kscale;  // multiplies B(k, :) when non-null
    int accumulate;        // C += A B instead of C = A B
    int conj_a;            // use conj(A) (complex A only)
    const int* a_iidx;     // row gather of A: A(i,k) uses row a_iidx[i] (nullable)
    const int* b_jidx;     // column gather of B: B(k,j) uses column b_jidx[j] (nullable)
    const double* dEa;     // dressing of the Dressed<T> operand: energies of its rows,
    const double* dEb;     // of its columns (after the gathers),
    cd dz;                 // and the frequency (or dzs[b] for batch item b when dzs is set)
    // batch of nb products with the same shapes (nb <= 0 counts as 1): item b
    // uses A + b*ba, B + b*bb, C + b*bc
    int nb;
    long ba, bb, bc;
    const cd* dzs;
    // a second output of the same strides (nullable): GEMM_CONJ the conjugate
    // of C; GEMM_CONJ_A conj(A) B and GEMM_CONJ_B A conj(B) (A and B complex),
    // which share the four real products of A B
    TC* C2;
    int mirror;
};
constexpr int GEMM_CONJ = 1, GEMM_CONJ_A = 2, GEMM_CONJ_B = 3;

// Bytes of the per-class tile index a launch_gemm_batch of nprobs problems needs.
inline size_t gemm_index_bytes(size_t nprobs) { return (nprobs + 16) * sizeof(int); }

__device__ __forceinline__ cd dress(double x, double ea, double eb, cd z) {
    const double dx = z.x - (eb - ea), t = x * recip_pos(fma(dx, dx, z.y * z.y));
    return cd{dx * t, -(z.y * t)};
}
__device__ __forceinline__ cd dress(cd x, double ea, double eb, cd z) {
    return x * inv_fast(cd{z.x - (eb - ea), z.y});
}
__device__ __forceinline__ double scale_by(double a, double s) { return a * s; }
__device__ __forceinline__ cd scale_by(cd a, double s) { return cd{a.x * s, a.y * s}; }
__device__ __forceinline__ double maybe_conj(double a, int) { return a; }
__device__ __forceinline__ cd maybe_conj(cd a, int c) { return c ? cd{a.x, -a.y} : a; }
__device__ __forceinline__ void store_c(double& dst, double v, int acc) { dst = acc ? dst + v : v; }
__device__ __forceinline__ void store_c(cd& dst, double v, int acc) {
    dst = acc ? cd{dst.x + v, dst.y} : cd{v, 0.0};
}
__device__ __forceinline__ void store_c(cd& dst, cd v, int acc) { dst = acc ? dst + v : v; }
template <typename T> __device__ __forceinline__ T zero_of();
template <> __device__ __forceinline__ double zero_of<double>() { return 0.0; }
template <> __device__ __forceinline__ cd zero_of<cd>() { return cd{0.0, 0.0}; }

constexpr int GEMM_BM = 64, GEMM_BN = 64, GEMM_THREADS = 256;

// ---- FP64 tensor-core step (mma.sync m8n8k4): D += A B for an 8 x 4 A and a
// 4 x 8 B.  Lane l holds A(l / 4, l % 4), B(l % 4, l / 4) and D(l / 4,
// 2 (l % 4) + {0, 1}).
__device__ __forceinline__ void mma_f64(double2& d, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d.x), "+d"(d.y)
        : "d"(a), "d"(b));
}
// Accumulator of one 8 x 8 tile: re (and im where an operand is complex).
struct AccR {
    double2 re;
};
struct AccC {
    double2 re, im;
};
// All four real products apart, for A B together with conj(A) B or A conj(B).
struct AccQ {
    double2 rr, ii, ri, ir;
};
__device__ __forceinline__ void mma_tile(AccQ& c, cd a, cd b) {
    mma_f64(c.rr, a.x, b.x);
    mma_f64(c.ri, a.x, b.y);
    mma_f64(c.ii, a.y, b.y);
    mma_f64(c.ir, a.y, b.x);
}
__device__ __forceinline__ void acc_zero(AccQ& c) { c.rr = c.ii = c.ri = c.ir = double2{0.0, 0.0}; }
__device__ __forceinline__ void acc_pair(const AccQ& c, int u, int mirror, cd& first, cd& second) {
    const double rr = u ? c.rr.y : c.rr.x, ii = u ? c.ii.y : c.ii.x, ri = u ? c.ri.y : c.ri.x, ir = u ? c.ir.y : c.ir.x;
    first = cd{rr - ii, ri + ir};
    second = cd{rr + ii, mirror == GEMM_CONJ_A ? ri - ir : ir - ri};
}
__device__ __forceinline__ void mma_tile(AccR& c, double a, double b) { mma_f64(c.re, a, b); }
__device__ __forceinline__ void mma_tile(AccC& c, cd a, double b) {
    mma_f64(c.re, a.x, b);
    mma_f64(c.im, a.y, b);
}
__device__ __forceinline__ void mma_tile(AccC& c, double a, cd b) {
    mma_f64(c.re, a, b.x);
    mma_f64(c.im, a, b.y);
}
__device__ __forceinline__ void mma_tile(AccC& c, cd a, cd b) {
    mma_f64(c.re, a.x, b.x);
    mma_f64(c.im, a.x, b.y);
    mma_f64(c.re, -a.y, b.y);
    mma_f64(c.im, a.y, b.x);
}
__device__ __forceinline__ void acc_zero(AccR& c) { c.re = double2{0.0, 0.0}; }
__device__ __forceinline__ void acc_zero(AccC& c) { c.re = c.im = double2{0.0, 0.0}; }
__device__ __forceinline__ double acc_at(const AccR& c, int u) { return u ? c.re.y : c.re.x; }
__device__ __forceinline__ cd acc_at(const AccC& c, int u) { return u ? cd{c.re.y, c.im.y} : cd{c.re.x, c.im.x}; }

// Element copies global -> shared without a register in between; the bytes of
// an element outside the problem are zero-filled (nothing is read).
__device__ __forceinline__ void cp_elem(double* dst, const double* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0));
}
__device__ __forceinline__ void cp_elem(cd* dst, const cd* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0));
}

// Tile shapes (BM x BN) and the rows of warps that share one (8 warps; a warp
// has BM / WR rows and BN / (8 / WR) columns, in 8 x 8 tiles of the FP64
// tensor cores).  Skinny shapes keep the products of a few anchors out of
// 64-row tiles.
__host__ __device__ constexpr int gemm_wr(int bm) { return bm <= 16 ? 1 : bm <= 48 ? 2 : bm <= 64 ? 4 : 8; }

// What bounds it: the FP64 pipe (a 64 x 64 complex tile has 16384 fused
// multiply-adds per k for 128 operand elements).  Shared memory is
// double-buffered: undressed operands go there by cp.async and dressed ones
// through registers, both issued before the current k-tile's products.  The
// leading dimensions (BM + 2 complex, BM + 4 real) put the 4 k x 4 (8) rows
// that a fragment load touches together in different banks.  Complex x complex
// 2048^3: 31.8 TFLOP/s (peak of the FP64 tensor path 37); the chi3 of Anderson
// 1+5 on 32 x 32 duplets, whose products these are: 23.3 ms with scalar FMAs
// on 4 x 4 register tiles, 17.6 ms when the products moved here.  Deeper
// k-tiles (16 for mixed types, 32 for real ones) measured no faster.
//
// QUAD: problems with GEMM_CONJ_A or GEMM_CONJ_B, in tiles of half the outputs
// (twice the accumulators each), so two complex products for the tensor work
// of one: 25 to 28 TFLOP/s of both in each of two launches side by side on the
// 7-site ring's G2, against 10.5 each one by one.
template <typename TA, typename TB, typename TC, int BM, int BN, bool QUAD>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
    gemm_tiles_kernel(const GemmProblem<TA, TB, TC>* __restrict__ probs, const int* __restrict__ tile0, int nprobs) {
    using VA = typename val_t<TA>::type;  // operand values as they enter the product
    using VB = typename val_t<TB>::type;
    constexpr bool CX = is_cd<VA>::value || is_cd<VB>::value;
    using Acc = typename std::conditional<QUAD, AccQ, typename std::conditional<CX, AccC, AccR>::type>::type;
    constexpr bool DA = is_dressed<TA>::value, DB = is_dressed<TB>::value;
    constexpr int BK = CX ? 8 : 16;
    constexpr int WR = gemm_wr(BM), WC = GEMM_THREADS / 32 / WR;
    constexpr int WM = BM / WR, WN = BN / WC, FM = WM / 8, FN = WN / 8;
    static_assert(FM * 8 * WR == BM && FN * 8 * WC == BN, "tile shape does not fit the warp grid");
    constexpr int LA = (BM * BK + GEMM_THREADS - 1) / GEMM_THREADS;
    constexpr int LB = (BN * BK + GEMM_THREADS - 1) / GEMM_THREADS;
    constexpr int LDA = BM + (is_cd<VA>::value ? 2 : 4), LDB = BN + (is_cd<VB>::value ? 2 : 4);
    __shared__ __align__(16) VA As[2][BK][LDA];
    __shared__ __align__(16) VB Bs[2][BK][LDB];

    // tile0[q] = first tile of problem q (prefix sum); find this CTA's problem
    const int tile = blockIdx.x;
    int lo = 0, hi = nprobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tile0[mid] <= tile) lo = mid;
        else hi = mid - 1;
    }
    const GemmProblem<TA, TB, TC>& p = probs[lo];
    const int tn_count = (p.N + BN - 1) / BN, per_item = ((p.M + BM - 1) / BM) * tn_count;
    const int local = tile - tile0[lo];
    const int item = local / per_item, rem = local % per_item;
    const int i0 = (rem / tn_count) * BM, j0 = (rem % tn_count) * BN;
    const auto* pA = p.A + item * p.ba;
    const auto* pB = p.B + item * p.bb;
    const int M = p.M, N = p.N, K = p.K;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int wr = warp / WC, wc = warp % WC;
    cd dz{0.0, 0.0};
    if constexpr (DA || DB) dz = p.dzs ? p.dzs[item] : p.dz;

    Acc acc[FM][FN];
#pragma unroll
    for (int a = 0; a < FM; ++a)
#pragma unroll
        for (int b = 0; b < FN; ++b) acc_zero(acc[a][b]);

    // Each thread copies the same elements of every k-tile (LA of A, LB of B);
    // their places, source pointers and row energies are set up once, since
    // recomputing them cost more issue slots than the products (18 instructions
    // per tensor instruction for a real x dressed product, and the tensor path
    // 44% busy).  Complex x complex 2048^3: 27.4 -> 31.8 TFLOP/s; the 7-site
    // ring's G2 (7^3): 386 -> 291 ms; chi3 of Anderson 1+5: 10.6 -> 8.9 ms.
    // k gathers, kscale and conj_a come with plain operands of one type only
    constexpr bool GATHER = std::is_same<TA, TB>::value;
    const bool a_reg = DA || (GATHER && p.conj_a), b_reg = DB || (GATHER && p.kscale != nullptr);
    const int *a_kidx = GATHER ? p.a_kidx : nullptr, *b_kidx = GATHER ? p.b_kidx : nullptr;
    const long sa_k = p.sa_k, sb_k = p.sb_k;
    using SA = typename src_t<TA>::type;
    using SB = typename src_t<TB>::type;
    const SA* srcA[LA];  // next element (k gathered: element k = 0 of its row)
    const SB* srcB[LB];
    int atA[LA], atB[LB];  // place in the tile
    int kA[LA], kB[LB];    // k inside the tile; beyond every K outside the problem
    SA ra[LA];
    SB rb[LB];
    double eA[DA ? LA : 1], eB[DB ? LB : 1];  // energies of the rows of A, columns of B
    double ek[DA || DB ? (DA ? LA : LB) : 1];
#pragma unroll
    for (int q = 0; q < LA; ++q) {
        const int l = tid + q * GEMM_THREADS;
        const bool fast = p.sa_i == 1;
        const int ii = fast ? l % BM : l / BK, kk = fast ? l / BM : l % BK;
        const bool in = (BM * BK % GEMM_THREADS == 0 || l < BM * BK) && i0 + ii < M;
        const long iq = !in ? 0 : p.a_iidx ? p.a_iidx[i0 + ii] : i0 + ii;
        atA[q] = kk * LDA + ii;
        kA[q] = in ? kk : 1 << 30;
        srcA[q] = pA + iq * p.sa_i + (a_kidx || !in ? 0 : kk * sa_k);
        if constexpr (DA) eA[q] = in ? p.dEa[iq] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < LB; ++q) {
        const int l = tid + q * GEMM_THREADS;
        const bool fast = p.sb_j == 1;
        const int jj = fast ? l % BN : l / BK, kk = fast ? l / BN : l % BK;
        const bool in = (BN * BK % GEMM_THREADS == 0 || l < BN * BK) && j0 + jj < N;
        const long jq = !in ? 0 : p.b_jidx ? p.b_jidx[j0 + jj] : j0 + jj;
        atB[q] = kk * LDB + jj;
        kB[q] = in ? kk : 1 << 30;
        srcB[q] = pB + jq * p.sb_j + (b_kidx || !in ? 0 : kk * sb_k);
        if constexpr (DB) eB[q] = in ? p.dEb[jq] : 0.0;
    }
    const long stepA = BK * sa_k, stepB = BK * sb_k;
    // Real operands: the gathered rows of a k-tile are looked up one k-tile
    // ahead of its loads, and a scale enters when the tile is stored, so no
    // instruction ahead of the products waits for memory: rotations of 64 models
    // of 3 to 6 bath sites 38.8 -> 26.4 ms, of the 7-site ring 2.5 -> 1.7.
    constexpr bool AHEAD = GATHER && !CX;
    int ia[AHEAD ? LA : 1], ib[AHEAD ? LB : 1];
    double sc[AHEAD ? LB : 1];
    auto look_up = [&](int k0) {
        if constexpr (AHEAD) {
            if (a_kidx) {
#pragma unroll
                for (int q = 0; q < LA; ++q) ia[q] = kA[q] < K - k0 ? a_kidx[k0 + kA[q]] : 0;
            }
            if (b_kidx) {
#pragma unroll
                for (int q = 0; q < LB; ++q) ib[q] = kB[q] < K - k0 ? b_kidx[k0 + kB[q]] : 0;
            }
        }
    };
    // issues the loads of the k-tile at k0 (buffer buf), k-tiles in order
    auto load = [&](int k0, int buf) {
        const int left = K - k0;
#pragma unroll
        for (int q = 0; q < LA; ++q) {
            if (BM * BK % GEMM_THREADS != 0 && tid + q * GEMM_THREADS >= BM * BK) continue;
            const bool in = kA[q] < left;
            const SA* src = srcA[q];
            if (a_kidx) src += AHEAD ? ia[AHEAD ? q : 0] * sa_k : in ? a_kidx[k0 + kA[q]] * sa_k : 0L;
            else srcA[q] += stepA;
            src = in ? src : pA;
            if constexpr (DA) {
                ra[q] = in ? *src : zero_of<SA>();
                ek[q] = in ? p.dEb[a_kidx ? a_kidx[k0 + kA[q]] : k0 + kA[q]] : 0.0;
            } else {
                if (a_reg) ra[q] = in ? maybe_conj(*src, 1) : zero_of<SA>();
                else cp_elem(&As[buf][0][0] + atA[q], src, in);
            }
        }
#pragma unroll
        for (int q = 0; q < LB; ++q) {
            if (BN * BK % GEMM_THREADS != 0 && tid + q * GEMM_THREADS >= BN * BK) continue;
            const bool in = kB[q] < left;
            const SB* src = srcB[q];
            if (b_kidx) src += AHEAD ? ib[AHEAD ? q : 0] * sb_k : in ? b_kidx[k0 + kB[q]] * sb_k : 0L;
            else srcB[q] += stepB;
            src = in ? src : pB;
            if constexpr (DB) {
                rb[q] = in ? *src : zero_of<SB>();
                ek[q] = in ? p.dEa[b_kidx ? b_kidx[k0 + kB[q]] : k0 + kB[q]] : 0.0;
            } else {
                if constexpr (AHEAD) {
                    if (b_reg) {
                        rb[q] = in ? *src : 0.0;
                        sc[q] = in ? p.kscale[k0 + kB[q]] : 0.0;
                    }
                } else if (b_reg) rb[q] = in ? scale_by(*src, p.kscale[k0 + kB[q]]) : zero_of<SB>();
                if (b_reg) continue;
                cp_elem(&Bs[buf][0][0] + atB[q], src, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // stores the register operands of that k-tile (dressed), then waits for its copies
    auto store = [&](int k0, int buf) {
        const int left = K - k0;
        if (a_reg) {
#pragma unroll
            for (int q = 0; q < LA; ++q) {
                if (BM * BK % GEMM_THREADS != 0 && tid + q * GEMM_THREADS >= BM * BK) continue;
                VA* at = &As[buf][0][0] + atA[q];
                if constexpr (DA) *at = kA[q] < left ? dress(ra[q], eA[q], ek[q], dz) : cd{0.0, 0.0};
                else *at = ra[q];
            }
        }
        if (b_reg) {
#pragma unroll
            for (int q = 0; q < LB; ++q) {
                if (BN * BK % GEMM_THREADS != 0 && tid + q * GEMM_THREADS >= BN * BK) continue;
                VB* at = &Bs[buf][0][0] + atB[q];
                if constexpr (DB) *at = kB[q] < left ? dress(rb[q], ek[q], eB[q], dz) : cd{0.0, 0.0};
                else if constexpr (AHEAD) *at = rb[q] * sc[q];
                else *at = rb[q];
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    };

    look_up(0);
    load(0, 0);
    look_up(BK);
    store(0, 0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK) {
        const bool more = k0 + BK < K;
        if (more) {
            load(k0 + BK, buf ^ 1);
            look_up(k0 + 2 * BK);
        }
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            VA a[FM];
            VB b[FN];
#pragma unroll
            for (int q = 0; q < FM; ++q) a[q] = As[buf][k4 + lane % 4][wr * WM + 8 * q + lane / 4];
#pragma unroll
            for (int q = 0; q < FN; ++q) b[q] = Bs[buf][k4 + lane % 4][wc * WN + 8 * q + lane / 4];
#pragma unroll
            for (int qa = 0; qa < FM; ++qa)
#pragma unroll
                for (int qb = 0; qb < FN; ++qb) mma_tile(acc[qa][qb], a[qa], b[qb]);
        }
        if (more) store(k0 + BK, buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
    TC* pC = p.C + item * p.bc;
    TC* pC2 = p.C2 ? p.C2 + item * p.bc : nullptr;
#pragma unroll
    for (int qa = 0; qa < FM; ++qa) {
        const int gi = i0 + wr * WM + 8 * qa + lane / 4;
        if (gi >= M) continue;
#pragma unroll
        for (int qb = 0; qb < FN; ++qb)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int gj = j0 + wc * WN + 8 * qb + 2 * (lane % 4) + u;
                if (gj >= N) continue;
                const long o = gi * p.sc_i + gj * p.sc_j;
                if constexpr (QUAD) {
                    cd first, second;
                    acc_pair(acc[qa][qb], u, p.mirror, first, second);
                    pC[o] = first;
                    pC2[o] = second;
                } else {
                    const auto v = acc_at(acc[qa][qb], u);
                    store_c(pC[o], v, p.accumulate);
                    if constexpr (is_cd<TC>::value)
                        if (pC2) pC2[o] = conj(tocd(v));
                }
            }
    }
}

template <typename T> struct type_tag_s {
    static const char* get() { return is_cd<T>::value ? "cd" : "double"; }
};
template <typename T> struct type_tag_s<Dressed<T>> {
    static const char* get() { return is_cd<T>::value ? "dressed<cd>" : "dressed<double>"; }
};
template <typename T> const char* type_tag() { return type_tag_s<T>::get(); }
template <typename TA, typename TB, typename TC> const char* gemm_name() {
    static const std::string n =
        std::string("gemm_tiles_kernel<") + type_tag<TA>() + ", " + type_tag<TB>() + ", " + type_tag<TC>() + ">";
    return n.c_str();
}

// Tile classes (BM x BN).  A problem takes the class that pads it least
// (ties: the larger tile); the classes other than 64x64 are used only when
// their short side covers the problem's M or N in one tile.
// The classes from GEMM_NCLS on are those of QUAD problems: 32 x 64 and 64 x 32
// (the dressed operand on the short side, where fewer elements are dressed),
// and the narrow ones.
constexpr int GEMM_NCLS = 9, GEMM_NCLS_ALL = 15;
constexpr int GEMM_CLS_M[GEMM_NCLS_ALL] = {64, 16, 128, 64, 64, 32, 48, 8, 128, 32, 64, 16, 128, 8, 128};
constexpr int GEMM_CLS_N[GEMM_NCLS_ALL] = {64, 128, 16, 32, 48, 64, 64, 128, 8, 64, 32, 128, 16, 128, 8};

template <typename TA, typename TB, typename TC> inline int gemm_quad_class(const GemmProblem<TA, TB, TC>& p) {
    int best = is_dressed<TB>::value ? 10 : 9;
    auto area = [&](int c) {
        return (long)ceil_div(p.M, GEMM_CLS_M[c]) * GEMM_CLS_M[c] * ((long)ceil_div(p.N, GEMM_CLS_N[c]) * GEMM_CLS_N[c]);
    };
    for (int c = GEMM_NCLS; c < GEMM_NCLS_ALL; ++c) {
        if ((GEMM_CLS_M[c] <= 16 && p.M > GEMM_CLS_M[c]) || (GEMM_CLS_N[c] <= 16 && p.N > GEMM_CLS_N[c])) continue;
        if (area(c) < area(best)) best = c;
    }
    return best;
}

template <typename P> inline int gemm_class(const P& p) {
    int best = 0;
    long best_area = (long)ceil_div(p.M, 64) * 64 * ((long)ceil_div(p.N, 64) * 64);
    for (int c = 1; c < GEMM_NCLS; ++c) {
        const int bm = GEMM_CLS_M[c], bn = GEMM_CLS_N[c];
        if (bm < 64 && p.M > bm) continue;
        if (bn < 64 && p.N > bn) continue;
        const long area = (long)ceil_div(p.M, bm) * bm * ((long)ceil_div(p.N, bn) * bn);
        if (area < best_area) {
            best = c;
            best_area = area;
        }
    }
    return best;
}

// ------------------------------------------------------------ tuned class choice
// A context's table of measured-fastest tile classes (pgx_autotune), keyed by
// the operand types and the (M, N) size buckets; -1 keeps the padding rule.
// The bucket bounds are the narrow classes' limits (8, 16, 32, 48), so a class
// measured at a bucket's upper bound is valid for every size in the bucket.
constexpr int GEMM_BUCKET_REP[GEMM_NBUCKET] = {8, 16, 32, 48, 64, 128, 256};
inline int gemm_bucket(int x) {
    return x <= 8 ? 0 : x <= 16 ? 1 : x <= 32 ? 2 : x <= 48 ? 3 : x <= 64 ? 4 : x <= 128 ? 5 : 6;
}
template <typename T> struct type_code { static constexpr int v = is_cd<T>::value ? 1 : 0; };
template <typename T> struct type_code<Dressed<T>> { static constexpr int v = 2 + (is_cd<T>::value ? 1 : 0); };
template <typename TA, typename TB, typename TC> constexpr int gemm_key() {
    return type_code<TA>::v * 8 + type_code<TB>::v * 2 + type_code<TC>::v;
}

inline bool gemm_class_valid(int c, int M, int N) {
    return (GEMM_CLS_M[c] >= 64 || M <= GEMM_CLS_M[c]) && (GEMM_CLS_N[c] >= 64 || N <= GEMM_CLS_N[c]);
}

template <typename TA, typename TB, typename TC> int gemm_class_for(const GemmProblem<TA, TB, TC>& p) {
    if (p.mirror >= GEMM_CONJ_A) return gemm_quad_class(p);
    const int f = forced_gemm_class();
    if (f >= 0 && gemm_class_valid(f, p.M, p.N)) return f;
    const GemmTune* t = active_tune();
    if (t) {
        const int c = t->cls[gemm_key<TA, TB, TC>()][gemm_bucket(p.M)][gemm_bucket(p.N)];
        if (c >= 0 && gemm_class_valid(c, p.M, p.N)) return c;
    }
    return gemm_class(p);
}

template <typename TA, typename TB, typename TC, int BM, int BN, bool QUAD = false>
void launch_gemm_class(const GemmProblem<TA, TB, TC>* dp, const int* d_index, size_t pb, size_t pe, int ntiles,
                       cudaStream_t st) {
    if (pe <= pb || ntiles <= 0) return;
    gemm_tiles_kernel<TA, TB, TC, BM, BN, QUAD><<<(unsigned)ntiles, GEMM_THREADS, 0, st>>>(dp + pb, d_index, (int)(pe - pb));
    check_launch("gemm_tiles_kernel");
}

// Classes of a few tiles join the 64 x 64 class, so that they need no launch of
// their own: the launches follow one another, each taking the latency of its
// longest k loop, about the same for every tile shape while the chip is nearly
// empty.  A class joins when its products are fewer tiles than a quarter of the
// SMs, and no more than twice as many of 64 x 64.  Two rotations of Anderson
// 1+5, nine launches of 8 to 34 us each before: 174 -> 78 us; the gradient of a
// Kanamori impurity, whole call: 3.75 -> 3.54 ms.  Classes that a caller's
// measurement chose are left alone.
template <typename TA, typename TB, typename TC>
void gemm_join_small(const std::vector<GemmProblem<TA, TB, TC>>& probs, std::vector<int>& cls) {
    if (forced_gemm_class() >= 0 || active_tune()) return;
    long own[GEMM_NCLS] = {}, square[GEMM_NCLS] = {};
    for (size_t q = 0; q < probs.size(); ++q) {
        const auto& g = probs[q];
        const int c = cls[q];
        if (c >= GEMM_NCLS || g.M <= 0 || g.N <= 0) continue;
        const long nb = std::max(g.nb, 1);
        own[c] += nb * ceil_div(g.M, GEMM_CLS_M[c]) * ceil_div(g.N, GEMM_CLS_N[c]);
        square[c] += nb * ceil_div(g.M, GEMM_CLS_M[0]) * ceil_div(g.N, GEMM_CLS_N[0]);
    }
    bool join[GEMM_NCLS] = {};
    int n = own[0] > 0;
    for (int c = 1; c < GEMM_NCLS; ++c) {
        join[c] = own[c] > 0 && own[c] <= 37 && square[c] <= 74;
        n += join[c];
    }
    if (n < 2) return;  // no launch fewer
    for (int& c : cls)
        if (c < GEMM_NCLS && join[c]) c = 0;
}

// Host helper: upload the problems (grouped by tile class) and, per class, the
// prefix sums of their tile counts into scratch buffers, and launch one kernel
// per tile class.  The index needs gemm_index_bytes(probs.size()) bytes.
template <typename TA, typename TB, typename TC>
void launch_gemm_batch(const std::vector<GemmProblem<TA, TB, TC>>& probs, void* d_probs, size_t probs_cap,
                       void* d_index, size_t index_cap, cudaStream_t st);

// Measures a batch for the tuner ahead of its real launch: per (M, N) bucket,
// the bucket's products run in every candidate class with each output
// redirected to its own stretch of scratch.  The inputs are read where they
// are, with the contents the real launch reads.
template <typename TA, typename TB, typename TC>
void record_gemm_batch(const std::vector<GemmProblem<TA, TB, TC>>& probs, cudaStream_t st) {
    TuneRecorder* rec = active_recorder();
    for (int mb = 0; mb < GEMM_NBUCKET; ++mb)
        for (int nb = 0; nb < GEMM_NBUCKET; ++nb) {
            std::vector<GemmProblem<TA, TB, TC>> grp;
            size_t bytes = 0;
            bool redirectable = true;
            for (const auto& g : probs) {
                if (g.mirror >= GEMM_CONJ_A) continue;  // one class rule, not tuned
                if (g.M <= 0 || g.N <= 0 || gemm_bucket(g.M) != mb || gemm_bucket(g.N) != nb) continue;
                if (g.sc_i < 0 || g.sc_j < 0 || g.bc < 0) redirectable = false;  // not laid out in scratch
                // the output's extent: last item's last element
                const long items = std::max(g.nb, 1);
                const long last = (items - 1) * g.bc + (long)(g.M - 1) * g.sc_i + (long)(g.N - 1) * g.sc_j;
                grp.push_back(g);
                grp.back().C = reinterpret_cast<TC*>(bytes);  // offset into the scratch, made a pointer below
                grp.back().C2 = nullptr;
                bytes += ((size_t)(last + 1) * sizeof(TC) + 255) & ~size_t(255);
            }
            if (grp.empty() || !redirectable) continue;
            tune_measure(*rec, gemm_key<TA, TB, TC>(), mb, nb, bytes,
                         [&grp](int cls, void* scratch, DevBuf& pb, DevBuf& ib, cudaStream_t s2) {
                             std::vector<GemmProblem<TA, TB, TC>> q = grp;
                             for (auto& g : q)
                                 g.C = reinterpret_cast<TC*>(static_cast<char*>(scratch) +
                                                             reinterpret_cast<size_t>(g.C));
                             pb.reserve(q.size() * sizeof(q[0]));
                             ib.reserve(gemm_index_bytes(q.size()));
                             forced_gemm_class() = cls;
                             launch_gemm_batch(q, pb.p, pb.bytes, ib.p, ib.bytes, s2);
                             forced_gemm_class() = -1;
                         },
                         st);
        }
}

template <typename TA, typename TB, typename TC>
void launch_gemm_batch(const std::vector<GemmProblem<TA, TB, TC>>& probs, void* d_probs, size_t probs_cap,
                       void* d_index, size_t index_cap, cudaStream_t st) {
    if (probs.empty()) return;
    if (active_recorder()) record_gemm_batch(probs, st);
    std::vector<GemmProblem<TA, TB, TC>> sorted;
    std::vector<int> index;  // per class: prefix over its problems, then the total
    size_t pstart[GEMM_NCLS_ALL + 1] = {}, istart[GEMM_NCLS_ALL] = {}, at[GEMM_NCLS_ALL];
    int ntiles[GEMM_NCLS_ALL] = {};
    long tiles[GEMM_NCLS_ALL] = {};
    std::vector<int> cls(probs.size());
    for (size_t q = 0; q < probs.size(); ++q) {
        const auto& g = probs[q];
        PGX_CHECK((std::is_same<TA, TB>::value || (!g.a_kidx && !g.b_kidx && !g.kscale && !g.conj_a)), PGX_ERR_ARG,
                  "k gathers need operands of one plain type");
        cls[q] = gemm_class_for(g);
    }
    gemm_join_small(probs, cls);
    for (size_t q = 0; q < probs.size(); ++q) {
        if (probs[q].M <= 0 || probs[q].N <= 0) cls[q] = -1;
        else ++pstart[cls[q] + 1];
    }
    for (int c = 0; c < GEMM_NCLS_ALL; ++c) {
        pstart[c + 1] += pstart[c];
        at[c] = pstart[c];
        istart[c] = pstart[c] + c;
    }
    sorted.resize(pstart[GEMM_NCLS_ALL]);
    index.resize(sorted.size() + GEMM_NCLS_ALL);
    for (size_t q = 0; q < probs.size(); ++q) {
        const int c = cls[q];
        if (c < 0) continue;
        const auto& g = probs[q];
        sorted[at[c]] = g;
        index[at[c]++ + c] = (int)tiles[c];
        tiles[c] += (long)std::max(g.nb, 1) * ceil_div(g.M, GEMM_CLS_M[c]) * ceil_div(g.N, GEMM_CLS_N[c]);
    }
    for (int c = 0; c < GEMM_NCLS_ALL; ++c) {
        PGX_CHECK(tiles[c] < (1L << 31), PGX_ERR_ARG, "gemm batch too large");
        index[pstart[c + 1] + c] = ntiles[c] = (int)tiles[c];
    }
    if (sorted.empty()) return;
    PGX_CHECK(sorted.size() * sizeof(sorted[0]) <= probs_cap, PGX_ERR_ARG, "gemm problem list overflow");
    PGX_CHECK(index.size() * sizeof(int) <= index_cap, PGX_ERR_ARG, "gemm tile index overflow");
    h2d(d_probs, sorted.data(), sorted.size() * sizeof(sorted[0]), st);
    h2d(d_index, index.data(), index.size() * sizeof(int), st);
    const auto* dp = static_cast<const GemmProblem<TA, TB, TC>*>(d_probs);
    const int* di = static_cast<const int*>(d_index);
    // real x real 2, real x complex 4, complex x complex 8 operations per product term;
    // minimum traffic: A, B and C once (C twice when accumulating)
    using VA = typename val_t<TA>::type;
    using VB = typename val_t<TB>::type;
    constexpr double mac = (is_cd<VA>::value && is_cd<VB>::value) ? 8.0
                           : (is_cd<VA>::value || is_cd<VB>::value) ? 4.0 : 2.0;
    double fl = 0.0, by = 0.0;
    for (const auto& q : sorted) {
        const double nb = std::max(q.nb, 1) * (q.mirror >= GEMM_CONJ_A ? 2.0 : 1.0);
        fl += nb * mac * q.M * (double)q.N * q.K;
        by += nb * ((double)q.M * q.K * sizeof(typename src_t<TA>::type) +
                    (double)q.K * q.N * sizeof(typename src_t<TB>::type) +
                    (q.accumulate ? 2.0 : 1.0) * q.M * (double)q.N * sizeof(TC));
    }
    ProfRange pr(gemm_name<TA, TB, TC>(), st, fl, by);
    launch_gemm_class<TA, TB, TC, 64, 64>(dp, di + istart[0], pstart[0], pstart[1], ntiles[0], st);
    launch_gemm_class<TA, TB, TC, 16, 128>(dp, di + istart[1], pstart[1], pstart[2], ntiles[1], st);
    launch_gemm_class<TA, TB, TC, 128, 16>(dp, di + istart[2], pstart[2], pstart[3], ntiles[2], st);
    launch_gemm_class<TA, TB, TC, 64, 32>(dp, di + istart[3], pstart[3], pstart[4], ntiles[3], st);
    launch_gemm_class<TA, TB, TC, 64, 48>(dp, di + istart[4], pstart[4], pstart[5], ntiles[4], st);
    launch_gemm_class<TA, TB, TC, 32, 64>(dp, di + istart[5], pstart[5], pstart[6], ntiles[5], st);
    launch_gemm_class<TA, TB, TC, 48, 64>(dp, di + istart[6], pstart[6], pstart[7], ntiles[6], st);
    launch_gemm_class<TA, TB, TC, 8, 128>(dp, di + istart[7], pstart[7], pstart[8], ntiles[7], st);
    launch_gemm_class<TA, TB, TC, 128, 8>(dp, di + istart[8], pstart[8], pstart[9], ntiles[8], st);
    // an unequal pair of operand types: a plain cd x cd product is never mirrored
    if constexpr (is_cd<VA>::value && is_cd<VB>::value && is_dressed<TA>::value != is_dressed<TB>::value &&
                  !std::is_same<TA, Dressed<cd>>::value && !std::is_same<TB, Dressed<cd>>::value) {
        launch_gemm_class<TA, TB, TC, 32, 64, true>(dp, di + istart[9], pstart[9], pstart[10], ntiles[9], st);
        launch_gemm_class<TA, TB, TC, 64, 32, true>(dp, di + istart[10], pstart[10], pstart[11], ntiles[10], st);
        launch_gemm_class<TA, TB, TC, 16, 128, true>(dp, di + istart[11], pstart[11], pstart[12], ntiles[11], st);
        launch_gemm_class<TA, TB, TC, 128, 16, true>(dp, di + istart[12], pstart[12], pstart[13], ntiles[12], st);
        launch_gemm_class<TA, TB, TC, 8, 128, true>(dp, di + istart[13], pstart[13], pstart[14], ntiles[13], st);
        launch_gemm_class<TA, TB, TC, 128, 8, true>(dp, di + istart[14], pstart[14], pstart[15], ntiles[14], st);
    } else {
        PGX_CHECK(pstart[GEMM_NCLS_ALL] == pstart[GEMM_NCLS], PGX_ERR_ARG, "mirrored product of these operand types");
    }
}

// C = A B through the int8 split scheme (pgx_ozaki.cu): S slices, plain
// strided operands (one of them may be dressed), items as in launch_gemm_batch.
struct OzWork;
template <typename TA, typename TB>
void oz_zgemm(const GemmProblem<TA, TB, cd>& g, int S, OzWork& w, cudaStream_t st);

}  // namespace pgx
