// K4, weight-anchored form of the G2 Lehmann sum.
//
// Every sub-term of TwoParticleGFPart::addMultiterm (TwoParticleGFPart.cpp:277-297)
// is a product of the matrix element M and ONE Boltzmann weight once the weight
// sums are split: -M(w2+w3) -> w2 and w3 parts, M(w1+w4) -> w1 and w4 parts, the
// resonant z1z2 term -> w1 (delta: beta w1, else -w1/D) and w3 (w3/D), the z2z3
// term -> w2 (delta: -beta w2, else w2/D) and w4 (-w4/D).  Each part only needs
// the states of its weighted ("anchor") index whose weight exceeds the anchor
// threshold; the other three indices are summed completely.  The dropped
// contribution is bounded by threshold * d * (beta/pi)^3 per chain, the same
// order as the reference's own CoefficientTolerance filter (:241, :283-297).
//
// With A(z1) = O1 / (z1 - (E2 - E1)), C(z3) = O3 / (z3 - (E4 - E3)) and H_b the
// anchor states of block b, the eight anchored sub-terms are
//   T1a  -s  w2 sum_3 O2[h,3] / (z2 - (E3 - E2h)) [C(z3) X4 A(z1)[:,h]]_3
//   T1b  -s  w3 sum_2 O2[2,h] / (z2 - (E3h - E2)) [C(z3)[h,:] X4 A(z1)]_2
//   T2a   s  w1 sum_4 X4[4,h] / (Z - (E4 - E1h))  [A(z1)[h,:] O2 C(z3)]_4
//   T2b   s  w4 sum_1 X4[h,1] / (Z - (E4h - E1))  [A(z1) O2 C(z3)[:,h]]_1
//   T3a   s  sum_3 [A(z1)[h,:] O2]_3 [C(z3) X4[:,h]]_3 (delta ? beta w1 : -w1/D)
//   T3b   s  sum_1 [A(z1) O2[:,h]]_1 [C(z3)[h,:] X4]_1 (delta ? 0 : w3/D)
//   T4a   s  sum_4 [O2[h,:] C(z3)]_4 [X4 A(z1)[:,h]]_4 (delta ? -beta w2 : w2/D)
//   T4b   s  sum_2 [O2 C(z3)[:,h]]_2 [X4[h,:] A(z1)]_2 (delta ? 0 : -w4/D)
// (Z = z1+z2+z3, D = s - (E_b - E_a) with s = z1+z2 for T3 and z2+z3 for T4).
// Where every state of both blocks is an anchor, T3a and T3b are one term with
// (w3 - w1)/D, and T4a and T4b one with (w2 - w4)/D: of nearly equal levels the
// weights cancel before the division by a small D, not between two sums whose
// rounding it has enlarged.
// Stages, each one launch for a batch of chains: anchored products per
// frequency (gather GEMMs); products per (z1, z3) stacked into GEMMs over all
// anchors; contractions of classes of triples as products (contract_gemm_kernel,
// resonant delta test in FP64).  A(z1) and C(z3) are never stored: the GEMM
// tile loads dress O1 and O3 with the frequency as they read them.

#include <algorithm>
#include <array>
#include <iterator>
#include <map>
#include <limits>
#include <tuple>
#include <unordered_map>

#include "pgx_common.cuh"
#include "pgx_g2plan.h"
#include "pgx_gemm.cuh"
#include "pgx_internal.h"

namespace pgx {

namespace {

struct DTerm {
    const void* VA;
    long a1, a3, ah, ak;
    const void* VB;
    long b1, b3, bh, bk;
    const double *Ek, *Eh, *wh;
    const double* wk;     // weights of the k states where they enter too (T3, T4 over every state), else null
    const int* hot;       // anchor states (inner indices) of the anchor block
    const int* gi1;       // per group: index of z1 in the plan
    const int* gi3;       // per group: index of z3 in the plan
    int nh, nk;
    int va_cplx, vb_cplx; // operand element types
    int va_hstate, vb_hstate;  // h stride applies to the anchor's state index instead of its position
    int use_delta;
    double sgn, cdelta, cnum, cwk, pref;
    // host side only: the plan and the frequency sum (0: z2, 1: z1+z2+z3,
    // 2: z1+z2, 3: z2+z3) of the sub-term
    int plan, sidx;
};

__device__ __forceinline__ cd load_v(const void* p, int cplx, long idx) {
    return cplx ? static_cast<const cd*>(p)[idx] : cd{static_cast<const double*>(p)[idx], 0.0};
}

// ---- contractions as products
// For one sub-term, the (z1, z3) groups of a plan whose triples carry the same
// list of frequency sums s_j form a class.  Over a class the contraction is a
// complex product
//   out[t(g, j)] += pref * sum_{h, k} AB[g, (h, k)] K[(h, k), j]
// with AB[g, (h, k)] = VA(g, h, k) VB(g, h, k) (the two anchored operand
// arrays, multiplied as the tile is loaded) and the Lehmann kernel
//   K[(h, k), j] = delta ? cdelta beta w_h : (cnum w_h + cwk w_k) / (s_j - sgn (E_k - E_h)),
// delta = |s_j - sgn (E_k - E_h)| <= PoleResolution (FP64, the reference's
// rule for resonant terms).  K is formed once per tile element and used by
// every row of the tile; the rows of a T1 class are all (z1, z3) groups, those
// of T2, T3, T4 classes the groups with equal z1 + z3, z1 or z3.  A work item
// is one tile of rows of a class over a range of anchors; items of the same
// outputs add their results with atomics.
struct CItem {
    int cls, row0, h0, h1;
};

constexpr int CG_THREADS = 128, CG_BK_MAX = 16;  // the latter: k's of a tile
// of its four warps, how many split the rows; the others split the k's of a tile
__host__ __device__ constexpr int cg_wr(int bm) { return bm >= 32 ? 4 : bm == 16 ? 2 : 1; }

// One CTA per work item: BM rows x BN columns in 8 x 8 tiles of the FP64
// tensor cores (mma_tile).  The next k-tile's operand loads are issued into
// registers before the current tile's products.  What bounds it: for 64-row
// classes the FP64 pipe, on the products and a tenth of them again to form the
// operands; for the small ones the latency of the loads, which is why their
// warps split the k's.  Anderson 1+5, 16^3: 2.2 ms of
// launches one after another with scalar FMAs, 1.1 together so; a plaquette 8^3,
// every state an anchor: 0.67 and 0.12 ms.
template <int BM, int BN>
__global__ void __launch_bounds__(CG_THREADS, 3)
    contract_gemm_kernel(const DTerm* __restrict__ terms, const CClass* __restrict__ classes,
                         const CItem* __restrict__ items, double beta, double tol2, cd* __restrict__ out) {
    constexpr int NT = CG_THREADS;
    constexpr int WR = cg_wr(BM), WK = 4 / WR, FM = BM / 8 / WR, FN = BN / 8;
    static_assert(FM * 8 * WR == BM && FN * 8 == BN, "tile shape does not fit the warps");
    // k-tile depth: two buffers within 48 KB
    constexpr int CG_BK = BM >= 64 ? CG_BK_MAX / 2 : CG_BK_MAX;
    constexpr int LA = (BM * CG_BK + NT - 1) / NT, LB = (BN * CG_BK + NT - 1) / NT;
    __shared__ __align__(16) cd As[2][CG_BK][BM + 2];
    __shared__ __align__(16) cd Bs[2][CG_BK][BN + 2];
    __shared__ cd s_s[BN];
    __shared__ long s_oa[BM], s_ob[BM];
    __shared__ DTerm s_term;  // the sub-term's descriptor, read once per CTA
    const CItem it = items[blockIdx.x];
    const CClass cc = classes[it.cls];
    const DTerm& d = s_term;
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32, wr = warp % WR, wk = warp / WR;
    if (tid == 0) s_term = terms[cc.term];
    __syncthreads();
    const int nrows = min(BM, cc.nrows - it.row0);
    for (int j = tid; j < BN; j += NT) s_s[j] = j < cc.ncols ? cc.s[j] : cd{0.0, 0.0};
    for (int r = tid; r < BM; r += NT) {
        long oa = 0, ob = 0;
        if (r < nrows) {
            const int g = cc.rows[it.row0 + r];
            const long i1 = d.gi1[g], i3 = d.gi3[g];
            oa = i1 * d.a1 + i3 * d.a3;
            ob = i1 * d.b1 + i3 * d.b3;
        }
        s_oa[r] = oa;
        s_ob[r] = ob;
    }
    AccC acc[FM][FN];
#pragma unroll
    for (int a = 0; a < FM; ++a)
#pragma unroll
        for (int b = 0; b < FN; ++b) acc_zero(acc[a][b]);
    __syncthreads();

    const int nk = d.nk;
    const int ktiles = (nk + CG_BK - 1) / CG_BK;
    const long nsteps = (long)(it.h1 - it.h0) * ktiles;
    // Operands of step q (anchor h0 + q / ktiles, k-tile q % ktiles): fetch()
    // issues the global loads of the raw values into registers before the
    // current step's products; finish() forms VA VB and the Lehmann kernel from
    // them and stores the tiles after the products, so the loads' latency is
    // covered by the inner loop instead of stalling ahead of it.
    cd rx[LA], ry[LA];
    double rek[LB], rwk[LB];
    double r_eh = 0.0, r_w = 0.0;
    auto fetch = [&](long q) {
        const int h = it.h0 + (int)(q / ktiles), k0 = (int)(q % ktiles) * CG_BK;
        const int hs = d.hot[h];
        const long oah = (long)(d.va_hstate ? hs : h) * d.ah, obh = (long)(d.vb_hstate ? hs : h) * d.bh;
#pragma unroll
        for (int u = 0; u < LA; ++u) {
            const int l = tid + u * NT;
            cd x{0.0, 0.0}, y{0.0, 0.0};
            if (l < BM * CG_BK) {
                const int r = l / CG_BK, kk = l % CG_BK, k = k0 + kk;
                if (r < nrows && k < nk) {
                    x = load_v(d.VA, d.va_cplx, s_oa[r] + oah + (long)k * d.ak);
                    y = load_v(d.VB, d.vb_cplx, s_ob[r] + obh + (long)k * d.bk);
                }
            }
            rx[u] = x;
            ry[u] = y;
        }
        r_eh = d.Eh[hs];
        r_w = d.wh[hs];
#pragma unroll
        for (int u = 0; u < LB; ++u) {
            const int l = tid + u * NT;
            double ek = 0.0, wk = 0.0;
            if (l < BN * CG_BK) {
                const int k = k0 + l / BN;
                if (k < nk) {
                    ek = d.Ek[k];
                    if (d.wk) wk = d.wk[k];
                }
            }
            rek[u] = ek;
            rwk[u] = d.cwk * wk;
        }
    };
    auto finish = [&](long q, int buf) {
        const int k0 = (int)(q % ktiles) * CG_BK;
#pragma unroll
        for (int u = 0; u < LA; ++u) {
            const int l = tid + u * NT;
            if (l < BM * CG_BK) As[buf][l % CG_BK][l / CG_BK] = rx[u] * ry[u];
        }
        const double cw = d.cnum * r_w, cdl = d.cdelta * beta * r_w;
#pragma unroll
        for (int u = 0; u < LB; ++u) {
            const int l = tid + u * NT;
            if (l < BN * CG_BK) {
                const int kk = l / BN, j = l % BN, k = k0 + kk;
                cd v{0.0, 0.0};
                if (k < nk && j < cc.ncols) {
                    const cd sv = s_s[j];
                    const double dx = sv.x - d.sgn * (rek[u] - r_eh);
                    const double m2 = fma(dx, dx, sv.y * sv.y);
                    if (d.use_delta && m2 <= tol2) {
                        v = cd{cdl, 0.0};
                    } else {
                        const double rr = (cw + rwk[u]) * recip_pos(m2);
                        v = cd{dx * rr, -sv.y * rr};
                    }
                }
                Bs[buf][kk][j] = v;
            }
        }
    };
    if (nsteps > 0) {
        fetch(0);
        finish(0, 0);
    }
    __syncthreads();
    int buf = 0;
    for (long q = 0; q < nsteps; ++q) {
        const bool more = q + 1 < nsteps;
        if (more) fetch(q + 1);
#pragma unroll
        for (int k4 = 0; k4 < CG_BK; k4 += 4 * WK) {
            const int kk = k4 + 4 * wk + lane % 4;
            cd a[FM], b[FN];
#pragma unroll
            for (int u = 0; u < FM; ++u) a[u] = As[buf][kk][8 * (wr * FM + u) + lane / 4];
#pragma unroll
            for (int u = 0; u < FN; ++u) b[u] = Bs[buf][kk][8 * u + lane / 4];
#pragma unroll
            for (int qa = 0; qa < FM; ++qa)
#pragma unroll
                for (int qb = 0; qb < FN; ++qb) mma_tile(acc[qa][qb], a[qa], b[qb]);
        }
        if (more) finish(q + 1, buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int qa = 0; qa < FM; ++qa) {
        const int r = 8 * (wr * FM + qa) + lane / 4;
        if (r >= nrows) continue;
#pragma unroll
        for (int qb = 0; qb < FN; ++qb)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j = 8 * qb + 2 * (lane % 4) + u;
                if (j >= cc.ncols) continue;
                const int t = cc.slots[(long)(it.row0 + r) * cc.ncols + j];
                const cd v = acc_at(acc[qa][qb], u);
                if (t >= 0 && (v.x != 0.0 || v.y != 0.0)) {
                    atomicAdd(&out[t].x, d.pref * v.x);
                    atomicAdd(&out[t].y, d.pref * v.y);
                }
            }
    }
}

// Column widths of the contraction tiles (at most CG_BN_MAX).
constexpr int CG_NBN = 4;
constexpr int CG_BNS[CG_NBN] = {8, 16, 24, 32};

template <int BM, int BN>
void launch_contract_t(unsigned n, cudaStream_t st, const DTerm* t, const CClass* c, const CItem* i, double beta,
                       double tol2, cd* out) {
    contract_gemm_kernel<BM, BN><<<n, CG_THREADS, 0, st>>>(t, c, i, beta, tol2, out);
}

template <int BM>
void launch_contract_m(int BN, unsigned n, cudaStream_t st, const DTerm* t, const CClass* c, const CItem* i,
                       double beta, double tol2, cd* out) {
    if (BN == 8) launch_contract_t<BM, 8>(n, st, t, c, i, beta, tol2, out);
    else if (BN == 16) launch_contract_t<BM, 16>(n, st, t, c, i, beta, tol2, out);
    else if (BN == 24) launch_contract_t<BM, 24>(n, st, t, c, i, beta, tol2, out);
    else launch_contract_t<BM, 32>(n, st, t, c, i, beta, tol2, out);
}

// Row-tile heights of the contraction (a class takes the smallest that holds
// its rows, 64-row tiles above 32 rows).
constexpr int CG_NBM = 5;
constexpr int CG_BMS[CG_NBM] = {8, 16, 24, 32, 64};

void launch_contract(int BM, int BN, unsigned n, cudaStream_t st, const DTerm* t, const CClass* c, const CItem* i,
                     double beta, double tol2, cd* out) {
    switch (BM) {
        case 8: launch_contract_m<8>(BN, n, st, t, c, i, beta, tol2, out); break;
        case 16: launch_contract_m<16>(BN, n, st, t, c, i, beta, tol2, out); break;
        case 24: launch_contract_m<24>(BN, n, st, t, c, i, beta, tol2, out); break;
        case 32: launch_contract_m<32>(BN, n, st, t, c, i, beta, tol2, out); break;
        default: launch_contract_m<64>(BN, n, st, t, c, i, beta, tol2, out); break;
    }
}

char* upload(const Blob& blob, DevBuf& buf, cudaStream_t st) {
    buf.reserve(std::max<size_t>(blob.h.size(), 16));
    if (!blob.h.empty()) h2d(buf.p, blob.h.data(), blob.h.size(), st);
    return buf.as<char>();
}

// The plans of a call.  Their classes are built on first use, while the first
// batch's products run.
struct Plans {
    std::vector<APlan> list;
    std::vector<PermIndex> perm;
    std::vector<int> perm_of;  // plan -> permutation
    bool have_classes = false;
    void upload_groups(const Blob& blob, DevBuf& buf, cudaStream_t st) {
        char* base = upload(blob, buf, st);
        for (APlan& pl : list) {
            rebase(pl.dZ1, base);
            rebase(pl.dZ3, base);
            rebase(pl.dgi1, base);
            rebase(pl.dgi3, base);
        }
    }
    void classes(DevBuf& buf, cudaStream_t st) {
        if (have_classes) return;
        have_classes = true;
        for (PermIndex& ix : perm) number_sums(ix);
        Blob blob;
        for (size_t i = 0; i < list.size(); ++i)
            for (int k = 0; k < 4; ++k) build_classes(list[i], k, perm[perm_of[i]], blob);
        char* base = upload(blob, buf, st);
        for (APlan& pl : list)
            for (auto& cls : pl.cls)
                for (CClass& c : cls) {
                    rebase(c.s, base);
                    rebase(c.rows, base);
                    rebase(c.slots, base);
                }
    }
};

// Workspace of one chain inside a batch (element offsets into one cd pool).
struct ChainWs {
    long Lc, Lr, Pr, Pc, Rho, Qc, Rr, Rc, V1a, V1b, V2a, V2b, end;
};

// Frequency dressing of a Lehmann factor: the operator block (rows in block
// Sa, columns in Sb) divided elementwise by z - (E_Sb - E_Sa), with z taken
// per batch item from the plan's frequency list.
struct Dress {
    const double *Ea, *Eb;
    const cd* z;
};

// One product per frequency of a list (nb items): only the output moves, by
// bc elements per item; the dressed operand takes the item's frequency.
template <typename TA, typename TB>
GemmProblem<TA, TB, cd> gp(const typename src_t<TA>::type* A, long sai, long sak, const typename src_t<TB>::type* B,
                           long sbk, long sbj, cd* C, long sci, int M, int N, int K, const int* aii, const int* bjj,
                           Dress dr, int nb, long bc, long scj = 1) {
    GemmProblem<TA, TB, cd> g{};
    g.A = A;
    g.B = B;
    g.C = C;
    g.M = M;
    g.N = N;
    g.K = K;
    g.sa_i = sai;
    g.sa_k = sak;
    g.sb_k = sbk;
    g.sb_j = sbj;
    g.sc_i = sci;
    g.sc_j = scj;
    g.a_iidx = aii;
    g.b_jidx = bjj;
    g.dEa = dr.Ea;
    g.dEb = dr.Eb;
    g.dzs = dr.z;
    g.nb = nb;
    g.bc = bc;
    return g;
}

}  // namespace

template <typename T>
static void run_batch(pgx_ctx* c, const std::vector<int>& idx, const std::vector<int>& bplan,
                      const std::vector<ChainWs>& wsl, const pgx_g2_part* parts, Plans& plans,
                      const std::vector<std::array<int, 4>>& rs, cd* pool, const int* d_hot,
                      const std::vector<long>& hot_off, double pole_res, int split, const std::vector<int>& bdig,
                      std::vector<cudaEvent_t>* gemm_ev, cd* d_out) {
    Problem& P = c->P;
    cudaStream_t st = c->stream;
    constexpr bool TC = is_cd<T>::value;
    // ---- anchored products per frequency and stacked products per (z1, z3);
    // A1(z1) = O1 / (z1 - (E2 - E1)) and C3(z3) = O3 / (z3 - (E4 - E3)) are
    // dressed inside the GEMM tile loads (Dressed<T> operands)
    using DT = Dressed<T>;
    std::vector<GemmProblem<T, DT, cd>> pa;   // operator x dressed
    std::vector<GemmProblem<DT, T, cd>> pb;   // dressed x operator
    std::vector<GemmProblem<DT, cd, cd>> pc;  // dressed x stacked anchors (per z1 or z3)
    std::vector<GemmProblem<cd, DT, cd>> pd;  // stacked anchors x dressed
    // digits of each split product: those of its anchor block (bdig)
    std::vector<int> pa_d, pb_d, pc_d, pd_d;
    auto push = [&](auto& list, std::vector<int>& digs, int anchor_block, const auto& prob) {
        list.push_back(prob);
        digs.push_back(bdig.empty() ? split : bdig[anchor_block]);
    };
    for (size_t j = 0; j < idx.size(); ++j) {
        const int q = idx[j];
        const pgx_g2_part& g = parts[q];
        const APlan& pl = plans.list[bplan[j]];
        const ChainWs& w = wsl[j];
        const int S1 = g.block[0], S2 = g.block[1], S3 = g.block[2], S4 = g.block[3];
        const int d1 = P.dims[S1], d2 = P.dims[S2], d3 = P.dims[S3], d4 = P.dims[S4];
        const int r1 = rs[q][0], r2 = rs[q][1], r3 = rs[q][2], r4 = rs[q][3];
        const int N1 = (int)pl.Z1.size(), N3 = (int)pl.Z3.size();
        const Operator &o1 = P.ops[g.op[0]], &o2 = P.ops[g.op[1]], &o3 = P.ops[g.op[2]], &o4 = P.ops[g.op[3]];
        const T* O1 = o1.mat.as<T>() + o1.parts[o1.by_left[S1]].off;
        const T* O2 = o2.mat.as<T>() + o2.parts[o2.by_left[S2]].off;
        const T* O3 = o3.mat.as<T>() + o3.parts[o3.by_left[S3]].off;
        const T* X4 = o4.mat.as<T>() + o4.parts[o4.by_left[S4]].off;
        const double *E1 = P.d_E + P.eoff[S1], *E2 = P.d_E + P.eoff[S2], *E3 = P.d_E + P.eoff[S3],
                     *E4 = P.d_E + P.eoff[S4];
        const int *H1 = d_hot + hot_off[S1], *H2 = d_hot + hot_off[S2], *H3 = d_hot + hot_off[S3], *H4 = d_hot + hot_off[S4];
        const Dress A1{E1, E2, pl.dZ1};  // A1(z1) = O1 dressed with z1: d1 x d2, row-major
        const Dress C3{E3, E4, pl.dZ3};  // C3(z3) = O3 dressed with z3: d3 x d4, row-major
        // A product over z3 covers the conjugate pairs of Z3 with one problem
        // for both halves (the product with the conjugate z3 is the second
        // output: the conjugate itself where the other factor is real, else
        // conj(A) B or A conj(B), which share the real products of A B), and
        // the unpaired z3 with another.  With z1 taken above the axis this
        // leaves a quarter of the real products of all (z1, z3).  7-site ring 7^3:
        // 633 -> 391 ms; the 8-site ring's largest chain, 16^3, split products:
        // 159 -> 93 ms.
        const int np3 = pl.n3p, rest3 = N3 - 2 * np3;
        auto over_items = [&](auto& list, std::vector<int>& digs, int anchor_block, auto prob, int mirror) {
            if (np3 > 0) {
                auto a = prob;
                a.nb = np3;
                a.C2 = prob.C + np3 * prob.bc;
                a.mirror = mirror;
                push(list, digs, anchor_block, a);
            }
            if (rest3 > 0) {
                prob.nb = rest3;
                prob.C += 2 * np3 * prob.bc;
                prob.dzs += 2 * np3;
                push(list, digs, anchor_block, prob);
            }
        };
        auto over_rows = [&](auto& list, std::vector<int>& digs, int anchor_block, auto prob, int r, int mirror) {
            if (np3 > 0) {
                auto a = prob;
                a.M = np3 * r;
                a.C2 = prob.C + (long)np3 * r * prob.sc_i;
                a.mirror = mirror;
                push(list, digs, anchor_block, a);
            }
            if (rest3 > 0) {
                prob.M = rest3 * r;
                prob.A += 2L * np3 * r * prob.sa_i;
                prob.C += 2L * np3 * r * prob.sc_i;
                push(list, digs, anchor_block, prob);
            }
        };
        auto over_cols = [&](auto& list, std::vector<int>& digs, int anchor_block, auto prob, int r, int mirror) {
            if (np3 > 0) {
                auto a = prob;
                a.N = np3 * r;
                a.C2 = prob.C + (long)np3 * r * prob.sc_j;
                a.mirror = mirror;
                push(list, digs, anchor_block, a);
            }
            if (rest3 > 0) {
                prob.N = rest3 * r;
                prob.B += 2L * np3 * r * prob.sb_j;
                prob.C += 2L * np3 * r * prob.sc_j;
                push(list, digs, anchor_block, prob);
            }
        };
        // T3a and T3b, T4a and T4b as one term each (split products keep them
        // apart: their digits follow the weights of one block)
        const bool all13 = !split && r1 == d1 && r3 == d3, all24 = !split && r2 == d2 && r4 == d4;
        // anchored products, one item per z1 (or z3)
        // outputs that the contractions read along k are stored k-contiguous
        if (r2) push(pa, pa_d, S2, gp<T, DT>(X4, d1, 1, O1, d2, 1, pool + w.Lc, 1, d4, r2, d1, nullptr, H2, A1, N1,
                                       (long)r2 * d4, d4));                               // Lc = X4 A1[:,H2]: [(i1,h)][k]
        if (r4 && !all24) push(pa, pa_d, S4, gp<T, DT>(X4, d1, 1, O1, d2, 1, pool + w.Lr, d2, r4, d2, d1, H4, nullptr, A1, N1,
                                       (long)r4 * d2));                                   // Lr = X4[H4,:] A1
        if (r1) push(pb, pb_d, S1, gp<DT, T>(O1, d2, 1, O2, d3, 1, pool + w.Pr, d3, r1, d3, d2, H1, nullptr, A1, N1,
                                       (long)r1 * d3));                                   // Pr = A1[H1,:] O2
        if (r3 && !all13) push(pb, pb_d, S3, gp<DT, T>(O1, d2, 1, O2, d3, 1, pool + w.Pc, 1, d1, r3, d2, nullptr, H3, A1, N1,
                                       (long)d1 * r3, d1));                               // Pc = A1 O2[:,H3]: [i1][h][k]
        if (r3) over_items(pb, pb_d, S3, gp<DT, T>(O3, d4, 1, X4, d1, 1, pool + w.Rho, d1, r3, d1, d4, H3, nullptr, C3, N3,
                                             (long)r3 * d1), GEMM_CONJ);                   // rho = C3[H3,:] X4
        if (r1) over_items(pb, pb_d, S1, gp<DT, T>(O3, d4, 1, X4, d1, 1, pool + w.Qc, 1, d3, r1, d4, nullptr, H1, C3, N3,
                                             (long)d3 * r1, d3), GEMM_CONJ);               // Qc = C3 X4[:,H1]: [i3][h][k]
        if (r2) over_items(pa, pa_d, S2, gp<T, DT>(O2, d3, 1, O3, d4, 1, pool + w.Rr, d4, r2, d4, d3, H2, nullptr, C3, N3,
                                             (long)r2 * d4), GEMM_CONJ);                   // Rr = O2[H2,:] C3
        if (r4) over_items(pa, pa_d, S4, gp<T, DT>(O2, d3, 1, O3, d4, 1, pool + w.Rc, 1, d2, r4, d3, nullptr, H4, C3, N3,
                                             (long)r4 * d2, d2), GEMM_CONJ);               // Rc = O2 C3[:,H4]: [(i3,h)][k]
        // products over (z1, z3): anchors of all frequencies stacked as columns / rows
        if (r2) over_items(pc, pc_d, S2, gp<DT, cd>(O3, d4, 1, pool + w.Lc, 1, d4, pool + w.V1a, 1, d3, N1 * r2, d4, nullptr,
                                              nullptr, C3, N3, (long)d3 * N1 * r2, d3),
                           GEMM_CONJ_A);                                                   // V1a = C3 LcAll: [i3][(i1,h)][k]
        if (r1) over_items(pd, pd_d, S1, gp<cd, DT>(pool + w.Pr, d3, 1, O3, d4, 1, pool + w.V2a, d4, N1 * r1, d4, d3, nullptr,
                                              nullptr, C3, N3, (long)N1 * r1 * d4),
                           GEMM_CONJ_B);                                                   // V2a = PrAll C3
        if (r3) over_rows(pd, pd_d, S3, gp<cd, DT>(pool + w.Rho, d1, 1, O1, d2, 1, pool + w.V1b, d2, N3 * r3, d2, d1, nullptr,
                                             nullptr, A1, N1, (long)N3 * r3 * d2),
                          r3, GEMM_CONJ_A);                                                // V1b = rhoAll A1
        if (r4) over_cols(pc, pc_d, S4, gp<DT, cd>(O1, d2, 1, pool + w.Rc, 1, d2, pool + w.V2b, 1, d1, N3 * r4, d2, nullptr,
                                             nullptr, A1, N1, (long)d1 * N3 * r4, d1),
                          r4, GEMM_CONJ_B);                                                // V2b = A1 RcAll: [i1][(i3,h)][k]
    }
    // descriptor buffers: one region per product list, sized once for the
    // largest list before any launch, so that lists on different streams do
    // not share one
    const long nprob = std::max<long>(1, (long)std::max({pa.size(), pb.size(), pc.size(), pd.size()}));
    const size_t preg = ((size_t)nprob * sizeof(GemmProblem<cd, cd, cd>) + 255) & ~size_t(255);
    const size_t ireg = (gemm_index_bytes(nprob) + 255) & ~size_t(255);
    c->scratch[7].reserve(4 * preg);
    c->scratch[8].reserve(4 * ireg);
    auto launch_on = [&](auto& probs, int region, cudaStream_t s2) {
        if (probs.empty()) return;
        launch_gemm_batch(probs, c->scratch[7].as<char>() + region * preg, preg, c->scratch[8].as<char>() + region * ireg,
                          ireg, s2);
    };
    // The stacked products read Lc, Pr, rho and Rc written by the first two
    // lists.  With `split` slices, products of at least g2_split_min_macs
    // complex multiply-adds (default 1e9) go to the int8 tensor cores: smaller
    // ones, such as every product of a 400-state block, run faster on the FP64
    // tiles than their digit preparation and 128 x 256 tile padding allow.
    // Complex Hamiltonians keep the anchored products in FP64.
    auto launch_split = [&](auto& probs, const std::vector<int>& digs, int region) {
        std::remove_reference_t<decltype(probs)> rest;
        for (size_t i = 0; i < probs.size(); ++i) {
            const auto& g = probs[i];
            const double macs = (double)g.M * g.N * g.K * std::max(g.nb, 1) * (g.C2 ? 2.0 : 1.0);
            if (macs < c->g2_split_min_macs) {
                rest.push_back(g);
                continue;
            }
            oz_zgemm(g, digs[i], c->oz, st);
        }
        launch_on(rest, region, st);
    };
    auto mark = [&]() {
        if (!gemm_ev) return;
        gemm_ev->push_back(c->prof.event());
        PGX_CUDA(cudaEventRecord(gemm_ev->back(), st));
    };
    mark();
    if (gemm_ev) {
        auto count = [&](const auto& list) {
            for (const auto& g : list) c->g2t.gemm_flops += (g.C2 ? 16.0 : 8.0) * g.nb * g.M * g.N * (double)g.K;
        };
        count(pc);
        count(pd);
    }
    if (split) {  // the split products share one workspace: one stream
        if constexpr (TC) {
            launch_on(pa, 0, st);
            launch_on(pb, 1, st);
        } else {
            launch_split(pa, pa_d, 0);
            launch_split(pb, pb_d, 1);
        }
        launch_split(pc, pc_d, 2);
        launch_split(pd, pd_d, 3);
    } else {
        // pa and pb are independent, and so are pc and pd (each needs both of
        // the first pair): each pair runs on two side streams at once
        ensure_side_streams(c);
        cudaStream_t s0 = c->aux[0], s1 = c->aux[1];
        PGX_CUDA(cudaEventRecord(c->fork, st));
        PGX_CUDA(cudaStreamWaitEvent(s0, c->fork, 0));
        PGX_CUDA(cudaStreamWaitEvent(s1, c->fork, 0));
        SideJoin join(c, st, 2);  // st waits for both side streams on every exit
        launch_on(pa, 0, s0);
        launch_on(pb, 1, s1);
        PGX_CUDA(cudaEventRecord(c->join[0], s0));
        PGX_CUDA(cudaEventRecord(c->join[1], s1));
        PGX_CUDA(cudaStreamWaitEvent(s0, c->join[1], 0));
        PGX_CUDA(cudaStreamWaitEvent(s1, c->join[0], 0));
        launch_on(pc, 2, s0);
        launch_on(pd, 3, s1);
    }
    mark();
    plans.classes(c->scratch[1], st);
    // ---- contractions per triple
    std::vector<DTerm> dt;
    for (size_t j = 0; j < idx.size(); ++j) {
        const int q = idx[j];
        const pgx_g2_part& g = parts[q];
        const APlan& pl = plans.list[bplan[j]];
        const ChainWs& w = wsl[j];
        const int S[4] = {g.block[0], g.block[1], g.block[2], g.block[3]};
        const int d1 = P.dims[S[0]], d2 = P.dims[S[1]], d3 = P.dims[S[2]], d4 = P.dims[S[3]];
        const int r1 = rs[q][0], r2 = rs[q][1], r3 = rs[q][2], r4 = rs[q][3];
        const bool all13 = !split && r1 == d1 && r3 == d3, all24 = !split && r2 == d2 && r4 == d4;
        const long N1 = (long)pl.Z1.size(), N3 = (long)pl.Z3.size();
        const Operator &o2 = P.ops[g.op[1]], &o4 = P.ops[g.op[3]];
        const T* O2 = o2.mat.as<T>() + o2.parts[o2.by_left[S[1]]].off;
        const T* X4 = o4.mat.as<T>() + o4.parts[o4.by_left[S[3]]].off;
        const double* E[4];
        const double* W[4];
        for (int k = 0; k < 4; ++k) {
            E[k] = P.d_E + P.eoff[S[k]];
            W[k] = P.d_w + P.eoff[S[k]];
        }
        const double sign = g.sign;
        auto base = [&](int anchor, int nh, int nk, int kb, double sgn, int sidx, int use_delta, double cd_, double cn,
                        double pref) {
            DTerm d{};
            d.Ek = E[kb];
            d.Eh = E[anchor];
            d.wh = W[anchor];
            d.hot = d_hot + hot_off[S[anchor]];
            d.nh = nh;
            d.nk = nk;
            d.gi1 = pl.dgi1;
            d.gi3 = pl.dgi3;
            d.plan = bplan[j];
            d.sidx = sidx;
            d.sgn = sgn;
            d.use_delta = use_delta;
            d.cdelta = cd_;
            d.cnum = cn;
            d.pref = pref;
            return d;
        };
        const int opc = TC ? 1 : 0;
        if (r2) {  // T1a: va = O2[h,k] (state h), vb = V1a[i3][(i1,h)][k]
            DTerm d = base(1, r2, d3, 2, +1.0, 0, 0, 0.0, 1.0, -sign);
            d.VA = O2; d.va_cplx = opc; d.va_hstate = 1; d.ah = d3; d.ak = 1;
            d.VB = pool + w.V1a; d.vb_cplx = 1; d.b3 = (long)d3 * N1 * r2; d.bk = 1; d.b1 = (long)r2 * d3; d.bh = d3;
            dt.push_back(d);
            // T4a: va = Rr[i3][h][k], vb = Lc[(i1,h)][k]
            DTerm e = base(1, r2, d4, 3, +1.0, 3, 1, -1.0, 1.0, sign);
            e.VA = pool + w.Rr; e.va_cplx = 1; e.a3 = (long)r2 * d4; e.ah = d4; e.ak = 1;
            e.VB = pool + w.Lc; e.vb_cplx = 1; e.bk = 1; e.b1 = (long)r2 * d4; e.bh = d4;
            if (all24) {
                e.wk = W[3];
                e.cwk = -1.0;
            }
            dt.push_back(e);
        }
        if (r3) {  // T1b: va = O2[k,h] (state h), vb = V1b[i1][(i3,h)][k]
            DTerm d = base(2, r3, d2, 1, -1.0, 0, 0, 0.0, 1.0, -sign);
            d.VA = O2; d.va_cplx = opc; d.va_hstate = 1; d.ah = 1; d.ak = d3;
            d.VB = pool + w.V1b; d.vb_cplx = 1; d.b1 = N3 * r3 * d2; d.b3 = (long)r3 * d2; d.bh = d2; d.bk = 1;
            dt.push_back(d);
            // T3b: va = Pc[i1][h][k], vb = rho[(i3,h)][k]
            DTerm e = base(2, r3, d1, 0, -1.0, 2, 1, 0.0, 1.0, sign);
            e.VA = pool + w.Pc; e.va_cplx = 1; e.a1 = (long)d1 * r3; e.ak = 1; e.ah = d1;
            e.VB = pool + w.Rho; e.vb_cplx = 1; e.b3 = (long)r3 * d1; e.bh = d1; e.bk = 1;
            if (!all13) dt.push_back(e);
        }
        if (r1) {  // T2a: va = X4[k,h] (state h), vb = V2a[i3][(i1,h)][k]
            DTerm d = base(0, r1, d4, 3, +1.0, 1, 0, 0.0, 1.0, sign);
            d.VA = X4; d.va_cplx = opc; d.va_hstate = 1; d.ah = 1; d.ak = d1;
            d.VB = pool + w.V2a; d.vb_cplx = 1; d.b3 = N1 * r1 * d4; d.b1 = (long)r1 * d4; d.bh = d4; d.bk = 1;
            dt.push_back(d);
            // T3a: va = PrAll[(i1,h)][k], vb = Qc[i3][h][k]
            DTerm e = base(0, r1, d3, 2, +1.0, 2, 1, 1.0, -1.0, sign);
            e.VA = pool + w.Pr; e.va_cplx = 1; e.a1 = (long)r1 * d3; e.ah = d3; e.ak = 1;
            e.VB = pool + w.Qc; e.vb_cplx = 1; e.b3 = (long)d3 * r1; e.bk = 1; e.bh = d3;
            if (all13) {
                e.wk = W[2];
                e.cwk = 1.0;
            }
            dt.push_back(e);
        }
        if (r4) {  // T2b: va = X4[h,k] (state h), vb = V2b[i1][(i3,h)][k]
            DTerm d = base(3, r4, d1, 0, -1.0, 1, 0, 0.0, 1.0, sign);
            d.VA = X4; d.va_cplx = opc; d.va_hstate = 1; d.ah = d1; d.ak = 1;
            d.VB = pool + w.V2b; d.vb_cplx = 1; d.b1 = (long)d1 * N3 * r4; d.bk = 1; d.b3 = (long)r4 * d1; d.bh = d1;
            dt.push_back(d);
            // T4b: va = Rc[(i3,h)][k], vb = Lr[i1][h][k]
            DTerm e = base(3, r4, d2, 1, -1.0, 3, 1, 0.0, -1.0, sign);
            e.VA = pool + w.Rc; e.va_cplx = 1; e.ak = 1; e.a3 = (long)r4 * d2; e.ah = d2;
            e.VB = pool + w.Lr; e.vb_cplx = 1; e.b1 = (long)r4 * d2; e.bh = d2; e.bk = 1;
            if (!all24) dt.push_back(e);
        }
    }
    if (!dt.empty()) {
        // classes of every sub-term, grouped by tile shape (BM 8, 16, 24, 32 or
        // 64 rows, BN 8 / 16 / 24 / 32 columns); a work item is one row tile of a class
        // over a range of anchors: as many multiply-adds as give each SM 32
        // items (one triple of a chain of 300, 2, 310 and 1 states: 60 us in the
        // kernel, 228 with anchors counted by their true k's), between 2^16 (less is lost in an item's start and its sums'
        // atomics) and 2^22
        std::vector<CClass> cls[CG_NBM][CG_NBN];
        std::vector<CItem> its[CG_NBM][CG_NBN];
        double macs[CG_NBM][CG_NBN] = {};
        double total = 0.0;
        for (const DTerm& d : dt)
            for (const CClass& c0 : plans.list[d.plan].cls[d.sidx]) total += (double)c0.nrows * c0.ncols * d.nh * d.nk;
        const long item = std::min(1L << 22, std::max(1L << 16, (long)(total / (148 * 32))));
        for (size_t q = 0; q < dt.size(); ++q) {
            const DTerm& d = dt[q];
            const APlan& pl = plans.list[d.plan];
            for (const CClass& c0 : pl.cls[d.sidx]) {
                int bm = 0, bn = 0;
                while (bm < CG_NBM - 1 && CG_BMS[bm] < c0.nrows) ++bm;
                while (CG_BNS[bn] < c0.ncols) ++bn;
                const int BM = CG_BMS[bm], BN = CG_BNS[bn];
                CClass c = c0;
                c.term = (int)q;
                const int ci = (int)cls[bm][bn].size();
                cls[bm][bn].push_back(c);
                // k's of a whole tile: where there are few of them, an item's
                // steps are one after another for every anchor
                const int hc = (int)std::max<long>(1, item / ((long)BM * BN * (ceil_div(d.nk, CG_BK_MAX) * CG_BK_MAX)));
                for (int r0 = 0; r0 < c.nrows; r0 += BM)
                    for (int h0 = 0; h0 < d.nh; h0 += hc) its[bm][bn].push_back(CItem{ci, r0, h0, std::min(d.nh, h0 + hc)});
                macs[bm][bn] += (double)c.nrows * c.ncols * d.nh * d.nk;
            }
        }
        size_t bytes = ((dt.size() * sizeof(DTerm) + 255) & ~size_t(255));
        for (int a = 0; a < CG_NBM; ++a)
            for (int b = 0; b < CG_NBN; ++b)
                bytes += ((cls[a][b].size() * sizeof(CClass) + 255) & ~size_t(255)) +
                         ((its[a][b].size() * sizeof(CItem) + 255) & ~size_t(255));
        DevBuf& bd = c->scratch[3];
        bd.reserve(bytes);
        char* base_p = bd.as<char>();
        size_t o = 0;
        auto put = [&](const void* h, size_t n) {
            char* d = base_p + o;
            if (n) h2d(d, h, n, st);
            o += (n + 255) & ~size_t(255);
            return d;
        };
        const DTerm* d_terms = reinterpret_cast<const DTerm*>(put(dt.data(), dt.size() * sizeof(DTerm)));
        // profiler ranges per tile shape; 8 FP64 operations per complex
        // multiply-add of (h, k, triple)
        static const char* const kName[CG_NBM][CG_NBN] = {
            {"contract_gemm_kernel<8,8>", "contract_gemm_kernel<8,16>", "contract_gemm_kernel<8,24>",
             "contract_gemm_kernel<8,32>"},
            {"contract_gemm_kernel<16,8>", "contract_gemm_kernel<16,16>", "contract_gemm_kernel<16,24>",
             "contract_gemm_kernel<16,32>"},
            {"contract_gemm_kernel<24,8>", "contract_gemm_kernel<24,16>", "contract_gemm_kernel<24,24>",
             "contract_gemm_kernel<24,32>"},
            {"contract_gemm_kernel<32,8>", "contract_gemm_kernel<32,16>", "contract_gemm_kernel<32,24>",
             "contract_gemm_kernel<32,32>"},
            {"contract_gemm_kernel<64,8>", "contract_gemm_kernel<64,16>", "contract_gemm_kernel<64,24>",
             "contract_gemm_kernel<64,32>"}};
        const double tol2 = pole_res < 0.0 ? -1.0 : pole_res * pole_res;  // none is within a negative resolution
        // the shapes' launches are independent (their sums meet in atomics):
        // dealt to the side streams, so that one's last wave overlaps the next
        struct Shape {
            int a, b;
            const CClass* c;
            const CItem* i;
        };
        std::vector<Shape> shapes;
        for (int a = 0; a < CG_NBM; ++a)
            for (int b = 0; b < CG_NBN; ++b) {
                if (its[a][b].empty()) continue;
                PGX_CHECK(its[a][b].size() < (1u << 31), PGX_ERR_ARG, "G2 contraction: too many work items");
                const CClass* dc = reinterpret_cast<const CClass*>(put(cls[a][b].data(), cls[a][b].size() * sizeof(CClass)));
                const CItem* di = reinterpret_cast<const CItem*>(put(its[a][b].data(), its[a][b].size() * sizeof(CItem)));
                shapes.push_back(Shape{a, b, dc, di});
            }
        std::sort(shapes.begin(), shapes.end(), [&](const Shape& x, const Shape& y) { return macs[x.a][x.b] > macs[y.a][y.b]; });
        ensure_side_streams(c);
        const int nside = (int)std::min<size_t>(4, shapes.size());
        PGX_CUDA(cudaEventRecord(c->fork, st));
        for (int i = 0; i < nside; ++i) PGX_CUDA(cudaStreamWaitEvent(c->aux[i], c->fork, 0));
        SideJoin join(c, st, nside);
        for (size_t i = 0; i < shapes.size(); ++i) {
            const Shape& x = shapes[i];
            cudaStream_t sx = c->aux[i % nside];
            ProfRange pr(kName[x.a][x.b], sx, 8.0 * macs[x.a][x.b], 0.0);
            launch_contract(CG_BMS[x.a], CG_BNS[x.b], (unsigned)its[x.a][x.b].size(), sx, d_terms, x.c, x.i, P.beta, tol2,
                            d_out);
        }
        check_launch("contract_gemm_kernel");
    }
    // the next batch reuses the device descriptor buffers in stream order
}

// Whether the sum over every state runs faster in this form, every state an
// anchor, than part by part in full matrices (pgx_g2.cu).  That form has two
// products per pair (z1', z3') that occurs and two per z1' and z3', this one
// four per pair of the (z1', z3') plane (z1' taken up to conjugation for a real
// Hamiltonian), two per z1' and four per z3', about 15% slower each for the
// dressing, on tiles of eight rows and columns at least; but that form spends
// some 0.12 ms per part, worth 3e9 operations, on its own launches and waits, and
// 30 ns per triple of a permutation's plan, this one 0.08 ms per call and 1 us
// per (z1', z3') that occurs.  Over 410 lists (cubes to 32^3, parts of them,
// scattered ones; one, six or all parts of models of 1 to 5 sites) the choice
// is 2% off the better one in the mean; the worst are 1.8 times the full matrices'
// time (one chain, 1024 triples of one z1) and 2.3 times this form's (one chain of
// 100 states, 16^3).  Wall times there and here: plaquette (96 parts) 8^3 12.5 and
// 0.87 ms, one triple 9.3 and 0.46; 6-site ring (216 parts, blocks to 400) 9^3 190
// and 64; Anderson 1+5 (blocks to 400) 8^3 153 and 38; 7-site ring (blocks to
// 1225) 4^3 779 and 393; an atom's 64^3 grid 93 and 77, a tenth of it 14 and 76;
// one chain of 300, 2, 310 and 1 states at 25 scattered triples 0.38 and 0.73, of
// 1, 7, 2 and 9 states at 60 scattered ones 0.22 and 0.27.
bool anchored_faster(const Problem& P, int nparts, const pgx_g2_part* parts, int nfreq, const Values& v) {
    const bool real = !P.is_complex;
    double all[3], up[3], closed[3];  // values that occur; those above the axis, and all, with their conjugates
    for (int k = 0; k < 3; ++k) {
        all[k] = v.occur[k];
        closed[k] = (double)v.val[k].size();
        up[k] = 0.0;
        for (const cd& x : v.val[k]) up[k] += x.y >= 0.0;
        if (!real) up[k] = all[k];
    }
    double extra = 0.0;
    double groups[9] = {};  // pairs of a permutation's plan
    for (int q = 0; q < nparts; ++q) {
        double d[4];
        for (int k = 0; k < 4; ++k) d[k] = std::max(8, P.dims[parts[q].block[k]]);
        const int a = parts[q].perm[0], b = parts[q].perm[2];
        const double m1 = d[0] * d[1] * d[3], m2 = d[0] * d[1] * d[2], m3 = d[0] * d[2] * d[3], m4 = d[1] * d[2] * d[3];
        const double pairs = std::min((double)nfreq, all[a] * all[b]);
        const double there = 8.0 * pairs * (m3 + m4) + 4.0 * (all[a] * (m1 + m2) + all[b] * (m3 + m4));
        const double z3 = real ? 0.5 * closed[b] : closed[b];  // conjugate z3 share their products
        const double here = 8.0 * up[a] * z3 * (m1 + m2 + m3 + m4) + 4.0 * up[a] * (m1 + m2) + 8.0 * z3 * (m3 + m4);
        extra += 1.15 * here - there;
        auto& n = groups[a * 3 + b];
        n = std::max(n, pairs);
    }
    for (double n : groups)
        if (n > 0.0) extra += 2.5e7 * n - 7.5e5 * nfreq;
    return extra <= 3e9 * nparts - 2e9;
}

void run_g2_anchored(pgx_ctx* c, int nparts, const pgx_g2_part* parts, int nfreq, Values values, double pole_res,
                     double anchor_tol, int split, bool exact, double* out) {
    Problem& P = c->P;
    cudaStream_t st = c->stream;
    Points pt;
    build_points(pt, std::move(values), nfreq, !P.is_complex);
    // anchor states per block (weights above the threshold)
    const std::vector<double>& w = P.w_host;  // copied when the weights were computed
    PGX_CHECK((long)w.size() == P.esize, PGX_ERR_STATE, "pgx_weights first");
    std::vector<int> hot;
    std::vector<long> hot_off(P.nblocks + 1, 0);
    std::vector<int> nhot(P.nblocks, 0);
    for (int b = 0; b < P.nblocks; ++b) {
        hot_off[b] = (long)hot.size();
        for (int i = 0; i < P.dims[b]; ++i)
            if (w[P.eoff[b] + i] > anchor_tol) hot.push_back(i);
        nhot[b] = (int)(hot.size() - hot_off[b]);
    }
    hot_off[P.nblocks] = (long)hot.size();
    // Digits of the split products per anchor block.  A product's error
    // reaches G2 multiplied by the Boltzmann weights of its anchor states, so a
    // block whose largest weight is a factor 254^k below the overall largest
    // (with the budget F of pgx_set_g2_split_weight_budget as allowance) drops
    // k digits, each of which multiplies the product's error by about 254: no
    // product then carries more than F times the error of a product of the
    // dominant block at the full digit count.  At least 3 digits are kept.
    std::vector<int> bdig;
    if (split > 0 && c->g2_split_weight_budget > 0.0) {
        double wall = 0.0;
        std::vector<double> wb(P.nblocks, 0.0);
        for (int b = 0; b < P.nblocks; ++b)
            for (int i = 0; i < P.dims[b]; ++i) wb[b] = std::max(wb[b], w[P.eoff[b] + i]);
        for (double x : wb) wall = std::max(wall, x);
        bdig.assign(P.nblocks, split);
        for (int b = 0; b < P.nblocks; ++b) {
            if (!(wb[b] > 0.0) || !(wall > 0.0)) continue;
            const int k = (int)std::floor(std::log(c->g2_split_weight_budget * wall / wb[b]) / std::log(254.0));
            bdig[b] = std::max(std::min(3, split), split - std::max(0, k));
        }
    }
    DevBuf& bh = c->scratch[11];
    bh.reserve(std::max<size_t>(hot.size(), 1) * sizeof(int));
    if (!hot.empty()) h2d(bh.p, hot.data(), hot.size() * sizeof(int), st);
    // permutations of the parts
    std::map<std::tuple<int, int, int>, int> perm_id;
    std::vector<std::array<int, 3>> perms;
    std::vector<int> part_perm(nparts);
    for (int q = 0; q < nparts; ++q) {
        auto key = std::make_tuple(parts[q].perm[0], parts[q].perm[1], parts[q].perm[2]);
        auto it = perm_id.find(key);
        if (it == perm_id.end()) {
            it = perm_id.emplace(key, (int)perms.size()).first;
            perms.push_back({parts[q].perm[0], parts[q].perm[1], parts[q].perm[2]});
        }
        part_perm[q] = it->second;
    }
    // anchor counts per part, and the workspace of one chain for N1 x N3 frequencies
    std::vector<std::array<int, 4>> rs(nparts);
    for (int q = 0; q < nparts; ++q)
        for (int k = 0; k < 4; ++k) rs[q][k] = nhot[parts[q].block[k]];
    auto chain_ws = [&](int q, long N1, long N3) {
        int d[4];
        for (int k = 0; k < 4; ++k) d[k] = P.dims[parts[q].block[k]];
        const auto& r = rs[q];
        ChainWs x{};
        long o = 0;
        auto take = [&](long n) {
            long r0 = o;
            o += (n + 1) & ~1L;  // keep 32-byte alignment of complex doubles
            return r0;
        };
        x.Lc = take((long)d[3] * N1 * r[1]);
        x.Lr = take(N1 * r[3] * d[1]);
        x.Pr = take(N1 * r[0] * d[2]);
        x.Pc = take(N1 * d[0] * r[2]);
        x.Rho = take(N3 * r[2] * d[0]);
        x.Qc = take(N3 * d[2] * r[0]);
        x.Rr = take(N3 * r[1] * d[3]);
        x.Rc = take((long)d[1] * N3 * r[3]);
        x.V1a = take(N3 * d[2] * N1 * r[1]);
        x.V1b = take(N1 * N3 * r[2] * d[1]);
        x.V2a = take(N3 * N1 * r[0] * d[3]);
        x.V2b = take(N1 * d[0] * N3 * r[3]);
        x.end = o;
        return x;
    };
    auto active = [&](int q) { return rs[q][0] + rs[q][1] + rs[q][2] + rs[q][3] > 0; };
    // Parts are batched up to `budget` of workspace.  One chain may take up to
    // `tile_budget` (by default half the free device memory, at most 48 GiB); beyond it
    // the permutation's (z1', z3') plane is cut into tiles, each with all of
    // its triples' z2'.  The stacked products are per (z1', z3') pair, so
    // tiling does not repeat them; the per-z1' and per-z3' anchored products
    // are repeated once per tile row or column.
    const long budget = (long)((c->g2_batch_bytes > 0 ? c->g2_batch_bytes : (3LL << 30)) / (long long)sizeof(cd));
    long tile_budget = -1;  // resolved when a chain exceeds the batch budget
    auto chain_limit = [&]() {
        if (tile_budget >= 0) return tile_budget;
        if (c->g2_chain_bytes > 0) {
            tile_budget = (long)(c->g2_chain_bytes / (long long)sizeof(cd));
        } else {
            size_t free_b = 0, total_b = 0;
            PGX_CUDA(cudaMemGetInfo(&free_b, &total_b));
            tile_budget = std::max(budget, (long)(std::min<size_t>(free_b / 2, size_t(48) << 30) / sizeof(cd)));
        }
        return tile_budget;
    };
    Plans plans;
    plans.perm.resize(perms.size());
    Blob blob;
    std::vector<std::vector<int>> perm_plans(perms.size());
    for (size_t p = 0; p < perms.size(); ++p) {
        PermIndex& ix = plans.perm[p];
        index_perm(ix, perms[p].data(), pt);
        const long N1 = (long)ix.Z1.size(), N3 = (long)ix.Z3.size();
        auto fits = [&](long b) {
            for (int q = 0; q < nparts; ++q) {
                if (part_perm[q] != (int)p || !active(q)) continue;
                const long e = chain_ws(q, std::min(N1, b), std::min(N3, b)).end;
                if (e > budget && e > chain_limit()) return false;
            }
            return true;
        };
        long B = std::max<long>(1, std::max(N1, N3));
        while (B > 1 && !fits(B)) B = std::max<long>(1, std::min(B - 1, B * 3 / 4));
        const long T1 = ceil_div(std::max<long>(N1, 1), std::min(std::max<long>(N1, 1), B));
        const long T3 = ceil_div(std::max<long>(N3, 1), std::min(std::max<long>(N3, 1), B));
        const long b1 = ceil_div(std::max<long>(N1, 1), T1), b3 = ceil_div(std::max<long>(N3, 1), T3);
        std::vector<std::vector<int>> tiles((size_t)(T1 * T3));
        if (T1 * T3 == 1) {
            tiles[0] = ix.pts;
        } else {
            for (int t : ix.pts) tiles[(size_t)((ix.j1[t] / b1) * T3 + ix.j3[t] / b3)].push_back(t);
        }
        for (long u = 0; u < T1; ++u)
            for (long v = 0; v < T3; ++v) {
                const auto& tl = tiles[(size_t)(u * T3 + v)];
                if (tl.empty()) continue;
                const int o1 = (int)(u * b1), o3 = (int)(v * b3);
                const int n1 = (int)std::min(b1, N1 - o1), n3 = (int)std::min(b3, N3 - o3);
                perm_plans[p].push_back((int)plans.list.size());
                plans.list.emplace_back();
                plans.perm_of.push_back((int)p);
                build_aplan(plans.list.back(), tl, ix, o1, n1, o3, n3, blob);
            }
    }
    plans.upload_groups(blob, c->scratch[10], st);
    DevBuf& pool_b = c->scratch[6];
    DevBuf& out_b = c->scratch[9];
    out_b.reserve(std::max(pt.npts, 1) * sizeof(cd));
    PGX_CUDA(cudaMemsetAsync(out_b.p, 0, std::max(pt.npts, 1) * sizeof(cd), st));
    std::vector<int> batch, bplan;
    std::vector<ChainWs> bws;
    // the full sum reports the time and operations of its products
    std::vector<cudaEvent_t> gemm_ev;
    std::vector<cudaEvent_t>* ev = exact ? &gemm_ev : nullptr;
    long used = 0;
    auto flush = [&]() {
        if (batch.empty()) return;
        pool_b.reserve(std::max<long>(used, 1) * sizeof(cd));
        if (P.is_complex)
            run_batch<cd>(c, batch, bplan, bws, parts, plans, rs, pool_b.as<cd>(), bh.as<int>(), hot_off, pole_res,
                          split, bdig, ev, out_b.as<cd>());
        else
            run_batch<double>(c, batch, bplan, bws, parts, plans, rs, pool_b.as<cd>(), bh.as<int>(), hot_off, pole_res,
                              split, bdig, ev, out_b.as<cd>());
        batch.clear();
        bplan.clear();
        bws.clear();
        used = 0;
    };
    for (size_t p = 0; p < perms.size(); ++p)
        for (int pid : perm_plans[p])
            for (int q = 0; q < nparts; ++q) {
                if (part_perm[q] != (int)p || !active(q)) continue;
                ChainWs x = chain_ws(q, (long)plans.list[pid].Z1.size(), (long)plans.list[pid].Z3.size());
                if (used > 0 && used + x.end > budget) flush();
                for (long* f : {&x.Lc, &x.Lr, &x.Pr, &x.Pc, &x.Rho, &x.Qc, &x.Rr, &x.Rc, &x.V1a, &x.V1b, &x.V2a,
                                &x.V2b, &x.end})
                    *f += used;
                used = x.end;
                batch.push_back(q);
                bplan.push_back(pid);
                bws.push_back(x);
            }
    flush();
    std::vector<cd> sum(pt.npts);
    PGX_CUDA(cudaMemcpyAsync(sum.data(), out_b.p, pt.npts * sizeof(cd), cudaMemcpyDeviceToHost, st));
    PGX_CUDA(cudaStreamSynchronize(st));
    if (pt.npts > pt.ncls)
        for (int u = 0; u < pt.ncls; ++u) sum[u] = sum[u] + conj(sum[pt.ncls + u]);
    for (int t = 0; t < nfreq; ++t) {
        const cd v = pt.flip[t] ? conj(sum[pt.cls[t]]) : sum[pt.cls[t]];
        out[2 * (size_t)t] = v.x;
        out[2 * (size_t)t + 1] = v.y;
    }
    if (exact) {
        for (size_t i = 0; i + 1 < gemm_ev.size(); i += 2) {
            float ms = 0.f;
            PGX_CUDA(cudaEventElapsedTime(&ms, gemm_ev[i], gemm_ev[i + 1]));
            c->g2t.gemm_ms += ms;
        }
        for (cudaEvent_t e : gemm_ev) c->prof.spare.push_back(e);
    }
}

}  // namespace pgx
