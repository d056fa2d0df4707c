// K1: batched FP64 symmetric eigensolver.
//
// Replaces Eigen::SelfAdjointEigenSolver as called by HamiltonianPart::computeImpl
// (HamiltonianPart.cpp:90-102).  Stages:
//   1. Householder reduction to tridiagonal form T (Golub & Van Loan, "Matrix
//      Computations", 4th ed., 8.3.1):
//      eigh_cluster_kernel, one thread-block cluster of 1-16 CTAs per block
//      with the matrix in distributed shared memory (blocks up to 513 states);
//      larger blocks: a blocked reduction (panels of 32 columns, one trailing
//      update per panel) over the whole GPU.
//   2. bisect_kernel: multisection with Sturm counts on the unreduced pieces
//      of T (8.4.1).
//   3. vector_kernel, one thread per eigenvalue: inverse iteration with a
//      partial-pivoting tridiagonal LU; ortho_kernel: modified Gram-Schmidt
//      inside chains of close eigenvalues; eigenvalues are ranked so that the
//      output is ascending.
//   4. the reflectors applied to Z panel by panel (bt_apply_kernel); blocks
//      beyond 3073 states form Q and U = Q Z by GEMMs.
// A non-finite eigenvector sets a device status word instead of trapping.

#include <cooperative_groups.h>

#include <cmath>
#include <cstring>

#include "pgx_common.cuh"
#include "pgx_gemm.cuh"
#include "pgx_internal.h"

namespace pgx {

namespace {


__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ----------------------------------------------------------------------------
// Householder stage for blocks too large for a cluster's shared memory
// (n > 513): the blocked reduction of LAPACK's dsytrd / dlatrd (lower).
// Panels of BHH_NB columns.  Column j of the panel that starts at k is first
// brought up to date with the panel's earlier reflectors,
//   a = A(j:, j) - V W(j, :)^T - W V(j, :)^T,
// then reflected (v, tau; d_j = a_j, e_j = alpha) and
//   w = tau (A(j+1:, j+1:) v - V (W^T v) - W (V^T v)),  w -= (tau/2)(w.v) v,
// with A the matrix as it was at the start of the panel: the trailing matrix
// is only read per column (bhh_symv_kernel) and written once per panel,
// A(k+p:, k+p:) -= V W^T + W V^T (bhh_update_kernel).
// The reflectors stay, scaled to tau = 1, in the rows of A right of the
// diagonal (zeros left of it).  Up to 3073 states the eigenvectors are formed from
// them directly (bt_apply_kernel); beyond, Q = H_0 ... H_{n-3} is formed panel
// by panel, from the last one, as
// Q(k+1:, k+1:) += V (-T) (V^T Q(k+1:, k+1:)), where T is the upper
// triangular factor of the panel's block reflector I - V T V^T (LAPACK
// dlarft).  Every such block of a problem advances in the same launches.
constexpr int BHH_NB = 32;  // panel width
constexpr int BHH_COL_THREADS = 512;
constexpr int BHH_SYMV_THREADS = 128;

struct BigBlk {
    long moff, eoff, boff;  // matrix and vector offsets; scratch offset in S (doubles)
    int n, pad;
};
struct BigArgs {
    const BigBlk* blk;  // the large blocks, largest first
    int nact;           // entries of `blk` this launch covers (a prefix)
    double* A;    // per block n x n row-major working copy of H
    double* Zc;   // per block Q, column-major
    double* S;    // scratch
    double* tri;  // per block: d (n), e (n)
    int k;        // first column of the current panel
    int fin;      // column whose w is completed (-1: none)
    int col;      // column to reflect (-1: none)
    int slots;    // the product before this column was left in slots (bhh_symv_tri_kernel)
    int ntri;     // tiles of the largest block there
};

// Scratch of one large block, in doubles: V and W (BHH_NB columns of n each),
// y (n), tau (n), then per panel its Gram matrix and -T (BHH_NB^2 each), the
// slots of y and the tiles' parts of v . (tau y) (bhh_symv_tri_kernel), and the dots of
// the panel's columns with the reflector (2 BHH_NB).
constexpr int TRI_T = 128;  // rows and columns of a tile there
__host__ __device__ inline long bhh_slots(int m) { return (m + TRI_T - 1) / TRI_T; }
__host__ __device__ inline long bhh_panels(int n) { return n > 2 ? (n - 2 + BHH_NB - 1) / BHH_NB : 0; }
__host__ __device__ inline long bhh_scratch_doubles(int n) {
    return 2L * BHH_NB * n + 2L * n + 2 * bhh_panels(n) * BHH_NB * BHH_NB + bhh_slots(n) * n +
           bhh_slots(n) * (bhh_slots(n) + 1) / 2 + 2 * BHH_NB;
}
__host__ __device__ inline long bhh_slots_at(int n) {
    return 2L * BHH_NB * n + 2L * n + 2 * bhh_panels(n) * BHH_NB * BHH_NB;
}
__host__ __device__ inline long bhh_dots_at(int n) { return bhh_scratch_doubles(n) - 2 * BHH_NB; }

// Completes w of column fin (in this panel) and brings column col = fin + 1 up
// to date; grid (row groups, block).  The column stays raw in V: the product
// kernel reflects it, and leaves tau and the reflector's leading entry v0 (in
// y[fin]), which takes its place in V here.  Every CTA finds w . v for itself,
//   w . v = v . (tau y) - 2 sum_s (V_s . v) (tau (W_s . v)),
// so CTAs need nothing of one another; tau enters each product first, as without
// it they grow with the cube of the matrix's scale.  Both vectors need every row's
// combination of the panel's earlier V and W columns: one sweep reads them for
// both (four lanes a row, each a quarter of the columns), the first eight rows
// of a warp ahead of the block sum.  What bounds it: the latency of one round
// of L2 reads, a block sum and the launch.  64 models of 3 to 6 bath sites: 26 ms
// for all columns, against 42 on clusters that reduced the column's norm and
// w . v between their CTAs; blocks of 4 x 1225 and 8 x 735 states, whole
// eigensolve: 24.8 -> 22.9 ms.
template <bool SLOTS>
__global__ void __launch_bounds__(BHH_COL_THREADS, SLOTS ? 1 : 2) bhh_col_kernel(BigArgs g) {
    __shared__ double dw[BHH_NB], dv[BHH_NB], jw[BHH_NB], jv[BHH_NB];
    __shared__ double red[BHH_COL_THREADS / 32], s_dd, s_yj;
    cudaTriggerProgrammaticLaunchCompletion();
    const BigBlk bl = g.blk[blockIdx.y];
    const int n = bl.n, last = n - 3;  // the last column with a reflector
    double* A = g.A + bl.moff;
    double* V = g.S + bl.boff;  // column t at V + t n
    double* W = V + (long)BHH_NB * n;
    const double* y = W + (long)BHH_NB * n;
    const double* tau = y + n;
    const double* dots = V + bhh_dots_at(n);
    const double* slot = V + bhh_slots_at(n);  // slot t of y at slot + t n
    const double* parts = slot + bhh_slots(n) * n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool fin = g.fin >= 0 && g.fin <= last, col = g.col >= 0 && g.col <= last;
    if (!fin && !col) return;
    const int f = g.fin, j = g.col, cf = fin ? f - g.k : 0, cc = col ? j - g.k : 0;
    const int lo = fin ? f + 1 : j;  // the first row of v, w and the column
    const int ns = SLOTS && fin ? (int)bhh_slots(n - lo) : 0;
    double* vf = V + (long)cf * n;
    const int sg = lane >> 3;
    cudaGridDependencySynchronize();
    double tf = 0.0, v0 = 0.0;
    if (fin) {
        tf = tau[f];
        v0 = y[f];
    }
    double pv[BHH_NB / 4], pw[BHH_NB / 4], x = 0.0, acc = 0.0, v = 0.0;
    auto load = [&](int r) {
        x = acc = v = 0.0;
        const bool in = r >= lo && r < n;
        if (in && fin) v = r == lo ? v0 : vf[r];
        if (in && sg == 0) {
            if (col) x = A[(long)j * n + r];  // row j holds column j (A symmetric)
            if (fin && !SLOTS) acc = y[r];
        }
        if constexpr (SLOTS)
            for (int t = sg; t < ns; t += 4) acc += in ? slot[(long)t * n + r] : 0.0;
#pragma unroll
        for (int q = 0; q < BHH_NB / 4; ++q) {
            const int s = sg + 4 * q;
            pv[q] = in && s < cf ? V[(long)s * n + r] : 0.0;
            pw[q] = in && s < cf ? W[(long)s * n + r] : 0.0;
        }
    };
    const int stride = 8 * (BHH_COL_THREADS / 32) * (int)gridDim.x;
    int rb = (lo & ~7) + 8 * (blockIdx.x * (BHH_COL_THREADS / 32) + wid);
    load(rb + (lane & 7));
    double K = 0.0, wj = 0.0;
    if (fin) {
        double vy = 0.0;
        if constexpr (SLOTS)
            for (int t = tid; t < ns * (ns + 1) / 2; t += BHH_COL_THREADS) vy += parts[t];
        else
            for (int r = lo + 1 + tid; r < n; r += BHH_COL_THREADS) vy = fma(vf[r], tf * y[r], vy);
        if (tid < BHH_NB) {
            double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
            if (tid < cf) {
                a = dots[2 * tid];
                b = dots[2 * tid + 1];
                c = col ? W[(long)tid * n + j] : 0.0;
                d = col ? V[(long)tid * n + j] : 0.0;
            }
            dw[tid] = a;
            dv[tid] = b;
            jw[tid] = c;
            jv[tid] = d;
            double yl = !SLOTS && tid == 0 ? y[lo] : 0.0;
            for (int t = tid; t < ns; t += 32) yl += slot[(long)t * n + lo];
            const double dd = warp_sum(a * tf * b), dj = warp_sum(d * a + c * b);
            yl = warp_sum(yl);
            if (tid == 0) {
                s_dd = dd;
                s_yj = yl - dj;
                if (!SLOTS) vy = fma(v0, tf * yl, vy);
            }
        }
        vy = warp_sum(vy);
        if (lane == 0) red[wid] = vy;
        __syncthreads();
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < BHH_COL_THREADS / 32; ++q) t += red[q];
        K = 0.5 * tf * (t - 2.0 * s_dd);
        wj = tf * s_yj - K * v0;
    }
    const double st = sqrt(tf);
    for (; rb < n; rb += stride) {
        const int r = rb + (lane & 7);
#pragma unroll
        for (int q = 0; q < BHH_NB / 4; ++q) {
            const int s = sg + 4 * q;
            if (s < cf) {
                acc -= pv[q] * dw[s] + pw[q] * dv[s];
                x -= pv[q] * jw[s] + pw[q] * jv[s];
            }
        }
#pragma unroll
        for (int o = 8; o < 32; o <<= 1) {
            acc += __shfl_xor_sync(0xffffffffu, acc, o);
            x += __shfl_xor_sync(0xffffffffu, x, o);
        }
        if (r >= lo && r < n) {
            const double w = tf * acc - K * v;
            if (fin && sg == 0) {
                W[(long)cf * n + r] = w;
                if (r == lo) vf[r] = v0;
            }
            if (fin && sg == 1) A[(long)f * n + r] = v * st;  // row f of A: sqrt(tau) v
            if (col && sg == 2) {
                x -= v * wj + w * v0;
                if (r == j) g.tri[2 * bl.eoff + j] = x;
                V[(long)cc * n + r] = x;
            }
        }
        if (rb + stride < n) load(r + stride);
    }
    if (fin)  // zeros up to the diagonal
        for (int r = blockIdx.x * BHH_COL_THREADS + tid; r < lo; r += gridDim.x * BHH_COL_THREADS) A[(long)f * n + r] = 0.0;
}

// A load that is issued where it stands: the compiler otherwise groups the row
// loads with their products, three or four in flight instead of the eight.
__device__ inline double ld_now(const double* p) {
    double r;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(p) : "memory");
    return r;
}

// Reflects column j = col of every active block (raw in V): v, tau, e_j, then
// y(j+1:) = A(j+1:, j+1:) v and the dots W_s . v, V_s . v of the panel's
// earlier columns as further rows.  v is the raw column but for its leading
// entry, which needs the column's norm: a warp sums the squares on its way
// through the column and adds that entry's product at the end.  Grid (rows,
// block), RW rows per warp and 8 / RW columns per lane at once, so eight row
// loads are in flight per lane, and with several rows each entry of v is loaded
// once for them.  What bounds it: the latency of L2 with the warps there are,
// hence fewer rows per warp for fewer rows (blocks of 4 x 1225 and 8 x 735
// states, whole eigensolve: 24.8 ms, against 32.3 with four rows per warp
// throughout; with the loads issued together 21.8, against 22.9 without).
template <int RW>
__global__ void __launch_bounds__(BHH_SYMV_THREADS, RW == 4 ? 10 : 6) bhh_symv_kernel(BigArgs g) {
    constexpr int U = 8 / RW;
    cudaTriggerProgrammaticLaunchCompletion();
    const BigBlk bl = g.blk[blockIdx.y];
    const int n = bl.n, j = g.col, cc = j - g.k, m = n - j - 1, rows = m + 2 * cc;
    double* V = g.S + bl.boff;
    const double* v = V + (long)cc * n + (j + 1);
    double* y = V + 2L * BHH_NB * n + (j + 1);
    double* dots = V + bhh_dots_at(n);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (m < 2) return;  // no reflector
    const int rr = (blockIdx.x * (BHH_SYMV_THREADS / 32) + wid) * RW;
    if (rr >= rows) return;
    const double* p[RW];
#pragma unroll
    for (int u = 0; u < RW; ++u) {
        const int r = min(rr + u, rows - 1), d = r - m;
        p[u] = r < m ? g.A + bl.moff + (long)(j + 1 + r) * n + (j + 1)
                     : V + ((d & 1) ? 0L : (long)BHH_NB * n) + (long)(d >> 1) * n + (j + 1);
    }
    cudaGridDependencySynchronize();
    double s[RW], sigma = 0.0;
#pragma unroll
    for (int u = 0; u < RW; ++u) s[u] = 0.0;
    int i = lane;
    for (; i + 32 * (U - 1) < m; i += 32 * U) {
        double x[U], a[RW][U];
#pragma unroll
        for (int t = 0; t < U; ++t) {
            x[t] = ld_now(v + i + 32 * t);
#pragma unroll
            for (int u = 0; u < RW; ++u) a[u][t] = ld_now(p[u] + i + 32 * t);
        }
        if (i == 0) x[0] = 0.0;  // the leading entry follows
#pragma unroll
        for (int t = 0; t < U; ++t) sigma = fma(x[t], x[t], sigma);
#pragma unroll
        for (int u = 0; u < RW; ++u)
#pragma unroll
            for (int t = 0; t < U; ++t) s[u] = fma(a[u][t], x[t], s[u]);
    }
    {  // the rest: up to U columns per lane
        double x[U], a[RW][U];
#pragma unroll
        for (int t = 0; t < U; ++t) {
            const bool in = i + 32 * t < m;
            x[t] = in ? v[i + 32 * t] : 0.0;
#pragma unroll
            for (int u = 0; u < RW; ++u) a[u][t] = in ? p[u][i + 32 * t] : 0.0;
        }
        if (i == 0) x[0] = 0.0;
#pragma unroll
        for (int t = 0; t < U; ++t) sigma = fma(x[t], x[t], sigma);
#pragma unroll
        for (int u = 0; u < RW; ++u)
#pragma unroll
            for (int t = 0; t < U; ++t) s[u] = fma(a[u][t], x[t], s[u]);
    }
    const double x0 = v[0];
    double a0[RW];
#pragma unroll
    for (int u = 0; u < RW; ++u) a0[u] = p[u][0];
    sigma = warp_sum(sigma);
    double alpha = x0, v0 = 0.0, tj = 0.0;
    if (sigma != 0.0) {
        const double t = fma(x0, x0, sigma), mu = t * rsqrt(t);
        alpha = (x0 > 0.0) ? -mu : mu;  // v0 = x0 - alpha without cancellation
        v0 = x0 - alpha;
        tj = 2.0 * recip_pos(fma(v0, v0, sigma));
    }
    if (rr == 0 && lane == 0) {
        g.tri[2 * bl.eoff + n + j] = alpha;
        V[2L * BHH_NB * n + n + j] = tj;
        V[2L * BHH_NB * n + j] = v0;
    }
#pragma unroll
    for (int u = 0; u < RW; ++u) {
        const double t = fma(a0[u], v0, warp_sum(s[u]));
        const int r = rr + u;
        if (lane == 0 && r < rows) {
            if (r < m) y[r] = t;
            else dots[r - m] = t;
        }
    }
}

// The same products and dots where the active blocks exceed L2: only tiles on or
// below the diagonal are read, each for both of its products, A_ij v_j and
// A_ij^T v_i.  CTA (tile, block): a warp 16 rows, a lane 4 columns of the tile, 16
// loads in flight; the products of rows of tile row R go to slot tj of y,
// those of its columns to slot ti, so every row finds its parts in slots 0 ..
// and nothing is added up in memory; the tile's part of v . (tau y) goes beside them.
// CTAs past the tiles take the dots, a row per warp.  Every CTA sums the
// column's squares itself.  What bounds it: reading the triangle from HBM, at
// half the copy rate, as a CTA's column sums and exchanges stand between its
// loads.  64 models of 3 to 6 bath sites: the 783 columns that take this path
// 67 ms, 3.7 TB/s with the diagonal tiles, the column kernel's sums of slots 5
// more; whole step 275 -> 266 ms.  Strips of 2 or 4 tiles per CTA: 70 to 77.
constexpr int SYT_THREADS = 256;
// The matrices' bytes above which one triangle is read: below, they come from L2,
// where twice the bytes cost less than the sums (7-site ring, 80 MB at first:
// whole solve 24.4 ms, against 29.7 with one triangle).
constexpr double SYT_BYTES = 100e6;
__global__ void __launch_bounds__(SYT_THREADS, 3) bhh_symv_tri_kernel(BigArgs g) {
    __shared__ double red[SYT_THREADS / 32], vi[TRI_T], cols[SYT_THREADS / 32][TRI_T];
    cudaTriggerProgrammaticLaunchCompletion();
    const BigBlk bl = g.blk[blockIdx.y];
    const int n = bl.n, j = g.col, cc = j - g.k, m = n - j - 1;
    if (m < 2) return;  // no reflector
    const int nt = (int)bhh_slots(m), tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const bool dot = tile >= g.ntri;
    if (!dot && tile >= nt * (nt + 1) / 2) return;
    if (dot && (tile - g.ntri) * (SYT_THREADS / 32) >= 2 * cc) return;
    double* V = g.S + bl.boff;
    const double* v = V + (long)cc * n + (j + 1);
    cudaGridDependencySynchronize();
    double sigma = 0.0;
    for (int i = 1 + tid; i < m; i += SYT_THREADS) sigma = fma(v[i], v[i], sigma);
    sigma = warp_sum(sigma);
    if (lane == 0) red[wid] = sigma;
    __syncthreads();
    sigma = 0.0;
#pragma unroll
    for (int q = 0; q < SYT_THREADS / 32; ++q) sigma += red[q];
    const double x0 = v[0];
    double alpha = x0, v0 = 0.0, tj = 0.0;
    if (sigma != 0.0) {
        const double t = fma(x0, x0, sigma), mu = t * rsqrt(t);
        alpha = (x0 > 0.0) ? -mu : mu;  // v0 = x0 - alpha without cancellation
        v0 = x0 - alpha;
        tj = 2.0 * recip_pos(fma(v0, v0, sigma));
    }
    if (tile == 0 && tid == 0) {
        g.tri[2 * bl.eoff + n + j] = alpha;
        V[2L * BHH_NB * n + n + j] = tj;
        V[2L * BHH_NB * n + j] = v0;
    }
    if (dot) {
        const int d = (tile - g.ntri) * (SYT_THREADS / 32) + wid;
        if (d >= 2 * cc) return;
        const double* p = V + ((d & 1) ? 0L : (long)BHH_NB * n) + (long)(d >> 1) * n + (j + 1);
        double t = 0.0;
        for (int i = lane; i < m; i += 32) t = fma(p[i], i == 0 ? v0 : v[i], t);
        t = warp_sum(t);
        if (lane == 0) V[bhh_dots_at(n) + d] = t;
        return;
    }
    int ti = (int)((sqrtf(8.0f * tile + 1.0f) - 1.0f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= tile) ++ti;
    while (ti * (ti + 1) / 2 > tile) --ti;
    const int ct = tile - ti * (ti + 1) / 2, i0 = ti * TRI_T, j0 = ct * TRI_T;
    if (tid < TRI_T) vi[tid] = i0 + tid == 0 ? v0 : i0 + tid < m ? v[i0 + tid] : 0.0;
    double vj[4], c[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int jj = j0 + lane + 32 * q;
        vj[q] = jj == 0 ? v0 : jj < m ? v[jj] : 0.0;
    }
    __syncthreads();
    const double* A = g.A + bl.moff + (long)(j + 1) * n + (j + 1);
    double s[16];
#pragma unroll
    for (int rb = 0; rb < 16; rb += 4) {
        double a[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            // clamped: v is 0 beyond
            const double* row = A + (long)min(i0 + 16 * wid + rb + u, m - 1) * n;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                a[u][q] = ld_now(row + min(j0 + lane + 32 * q, m - 1));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const double w = vi[16 * wid + rb + u];
            s[rb + u] = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                s[rb + u] = fma(a[u][q], vj[q], s[rb + u]);
                c[q] = fma(a[u][q], w, c[q]);
            }
        }
    }
    // the 16 row sums: halving the rows a lane holds at each exchange, lane -> row lane / 2
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool up = lane & (2 * h);
#pragma unroll
        for (int u = 0; u < h; ++u) {
            const double keep = up ? s[u + h] : s[u], give = up ? s[u] : s[u + h];
            s[u] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    const double ys = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 1);
    double* slot = V + bhh_slots_at(n);
    const int row = 16 * wid + (lane >> 1);
    if (!(lane & 1) && i0 + row < m) slot[(long)ct * n + j + 1 + i0 + row] = ys;
    const double part = warp_sum(lane & 1 ? 0.0 : tj * ys * vi[row]);
    if (ct != ti)
#pragma unroll
        for (int q = 0; q < 4; ++q) cols[wid][lane + 32 * q] = c[q];
    if (lane == 0) red[wid] = part;
    __syncthreads();
    if (ct != ti && tid < TRI_T) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < SYT_THREADS / 32; ++q) t += cols[q][tid];
        slot[(long)ti * n + j + 1 + j0 + tid] = t;
    }
    if (tid == 0) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < SYT_THREADS / 32; ++q) t += red[q];
        (slot + bhh_slots(n) * n)[tile] = ct == ti ? t : 2.0 * t;
    }
}

// A(k+p:, k+p:) -= V W^T + W V^T after the panel's p columns: one 64 x 64 tile on
// or below the diagonal per CTA on the FP64 tensor cores, both operands of the
// tile whole in shared memory (up to 32 columns of V and W each), each of four
// warps 32 x 32 of it; every element is also written in its mirrored place, as
// the product kernel reads rows.  Grid (tiles of the largest block, block).
// What bounds it: the FP64 pipe for full tiles, the latency of one round of
// loads when few are left.  64 models of 3 to 6 bath sites, all panels: 10.4 ms,
// against 34 with general products of inner size 2p, whose columns were gathered
// and scaled and whose tiles covered both triangles; 7-site ring 1.0 against 2.5.
constexpr int UPD_T = 64, UPD_LD = UPD_T + 4, UPD_THREADS = 128;
constexpr size_t UPD_SMEM = 4UL * BHH_NB * UPD_LD * sizeof(double);
__global__ void __launch_bounds__(UPD_THREADS, 3) bhh_update_kernel(BigArgs g) {
    extern __shared__ double sh[];
    const BigBlk bl = g.blk[blockIdx.y];
    const int n = bl.n, p = min(BHH_NB, n - 2 - g.k), kp = g.k + p, m = n - kp;
    int ti = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
    while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
    const int tj = blockIdx.x - ti * (ti + 1) / 2, i0 = ti * UPD_T, j0 = tj * UPD_T;
    if (i0 >= m) return;
    const double* V = g.S + bl.boff + kp;
    const double* W = V + (long)BHH_NB * n;
    double* A = g.A + bl.moff + (long)kp * n + kp;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *Vi = sh, *Wi = sh + BHH_NB * UPD_LD, *Vj = Vi, *Wj = Wi;
    const int p4 = (p + 3) & ~3;
    auto fill = [&](double* dst, const double* src, int at) {
        for (int e = tid; e < p4 * UPD_T; e += UPD_THREADS) {
            const int s = e / UPD_T, r = e % UPD_T;
            const bool in = s < p && at + r < m;
            cp_elem(dst + s * UPD_LD + r, in ? src + (long)s * n + at + r : src, in);
        }
    };
    fill(Vi, V, i0);
    fill(Wi, W, i0);
    if (ti != tj) {
        Vj = Wi + BHH_NB * UPD_LD;
        Wj = Vj + BHH_NB * UPD_LD;
        fill(Vj, V, j0);
        fill(Wj, W, j0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int wr = 32 * (wid >> 1), wc = 32 * (wid & 1), fr = lane / 4, fk = lane % 4;
    double2 acc[4][4], old[4][4];
    auto mine = [&](int i, int j) { return i < m && j < m && j <= i; };
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const int i = i0 + wr + 8 * x + fr, j = j0 + wc + 8 * y + 2 * fk;
            acc[x][y] = double2{0.0, 0.0};
            old[x][y].x = mine(i, j) ? A[(long)i * n + j] : 0.0;
            old[x][y].y = mine(i, j + 1) ? A[(long)i * n + j + 1] : 0.0;
        }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (ti == tj && wc > wr) return;  // above the diagonal
    for (int s0 = 0; s0 < p4; s0 += 4) {
        const int at = (s0 + fk) * UPD_LD + fr;
        double av[4], aw[4], bv[4], bw[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            av[x] = Vi[at + wr + 8 * x];
            aw[x] = Wi[at + wr + 8 * x];
            bv[x] = Vj[at + wc + 8 * x];
            bw[x] = Wj[at + wc + 8 * x];
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) mma_f64(acc[x][y], av[x], bw[y]);
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) mma_f64(acc[x][y], aw[x], bv[y]);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = i0 + wr + 8 * x + fr, j = j0 + wc + 8 * y + 2 * fk + u;
                if (!mine(i, j)) continue;
                const double r = u ? old[x][y].y - acc[x][y].y : old[x][y].x - acc[x][y].x;
                A[(long)i * n + j] = r;
                A[(long)j * n + i] = r;
            }
}

// the last 2 x 2 of the tridiagonal, and Q = I for the first nact blocks (those that form Q)
__global__ void bhh_finish_kernel(BigArgs g) {
    const BigBlk bl = g.blk[blockIdx.x];
    const int n = bl.n;
    const double* A = g.A + bl.moff;
    double* Z = g.Zc + bl.moff;
    const long eo = bl.eoff;
    if (threadIdx.x == 0) {
        if (n >= 2) {
            g.tri[2 * eo + n - 2] = A[(long)(n - 2) * n + (n - 2)];
            g.tri[2 * eo + n + n - 2] = A[(long)(n - 1) * n + (n - 2)];
        }
        g.tri[2 * eo + n - 1] = A[(long)(n - 1) * n + (n - 1)];
        g.tri[2 * eo + n + n - 1] = 0.0;
    }
    if ((int)blockIdx.x < g.nact)
        for (long i = threadIdx.x; i < (long)n * n; i += blockDim.x) Z[i] = ((i / n) == (i % n)) ? 1.0 : 0.0;
}

// -T of every panel's block reflector from its Gram matrix G = V^T V (LAPACK
// dlarft, forward, columnwise; tau = 1): T_ii = 1, T(0:i, i) = -T(0:i, 0:i) G(0:i, i).
// One warp per (block, panel); lane t owns row t of T.
__global__ void bhh_tfactor_kernel(BigArgs g) {
    int q = blockIdx.x, bi = 0;
    for (; bi < g.nact; ++bi) {
        const int np = (int)bhh_panels(g.blk[bi].n);
        if (q < np) break;
        q -= np;
    }
    if (bi >= g.nact) return;
    const int n = g.blk[bi].n;
    const int k = q * BHH_NB, p = min(BHH_NB, n - 2 - k);
    double* base = g.S + g.blk[bi].boff;
    const double* G = base + 2L * BHH_NB * n + 2L * n + (long)q * BHH_NB * BHH_NB;
    double* nT = base + 2L * BHH_NB * n + 2L * n + (bhh_panels(n) + q) * BHH_NB * BHH_NB;
    const int t = threadIdx.x;
    double row[BHH_NB];
#pragma unroll
    for (int i = 0; i < BHH_NB; ++i) row[i] = 0.0;
#pragma unroll
    for (int i = 0; i < BHH_NB; ++i) {
        if (i < p) {
            if (t == i) row[i] = 1.0;
            if (t < i) {
                double acc = 0.0;
#pragma unroll
                for (int s2 = 0; s2 < BHH_NB; ++s2)
                    if (s2 >= t && s2 < i) acc = fma(row[s2], G[s2 * BHH_NB + i], acc);
                row[i] = -acc;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < BHH_NB; ++i) nT[t * BHH_NB + i] = -row[i];
}

// ----------------------------------------------------------------------------
// Householder stage on a thread-block cluster (blocks whose matrix fits in
// the shared memory of up to 16 CTAs, 513 states).
//
// The C CTAs of a cluster hold the block's symmetric matrix in distributed
// shared memory, row r in CTA r mod C (cyclic, so the shrinking trailing
// matrix stays spread over all CTAs).  Every CTA also holds the current row k
// (the column below the diagonal), up to date, one element per thread.  Step k:
//   every CTA forms the Householder vector v and tau from its copy of row k;
//   one sweep over its own rows r > k applies the PREVIOUS step's update
//   B -= v' w'^T + w' v'^T and forms p = tau B v with the result (up to eight
//   rows per warp, whose sums over the lanes share five shuffle rounds), and the
//   warp pushes p_r and the row's element in column k + 1 into every CTA's
//   buffer of this step's parity;
//   cluster barrier;
//   every CTA forms w = p - (tau/2)(v.p) v and from the pushed column its copy
//   of row k + 1, less v_{k+1} w + w_{k+1} v.
// So the matrix is read and written once per step, nothing is fetched from
// another CTA after the barrier, and a step has one cluster barrier and three
// CTA barriers.  A CTA one step ahead writes the other parity's buffers, and
// cannot get two steps ahead before the others pass the barrier.  What bounds
// it: those barriers and the push in large part, then shared-memory reads.
// CTA 0 stores d_k, e_k and sqrt(tau) v (row k of V in global memory), from
// which the eigenvectors are formed (bt_apply_kernel).  Anderson 1+5, the
// 400-state block: 1.16 ms, against 2.04 with a fetch from the other CTAs after
// the barrier and a sweep each for the update and the product.
constexpr int CL_THREADS = 256, CL_NW = CL_THREADS / 32;
constexpr int CL_MAX_DIM = 513;
constexpr int CL_EL = (CL_MAX_DIM + CL_THREADS - 1) / CL_THREADS;  // elements of a row per thread

struct ClusterArgs {
    const int* blocks;  // cluster -> block
    const int* dims;
    const long* moff;
    const long* eoff;
    const double* H;
    double* V;          // per block n x n: row k holds sqrt(tau_k) v_k in columns k+1..n-1
    double* tri;
};

__host__ __device__ inline size_t cluster_smem_doubles(int n, int C) {
    const int R = (n + C - 1) / C;
    return (size_t)R * n + 7 * (size_t)n;
}

__global__ void __launch_bounds__(CL_THREADS) eigh_cluster_kernel(ClusterArgs g) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double sh[];
    __shared__ double red[2][CL_NW], s_dot[2][CL_NW], s_x[2];
    const int C = (int)cl.num_blocks();
    const int c = (int)cl.block_rank();
    const int b = g.blocks[blockIdx.x / C];
    const int n = g.dims[b];
    const long mo = g.moff[b], eo = g.eoff[b];
    const int nrows = (n - c + C - 1) / C;                // rows c, c + C, ...
    double2* pb = reinterpret_cast<double2*>(sh);         // 2 n: (p_r, element of column k + 1) by parity
    double* v = sh + 4 * n;                               // 2 n: v by parity
    double* w = v + 2 * n;                                // n
    double* slab = w + n;                                 // nrows x n
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const double* Hb = g.H + mo;
    double* V = g.V + mo;

    for (int idx = tid; idx < nrows * n; idx += CL_THREADS) {
        const int lr = idx / n, j = idx % n;
        slab[idx] = Hb[(long)(c + C * lr) * n + j];
    }
    double x[CL_EL];  // this thread's elements (columns tid + CL_THREADS e) of row k
#pragma unroll
    for (int e = 0; e < CL_EL; ++e) {
        const int r = tid + CL_THREADS * e;
        x[e] = r < n ? Hb[r] : 0.0;
        if (r < n) {
            w[r] = 0.0;
            v[n + r] = 0.0;  // the step before the first
        }
    }
    cl.sync();  // every CTA of the cluster runs before the first push
    for (int k = 0; k + 2 < n; ++k) {
        const int par = k & 1;
        double *vk = v + par * n, *vo = v + (par ^ 1) * n;
        double part = 0.0;
#pragma unroll
        for (int e = 0; e < CL_EL; ++e) {
            const int r = tid + CL_THREADS * e;
            if (r < n && r >= k + 2) part = fma(x[e], x[e], part);
            if (r == k + 1) s_x[par] = x[e];
        }
        part = warp_sum(part);
        if (lane == 0) red[par][wid] = part;
        __syncthreads();  // also: w of the previous step is complete
        double sigma = 0.0;
#pragma unroll
        for (int q = 0; q < CL_NW; ++q) sigma += red[par][q];
        const double x0 = s_x[par];
        double tau = 0.0, alpha = x0, v0 = x0;
        if (sigma != 0.0) {
            const double t = fma(x0, x0, sigma), mu = t * rsqrt(t);
            alpha = (x0 > 0.0) ? -mu : mu;  // v0 = x0 - alpha without cancellation
            v0 = x0 - alpha;
            tau = 2.0 * recip_pos(fma(v0, v0, sigma));
        }
#pragma unroll
        for (int e = 0; e < CL_EL; ++e) {
            const int r = tid + CL_THREADS * e;
            if (r < n) vk[r] = r > k + 1 ? x[e] : r == k + 1 ? v0 : 0.0;
        }
        __syncthreads();
        // ---- own rows r > k: previous update, then p = tau B v; up to eight rows a warp at once
        const int m = n - k - 1;
        const double *pn = vk + k + 1, *po = vo + k + 1, *qo = w + k + 1;
        // NU rows base, base + CL_NW, ... of this warp
        auto sweep = [&](auto nu_c, int base) {
            constexpr int NU = decltype(nu_c)::value;
            const int stride = CL_NW * n;
            double* row = slab + base * n + (k + 1);
            double va[NU], wa[NU], s[NU];
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                const int r = c + C * (base + CL_NW * u);
                va[u] = vo[r];
                wa[u] = w[r];
                s[u] = 0.0;
            }
            for (int j = lane; j < m; j += 32) {
                const double a = pn[j], p = po[j], q = qo[j];
                double y[NU];
#pragma unroll
                for (int u = 0; u < NU; ++u) y[u] = row[u * stride + j];
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                    y[u] -= fma(va[u], q, wa[u] * p);
                    s[u] = fma(y[u], a, s[u]);
                    row[u * stride + j] = y[u];
                }
            }
            // sums over the lanes, halving the rows a lane holds: lane l ends with row l NU / 32
            int o = 16;
#pragma unroll
            for (int h = NU / 2; h > 0; h >>= 1, o >>= 1)
#pragma unroll
                for (int u = 0; u < h; ++u) {
                    const bool up = lane & o;
                    const double give = up ? s[u] : s[u + h], keep = up ? s[u + h] : s[u];
                    s[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            double sum = s[0];
            for (; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            __syncwarp();  // the rows' first elements are written
            constexpr int LU = 32 / NU;
            const int lr = base + CL_NW * (lane / LU);
            const double2 pa{sum * tau, slab[lr * n + k + 1]};
            for (int q = lane % LU; q < C; q += LU) cl.map_shared_rank(pb, q)[par * n + c + C * lr] = pa;
        };
        for (int base = (k + 1 - c + C - 1) / C + wid; base < nrows;) {
            const int left = (nrows - base + CL_NW - 1) / CL_NW;
            if (left >= 8) {
                sweep(std::integral_constant<int, 8>{}, base);
                base += 8 * CL_NW;
            } else if (left >= 4) {
                sweep(std::integral_constant<int, 4>{}, base);
                base += 4 * CL_NW;
            } else if (left >= 2) {
                sweep(std::integral_constant<int, 2>{}, base);
                base += 2 * CL_NW;
            } else {
                sweep(std::integral_constant<int, 1>{}, base);
                base += CL_NW;
            }
        }
        if (C > 1) cl.sync();  // p and the column k + 1 have arrived
        else __syncthreads();
        double dot = 0.0;
        double2 pa[CL_EL];
#pragma unroll
        for (int e = 0; e < CL_EL; ++e) {
            const int r = tid + CL_THREADS * e;
            pa[e] = double2{0.0, 0.0};
            if (r >= n || r <= k) continue;
            pa[e] = pb[par * n + r];
            dot = fma(vk[r], pa[e].x, dot);
        }
        const double p1 = pb[par * n + k + 1].x;
        dot = warp_sum(dot);
        if (lane == 0) s_dot[par][wid] = dot;
        if (c == 0) {  // this step's outputs, while the others wait for the sum
            const double st = sqrt(tau);
#pragma unroll
            for (int e = 0; e < CL_EL; ++e) {
                const int r = tid + CL_THREADS * e;
                if (r < n && r > k) V[(long)k * n + r] = vk[r] * st;
                if (r == k) {
                    g.tri[2 * eo + k] = x[e];
                    g.tri[2 * eo + n + k] = alpha;
                }
            }
        }
        __syncthreads();
        double dtot = 0.0;
#pragma unroll
        for (int q = 0; q < CL_NW; ++q) dtot += s_dot[par][q];
        const double K = 0.5 * tau * dtot, w1 = p1 - K * v0;
#pragma unroll
        for (int e = 0; e < CL_EL; ++e) {
            const int r = tid + CL_THREADS * e;
            if (r >= n || r <= k) continue;
            const double vr = vk[r], wr = pa[e].x - K * vr;
            w[r] = wr;
            x[e] = pa[e].y - fma(v0, wr, w1 * vr);
        }
    }
    __syncthreads();
    // the last 2 x 2: row n-2 is this CTA's copy; element (n-1, n-1) its owner's, which lacks the last update
    if (c == 0 && n >= 2) {
#pragma unroll
        for (int e = 0; e < CL_EL; ++e) {
            const int r = tid + CL_THREADS * e;
            if (r == n - 2) g.tri[2 * eo + n - 2] = x[e];
            if (r == n - 1) g.tri[2 * eo + n + n - 2] = x[e];
        }
    }
    if (c == (n - 1) % C && tid == 0) {
        double last = slab[(long)((n - 1) / C) * n + n - 1];
        if (n >= 3) last -= 2.0 * v[((n - 3) & 1) * n + n - 1] * w[n - 1];
        g.tri[2 * eo + n - 1] = last;
        g.tri[2 * eo + n + n - 1] = 0.0;
    }
}

// ----------------------------------------------------------------------------
// Back-transformation U = H_0 ... H_{n-3} Z without forming Q: panels of
// BT_NB reflectors as block reflectors I - V T V^T (LAPACK dlarft, reflectors
// scaled to tau = 1, so T_ii = 1), applied from the last panel to the first.
// bt_tfactor_kernel forms -T of every panel from its Gram matrix; then each
// CTA of bt_apply_kernel keeps BT columns of Z in shared memory through all
// panels (columns of Z are independent), reading the panels from L2:
//   W = V^T Z,  W <- -T W,  Z += V W, all on the FP64 tensor cores.
// 2 n^3 operations and two launches for all blocks, against 4/3 n^3 + 2 n^3
// in 2 n steps of a cluster, or three GEMM launches per panel, and a product
// Q Z.  What bounds it: the FP64 pipe for the wide classes; reading V (twice
// per panel) from L2 for the narrow ones.  Anderson 1+5
// (blocks to 400 states): 0.13 ms, against 0.74 ms of the clusters' time and
// 0.09 ms of products; 7-site ring (blocks to 1225): 2.2 ms against 11; one
// block of 3070 states, whole eigensolve: 51 ms, of 3080, by GEMMs: 63.
// Reflector k is row k of V, right of the diagonal.
constexpr int BT_NB = 32, BT_THREADS = 256, BT_ROWS = 32;  // reflectors a panel, threads, rows of V a tile
constexpr int BT_LDV = BT_NB + 4;                          // 4 mod 16 doubles: conflict-free fragment loads
constexpr int BT_STAGES = 3;                               // tiles of V in flight or in use
// Columns of Z per CTA and the largest n whose slab fits 227 KB beside the
// tiles of V and W: 32 up to 697 states, 16 to 1489, 8 to 3073; larger blocks
// form Q by GEMMs (launch_big).
constexpr int BT_NCLS = 3;
constexpr int BT_COLS[BT_NCLS] = {32, 16, 8};
constexpr size_t BT_SMEM_MAX = 227 * 1024;
__host__ __device__ constexpr size_t bt_smem_doubles(int n, int C) {
    return (size_t)(n + BT_ROWS - 1) * C + BT_STAGES * BT_ROWS * BT_LDV + 2 * BT_NB * (C + 4);
}
// the largest n of the last class
constexpr int BT_MAX_DIM =
    (int)((BT_SMEM_MAX / sizeof(double) - bt_smem_doubles(0, BT_COLS[BT_NCLS - 1])) / BT_COLS[BT_NCLS - 1]);
static int bt_class(int n) {
    for (int q = 0; q < BT_NCLS; ++q)
        if (bt_smem_doubles(n, BT_COLS[q]) * sizeof(double) <= BT_SMEM_MAX) return q;
    return -1;
}
__host__ __device__ inline int bt_panels(int n) { return n > 2 ? (n - 2 + BT_NB - 1) / BT_NB : 0; }

struct BtItem {
    int block, at;    // block; its panel (T factors) or first column (application)
    int n, pad;
    long moff, toff;  // matrix offset; offset of the block's T factors in T
};

// tile of BT_ROWS rows of the panel's V from row r0, zero outside it: lane =
// row, warp = column mod 8
__device__ __forceinline__ void bt_load_v(double* dst, const double* V, int n, int k0, int r0) {
    static_assert(BT_ROWS == 32 && BT_THREADS == 256, "a warp loads 32 rows");
    const int gr = r0 + (threadIdx.x & 31), gk = k0 + (threadIdx.x >> 5);
    const double* src = V + (long)gk * n + gr;
    dst += (threadIdx.x & 31) * BT_LDV + (threadIdx.x >> 5);
    const int lim = gr < n ? min(gr, n - 2) : 0;  // columns of this row
#pragma unroll
    for (int u = 0; u < BT_NB / 8; ++u) {
        const bool in = gk + 8 * u < lim;
        cp_elem(dst + 8 * u, in ? src : V, in);
        src += 8L * n;
    }
}
__device__ __forceinline__ void bt_load_v_group(double* dst, const double* V, int n, int k0, int r0) {
    bt_load_v(dst, V, n, k0, r0);
    asm volatile("cp.async.commit_group;" ::: "memory");
}

__global__ void __launch_bounds__(BT_THREADS) bt_tfactor_kernel(const BtItem* items, const double* Vall, double* T) {
    __shared__ __align__(16) double vt[2][BT_ROWS * BT_LDV];
    __shared__ double G[BT_NB][BT_NB + 1];
    const BtItem it = items[blockIdx.x];
    const int n = it.n, k0 = it.at * BT_NB;
    const double* V = Vall + it.moff;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // G = V^T V: warp -> rows 8 (warp % 4), columns 16 (warp / 4)
    const int gi = 8 * (warp % 4), gj = 16 * (warp / 4);
    double2 acc[2] = {{0.0, 0.0}, {0.0, 0.0}};
    bt_load_v_group(vt[0], V, n, k0, k0 + 1);
    int buf = 0;
    for (int r0 = k0 + 1; r0 < n; r0 += BT_ROWS) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (r0 + BT_ROWS < n) bt_load_v_group(vt[buf ^ 1], V, n, k0, r0 + BT_ROWS);
        const double* v = vt[buf];
#pragma unroll
        for (int r = 0; r < BT_ROWS; r += 4) {
            const double a = v[(r + lane % 4) * BT_LDV + gi + lane / 4];
#pragma unroll
            for (int u = 0; u < 2; ++u) mma_f64(acc[u], a, v[(r + lane % 4) * BT_LDV + gj + 8 * u + lane / 4]);
        }
        buf ^= 1;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        G[gi + lane / 4][gj + 8 * u + 2 * (lane % 4)] = acc[u].x;
        G[gi + lane / 4][gj + 8 * u + 2 * (lane % 4) + 1] = acc[u].y;
    }
    __syncthreads();
    if (warp > 0) return;
    // T(0:i, i) = -T(0:i, 0:i) G(0:i, i), lane t owning row t of T; stored as -T
    double row[BT_NB];
#pragma unroll
    for (int i = 0; i < BT_NB; ++i) row[i] = 0.0;
#pragma unroll
    for (int i = 0; i < BT_NB; ++i) {
        double acc2 = 0.0;
#pragma unroll
        for (int s = 0; s < i; ++s) acc2 = fma(row[s], G[s][i], acc2);  // row[s] = 0 for s < lane
        row[i] = lane == i ? 1.0 : lane < i ? -acc2 : 0.0;
    }
    double* out = T + it.toff + (long)it.at * BT_NB * BT_NB;
#pragma unroll
    for (int i = 0; i < BT_NB; ++i) out[lane * BT_NB + i] = -row[i];
}

// Warps: MG groups of 8 MF rows of W, NG of 8 NF columns and two halves of the
// rows of Z for W = V^T Z; one 8-row strip at a time for Z += V W.  The tiles of
// V of all panels, each panel's forward and then backward, form one sequence
// that runs BT_STAGES - 1 tiles ahead of the products, through the panels' ends:
// a tile's products take 256 cycles, a third of the latency of L2.  Addresses
// advance by constants from tile to tile, since two warps a scheduler leave few
// issue slots (rows beyond the last get a tile's rows of zeros instead of a
// bound).  Columns of the slab are swizzled by row, so that fragments and pairs
// are read without bank conflicts.  7-site ring 3.6 -> 2.2 ms, 64 models of 3 to
// 6 bath sites 54 -> 33 against one tile ahead with addresses found per tile
// (tiles further ahead alone: 3.1 and 47).
template <int C>
__global__ void __launch_bounds__(BT_THREADS) bt_apply_kernel(const BtItem* items, const double* Vall, const double* T,
                                                               const double* Zall, double* Uall) {
    constexpr int LDW = C + 4, NF = C >= 16 ? 2 : 1, NG = C / (8 * NF), MG = 4 / NG, MF = 4 / MG;
    constexpr int TILE = BT_ROWS * BT_LDV;
    extern __shared__ __align__(16) double sh[];
    const BtItem it = items[blockIdx.x];
    const int n = it.n, c0 = it.at, nc = min(C, n - c0), np = bt_panels(n);
    const double* V = Vall + it.moff;
    const double* Z = Zall + it.moff;  // column-major
    double* vt = sh;                         // BT_STAGES tiles of V
    double* W = vt + BT_STAGES * TILE;       // 2 partial W; the first then holds -T W
    double* zs = W + 2 * BT_NB * LDW;        // n x C slab of Z
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int l4 = lane % 4, l8 = lane / 4;
    auto at = [&](int r, int c) { return r * C + (c ^ (C >= 16 ? (r & 1) << 3 | (r & 2) << 1 : (r & 2) << 1)); };
    auto tiles = [&](int q) { return (n - q * BT_NB - 1 + BT_ROWS - 1) / BT_ROWS; };
    int lq = np - 1, ls = 0, lnt = np > 0 ? tiles(lq) : 0, lstage = 0;  // the next tile to load: panel, step in it
    auto issue = [&]() {
        if (lq >= 0) {
            const int t = ls < lnt ? ls : 2 * lnt - 1 - ls;
            bt_load_v(vt + lstage * TILE, V, n, lq * BT_NB, lq * BT_NB + 1 + t * BT_ROWS);
            lstage = lstage + 1 == BT_STAGES ? 0 : lstage + 1;
            if (++ls == 2 * lnt) {
                ls = 0;
                if (--lq >= 0) lnt = tiles(lq);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int u = 0; u < BT_STAGES - 1; ++u) issue();
    for (long l = tid; l < (long)n * C; l += BT_THREADS) {
        const int c = (int)(l / n), r = (int)(l % n);
        zs[at(r, c)] = c < nc ? Z[(long)(c0 + c) * n + r] : 0.0;
    }
    for (int l = tid; l < (BT_ROWS - 1) * C; l += BT_THREADS) zs[n * C + l] = 0.0;  // rows of the last tile beyond n
    const int half = warp / 4, wm = (warp % 4) / NG * 8 * MF, wn = (warp % 4) % NG * 8 * NF;
    int stage = 0;
    // the next tile of the sequence; the one before it is free for every warp
    auto next = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(BT_STAGES - 2) : "memory");
        __syncthreads();
        issue();
        const double* v = vt + stage * TILE;
        stage = stage + 1 == BT_STAGES ? 0 : stage + 1;
        return v;
    };
    for (int q = np - 1; q >= 0; --q) {
        const int rb = q * BT_NB + 1, nt = tiles(q);
        // ---- W = V^T Z
        double2 w[MF][NF];
        double ta[BT_NB / 4][MF];
        const double* nT = T + it.toff + (long)q * BT_NB * BT_NB;
#pragma unroll
        for (int a = 0; a < MF; ++a) {
#pragma unroll
            for (int b = 0; b < NF; ++b) w[a][b] = double2{0.0, 0.0};
#pragma unroll
            for (int k = 0; k < BT_NB / 4; ++k) ta[k][a] = half == 0 ? nT[(wm + 8 * a + l8) * BT_NB + 4 * k + l4] : 0.0;
        }
        const double* zb[NF];  // rows 4 apart have the same swizzle
#pragma unroll
        for (int u = 0; u < NF; ++u) zb[u] = zs + at(rb + half * (BT_ROWS / 2) + l4, wn + 8 * u + l8);
        for (int t = 0; t < nt; ++t) {
            const double* v = next() + (half * (BT_ROWS / 2) + l4) * BT_LDV + wm + l8;
#pragma unroll
            for (int r = 0; r < BT_ROWS / 2; r += 4) {
                double a[MF], b[NF];
#pragma unroll
                for (int u = 0; u < MF; ++u) a[u] = v[r * BT_LDV + 8 * u];
#pragma unroll
                for (int u = 0; u < NF; ++u) b[u] = zb[u][r * C];
#pragma unroll
                for (int x = 0; x < MF; ++x)
#pragma unroll
                    for (int y = 0; y < NF; ++y) mma_f64(w[x][y], a[x], b[y]);
            }
#pragma unroll
            for (int u = 0; u < NF; ++u) zb[u] += BT_ROWS * C;
        }
#pragma unroll
        for (int x = 0; x < MF; ++x)
#pragma unroll
            for (int y = 0; y < NF; ++y)
                *reinterpret_cast<double2*>(&W[half * BT_NB * LDW + (wm + 8 * x + l8) * LDW + wn + 8 * y + 2 * l4]) = w[x][y];
        __syncthreads();
        // ---- W <- -T (W_0 + W_1), by the first four warps
#pragma unroll
        for (int x = 0; x < MF; ++x)
#pragma unroll
            for (int y = 0; y < NF; ++y) w[x][y] = double2{0.0, 0.0};
        if (half == 0) {
#pragma unroll
            for (int k = 0; k < BT_NB; k += 4) {
                double b[NF];
#pragma unroll
                for (int u = 0; u < NF; ++u) {
                    const int o = (k + l4) * LDW + wn + 8 * u + l8;
                    b[u] = W[o] + W[BT_NB * LDW + o];
                }
#pragma unroll
                for (int x = 0; x < MF; ++x)
#pragma unroll
                    for (int y = 0; y < NF; ++y) mma_f64(w[x][y], ta[k / 4][x], b[y]);
            }
        }
        __syncthreads();
        if (half == 0)
#pragma unroll
            for (int x = 0; x < MF; ++x)
#pragma unroll
                for (int y = 0; y < NF; ++y)
                    *reinterpret_cast<double2*>(&W[(wm + 8 * x + l8) * LDW + wn + 8 * y + 2 * l4]) = w[x][y];
        __syncthreads();
        // ---- Z += V W, tiles of V in reverse, strips of 8 rows: four warps a tile, C / 2 columns each
        constexpr int HC = C >= 16 ? C / 16 : 1;  // 8-column tiles a warp takes
        const int strip = 8 * (warp % 4), hc = C >= 16 ? warp / 4 * (C / 2) : 0;
        const bool mine = C >= 16 || warp < 4;
        double wb[BT_NB / 4][HC];
#pragma unroll
        for (int k = 0; k < BT_NB / 4; ++k)
#pragma unroll
            for (int y = 0; y < HC; ++y) wb[k][y] = W[(4 * k + l4) * LDW + hc + 8 * y + l8];
        double* zp[HC];
#pragma unroll
        for (int y = 0; y < HC; ++y) zp[y] = zs + at(rb + (nt - 1) * BT_ROWS + strip + l8, hc + 8 * y + 2 * l4);
        for (int t = nt - 1; t >= 0; --t) {
            const double* v = next() + (strip + l8) * BT_LDV + l4;
            if (mine) {
                double2 z[HC];
#pragma unroll
                for (int y = 0; y < HC; ++y) z[y] = *reinterpret_cast<double2*>(zp[y]);
#pragma unroll
                for (int k = 0; k < BT_NB / 4; ++k) {
                    const double a = v[4 * k];
#pragma unroll
                    for (int y = 0; y < HC; ++y) mma_f64(z[y], a, wb[k][y]);
                }
#pragma unroll
                for (int y = 0; y < HC; ++y) {
                    *reinterpret_cast<double2*>(zp[y]) = z[y];
                    zp[y] -= BT_ROWS * C;
                }
            }
        }
    }
    __syncthreads();
    double* U = Uall + it.moff;
    for (long l = tid; l < (long)n * C; l += BT_THREADS) {
        const int r = (int)(l / C), c = (int)(l % C);
        if (c < nc) U[(long)r * n + c0 + c] = zs[at(r, c)];
    }
}

// ----------------------------------------------------------------------------
// Tridiagonal stage.  T (diagonal d, sub-diagonal e) is split into unreduced
// pieces where |e_i| <= eps (|d_i| + |d_i+1|) or |e_i| <= 8 eps ||T|| (a
// perturbation of T of the size of the Householder stage's own backward
// error).  Exact degeneracies of H show up as such splits, so eigenvectors of
// different pieces are orthogonal by support.
//   * eigenvalues: multisection with Sturm counts (Golub & Van Loan, 8.4.1);
//   * eigenvectors: two steps of inverse iteration, one thread per
//     eigenvalue (Golub & Van Loan, 8.2.2).  Each solve factors T - lambda I
//     by Gaussian elimination with partial pivoting.  In a chain of
//     eigenvalues whose neighbours are closer than 1e-4 ||T|| the shifts are
//     nudged apart, so coincident eigenvalues get distinct vectors, and a
//     second kernel orthogonalises each member (modified Gram-Schmidt, twice)
//     against the earlier members closer than 1e-4 ||T||; mixing only among
//     such close eigenvalues keeps the residuals at the eps ||T|| level.  The
//     start vector is a fixed hash of (index, row).
struct TriItem {
    int block, j0, j1, pad;
    long soff;  // vector_kernel: this CTA's scratch, 4 n TRI_THREADS doubles at S + soff
};

struct TriArgs {
    const TriItem* items;
    const int* dims;
    const long* moff;
    const long* eoff;
    const double* tri;  // per block: d (n), e (n)
    double* lam;        // per block: eigenvalues, ascending inside each piece
    int* sb;            // per block: 2 n ints (first and last row of the piece)
    int* rank;          // per block: n ints (position in the ascending order)
    double *Z, *Zq;     // per block: n x n column-major eigenvectors of T, sorted: Z, or Zq where Q was formed
    double* S;          // per vector_kernel CTA: 4 arrays of n x TRI_THREADS, thread-interleaved
    double* E;          // eigenvalues, ascending
    int* status;
};

constexpr int TRI_THREADS = 32;  // vector_kernel: one warp per CTA, so the CTAs spread over all SMs
constexpr double EPS = 2.220446049250313e-16;
constexpr double SAFE_MIN = 2.2250738585072014e-308;
constexpr double SPLIT_ABS = 8.0;   // absolute split threshold, units of eps ||T||
constexpr double CHAIN_TOL = 1e-4;  // chain / orthogonalisation window, units of ||T||
constexpr int INV_ITERS = 2;        // inverse iterations per eigenvector

// Loads d and e of one block into shared memory, zeroes the split points and
// returns ||T|| (max row sum); every thread of the CTA must call it.
__device__ double load_tri(const double* tri, long eo, int n, double* d, double* e) {
    __shared__ double red[32];
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        d[i] = tri[2 * eo + i];
        e[i] = (i < n - 1) ? tri[2 * eo + n + i] : 0.0;
    }
    __syncthreads();
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        m = fmax(m, fabs(d[i]) + fabs(e[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    double tn = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tn = fmax(tn, red[w]);
    for (int i = threadIdx.x; i < n - 1; i += blockDim.x)
        if (fabs(e[i]) <= EPS * (fabs(d[i]) + fabs(d[i + 1])) || fabs(e[i]) <= SPLIT_ABS * EPS * tn) e[i] = 0.0;
    __syncthreads();
    return tn;
}


// Eigenvalues by multisection with Sturm counts: `lp` lanes (a power of two)
// take the counts at lp equally spaced interior points of their eigenvalue's
// bracketing interval, narrowing it lp + 1-fold a round.  One lane (bisection)
// needs the fewest counts, 53 sweeps of T per eigenvalue; 32 lanes need
// 32 x 11 but only 11 in a row.  bisect_lanes() takes as many lanes as keep
// the GPU's threads busy and no more.
//
// A count is the number of sign changes of the leading principal minors
//   p_i = (d_i - x) p_i-1 - e_i-1^2 p_i-2
// (Golub & Van Loan, 8.4.1), T scaled by a power of two to norm about one and
// the pair (p_i, p_i-1) rescaled by a power of two every eight steps: a step
// grows it at most fivefold and shrinks it at most by the smallest kept e^2,
// so eight steps stay far inside the double range.  An exact zero counts as
// positive; the sum over it and its neighbour is that of either sign.  One
// step is three FP64 operations with one FMA in the dependent chain, where the
// quotient form has a division there.  64 models of 3 to 6 bath sites
// (312 832 eigenvalues): 86 -> 4.6 ms; Anderson 1+5 (4096
// eigenvalues): 0.57 -> 0.18 ms.
constexpr int BIS_THREADS = 256;

// lanes per eigenvalue for `total` eigenvalues: 148 SMs x 1024 threads
__host__ inline int bisect_lanes(long total) {
    int lp = 32;
    while (lp > 1 && total * lp > 148L * 1024) lp /= 2;
    return lp;
}

// number of eigenvalues of T[a..b] below x (e2: squared sub-diagonal)
__device__ int sturm(const double* d, const double* e2, int a, int b, double x) {
    double p0 = 1.0, p1 = d[a] - x;
    int h1 = __double2hiint(p1);
    unsigned cnt = (unsigned)h1 >> 31;
    auto step = [&](int i) {
        const double pn = fma(d[i] - x, p1, -(e2[i - 1] * p0));
        const int hn = __double2hiint(pn);
        cnt += (unsigned)(hn ^ h1) >> 31;
        p0 = p1;
        p1 = pn;
        h1 = hn;
    };
    int i = a + 1;
    for (; i + 7 <= b; i += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) step(i + u);
        const int ex = max(h1 & 0x7ff00000, __double2hiint(p0) & 0x7ff00000);
        const double sc = __hiloint2double(0x7fe00000 - min(ex, 0x7fd00000), 0);
        p0 *= sc;
        p1 *= sc;
    }
    for (; i <= b; ++i) step(i);
    return (int)cnt;
}

__global__ void __launch_bounds__(BIS_THREADS) bisect_kernel(TriArgs g, const TriItem* bitems, int lp) {
    extern __shared__ double sh[];
    __shared__ int s_first[BIS_THREADS], s_last[BIS_THREADS];  // split points around each thread's share of the rows
    const TriItem it = bitems[blockIdx.x];
    const int n = g.dims[it.block];
    const long eo = g.eoff[it.block];
    double* d = sh;
    double* e = sh + n;
    const double tn = load_tri(g.tri, eo, n, d, e);
    const int tid = threadIdx.x, lane = tid & 31;
    // piece of a row: the nearest split at or before it, and at or after it
    const int per = (n + BIS_THREADS - 1) / BIS_THREADS;
    const int c0 = tid * per, c1 = min(n, c0 + per);
    int fs = -1, ls = n;
    for (int i = c0; i < c1; ++i)
        if (i == 0 || e[i - 1] == 0.0) fs = i;
    for (int i = c1 - 1; i >= c0; --i)
        if (i == n - 1 || e[i] == 0.0) ls = i;
    s_first[tid] = fs;
    s_last[tid] = ls;
    __syncthreads();
    for (int o = 1; o < BIS_THREADS; o *= 2) {
        const int x = tid >= o ? max(s_first[tid], s_first[tid - o]) : s_first[tid];
        const int y = tid + o < BIS_THREADS ? min(s_last[tid], s_last[tid + o]) : s_last[tid];
        __syncthreads();
        s_first[tid] = x;
        s_last[tid] = y;
        __syncthreads();
    }
    const int j = it.j0 + tid / lp, gl = tid % lp;
    const bool active = j < it.j1;
    int a = 0, b = 0;
    if (active) {
        const int t = j / per;
        for (a = j; a >= t * per && !(a == 0 || e[a - 1] == 0.0); --a) {}
        if (a < t * per) a = s_first[t - 1];
        const int end = min(n, (t + 1) * per);
        for (b = j; b < end && !(b == n - 1 || e[b] == 0.0); ++b) {}
        if (b == end) b = s_last[t + 1];
    }
    // Gershgorin interval of the piece
    double lo = 1e300, hi = -1e300;
    if (active)
        for (int i = a + gl; i <= b; i += lp) {
            const double r = (i > a ? fabs(e[i - 1]) : 0.0) + (i < b ? fabs(e[i]) : 0.0);
            lo = fmin(lo, d[i] - r);
            hi = fmax(hi, d[i] + r);
        }
    for (int o = lp / 2; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    // scale T to norm [1, 2) and square the sub-diagonal
    const int te = tn > 0.0 ? max(-1000, min(1000, ilogb(tn))) : 0;
    const double sc = scalbn(1.0, -te);
    __syncthreads();
    for (int i = tid; i < n; i += BIS_THREADS) {
        const double ei = e[i] * sc;
        d[i] *= sc;
        e[i] = ei * ei;
    }
    __syncthreads();
    lo *= sc;
    hi *= sc;
    const double gn = fmax(fabs(lo), fabs(hi));
    const double w = 2.0 * EPS * gn + SAFE_MIN;
    lo -= w;
    hi += w;
    const double atol = 0.25 * EPS * gn + SAFE_MIN;
    const int k = j - a;
    const unsigned shift = lane / lp * lp, mask = lp == 32 ? 0xffffffffu : (1u << lp) - 1u;
    const double part = 1.0 / (lp + 1);
    // the lanes of an eigenvalue hold the same lo, hi; those of a warp leave together
    for (int round = 0; round < 128; ++round) {
        const double step = (hi - lo) * part;
        const bool go = active && hi - lo > atol + 2.0 * EPS * fmin(fabs(lo), fabs(hi)) && lo + step > lo &&
                        lo + step * lp < hi;  // else converged, or at the resolution of doubles
        if (!__any_sync(0xffffffffu, go)) break;
        int cnt = 0;
        if (go) cnt = sturm(d, e, a, b, lo + step * (gl + 1));
        // counts grow with x: the eigenvalue lies between point `below` and `below + 1`
        const unsigned vote = __ballot_sync(0xffffffffu, go && cnt <= k);
        if (go) {
            const int below = __popc((vote >> shift) & mask);
            const double nlo = (below > 0) ? lo + step * below : lo;
            const double nhi = (below < lp) ? lo + step * (below + 1) : hi;
            lo = nlo;
            hi = nhi;
        }
    }
    if (active && gl == 0) {
        g.lam[eo + j] = scalbn(0.5 * (lo + hi), te);
        g.sb[2 * eo + j] = a;
        g.sb[2 * eo + n + j] = b;
    }
}

// pseudo-random start vector entry in [-1, 1) for eigen-index j, row i
__device__ __forceinline__ double start_entry(int j, int i) {
    unsigned x = (unsigned)j * 0x9E3779B1u + (unsigned)i * 0x85EBCA77u + 0x165667B1u;
    x ^= x >> 15;
    x *= 0x2C1B3C6Du;
    x ^= x >> 12;
    x *= 0x297A2D39u;
    x ^= x >> 15;
    return (double)x * (2.0 / 4294967296.0) - 1.0;
}

// z := (T[a..b] - lm I)^-1 z by Gaussian elimination with partial pivoting;
// the factorisation and the forward elimination share one sweep, the upper
// factor's three diagonals are kept in u1, u2, u3 for the back substitution.
// Pivots smaller than pfloor in magnitude are replaced by +-pfloor.
// Both sweeps are a chain of dependent divisions; the values the chain
// passes on stay in registers, and the vector entries each sweep reads are
// loaded LU_BATCH rows ahead, so a batch waits for memory once.  Entry i of
// each vector is at index i * st: the lanes of a warp interleave their
// vectors, so a warp at the same row reads and writes one contiguous segment.
constexpr int LU_BATCH = 8;

__device__ void lu_solve(const double* d, const double* e, int a, int b, double lm, double pfloor,
                         double* __restrict__ z, double* __restrict__ u1, double* __restrict__ u2,
                         double* __restrict__ u3, int st) {
    double p = d[a] - lm, q = (a < b) ? e[a] : 0.0;
    double zk = z[(long)a * st];
    for (int k0 = a; k0 < b; k0 += LU_BATCH) {
        double zn[LU_BATCH];
#pragma unroll
        for (int t = 0; t < LU_BATCH; ++t)
            if (k0 + t < b) zn[t] = z[(long)(k0 + t + 1) * st];
#pragma unroll
        for (int t = 0; t < LU_BATCH; ++t) {
            const int k = k0 + t;
            if (k >= b) break;
            const double sub = e[k], dn = d[k + 1] - lm, en = (k + 1 < b) ? e[k + 1] : 0.0;
            const double zk1 = zn[t];
            // row interchange when the sub-diagonal entry is the larger pivot; both
            // cases share one division and are selected without branching
            const bool sw = fabs(sub) > fabs(p);
            const double num = sw ? p : sub, den = sw ? sub : p;
            const double l = (den != 0.0) ? num / den : 0.0;
            const double w1 = sw ? sub : p, w2 = sw ? dn : q, w3 = sw ? en : 0.0;
            const double np = sw ? q - l * dn : dn - l * q;
            const double nq = sw ? -l * en : en;
            const double zout = sw ? zk1 : zk;
            const double znext = sw ? zk - l * zk1 : zk1 - l * zk;
            const long o = (long)k * st;
            u1[o] = w1;
            u2[o] = w2;
            u3[o] = w3;
            z[o] = zout;
            zk = znext;
            p = np;
            q = nq;
        }
    }
    // back substitution; x1, x2 carry the two solution entries below row k
    double x1 = 0.0, x2 = 0.0;
    for (int k0 = b; k0 >= a; k0 -= LU_BATCH) {
        double v1[LU_BATCH], v2[LU_BATCH], v3[LU_BATCH], vz[LU_BATCH];
#pragma unroll
        for (int t = 0; t < LU_BATCH; ++t) {
            const int k = k0 - t;
            if (k < a) break;
            const long o = (long)k * st;
            v1[t] = (k == b) ? p : u1[o];
            vz[t] = (k == b) ? zk : z[o];
            v2[t] = (k + 1 <= b) ? u2[o] : 0.0;
            v3[t] = (k + 2 <= b) ? u3[o] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < LU_BATCH; ++t) {
            const int k = k0 - t;
            if (k < a) break;
            double piv = v1[t];
            if (fabs(piv) < pfloor) piv = (piv >= 0.0) ? pfloor : -pfloor;
            double r = vz[t];
            if (k + 1 <= b) r -= v2[t] * x1;
            if (k + 2 <= b) r -= v3[t] * x2;
            const double xk = r / piv;
            z[(long)k * st] = xk;
            x2 = x1;
            x1 = xk;
        }
    }
}

// z /= ||z|| over rows a..b (stride st); false when the norm is zero or not finite
__device__ bool normalize(double* z, int a, int b, int st) {
    double nn = 0.0;
    for (int i = a; i <= b; ++i) nn = fma(z[(long)i * st], z[(long)i * st], nn);
    if (!(nn > 0.0) || !isfinite(nn)) return false;
    const double inv = rsqrt(nn);
    for (int i = a; i <= b; ++i) z[(long)i * st] *= inv;
    return true;
}

// One thread per eigenvalue, the same work in every thread: two steps of
// inverse iteration.  Within a chain (neighbours closer than CHAIN_TOL ||T||)
// the shifts are nudged apart so coincident eigenvalues start from distinct
// shifts; ortho_kernel then orthogonalises the members of each chain.
__global__ void __launch_bounds__(TRI_THREADS) vector_kernel(TriArgs g) {
    extern __shared__ double sh[];
    const TriItem it = g.items[blockIdx.x];
    const int n = g.dims[it.block];
    const long eo = g.eoff[it.block], mo = g.moff[it.block];
    double* d = sh;
    double* e = sh + n;
    double* lam = sh + 2 * n;
    const double tn = load_tri(g.tri, eo, n, d, e);
    for (int i = threadIdx.x; i < n; i += blockDim.x) lam[i] = g.lam[eo + i];
    __syncthreads();
    const double ortol = CHAIN_TOL * tn;
    const double pfloor = (tn > 0.0) ? EPS * tn : 1.0;
    const int* sa = g.sb + 2 * eo;
    const int* sbe = sa + n;
    double* Zb = (n > BT_MAX_DIM ? g.Zq : g.Z) + mo;
    // this thread's working vector and LU diagonals, interleaved with the CTA's other threads
    const int st = blockDim.x;
    double* zt = g.S + it.soff + threadIdx.x;
    double* u1 = zt + (long)n * st;
    double* u2 = u1 + (long)n * st;
    double* u3 = u2 + (long)n * st;
    for (int j = it.j0 + threadIdx.x; j < it.j1; j += blockDim.x) {
        const int a = sa[j], b = sbe[j];
        // shift: the eigenvalue, raised above its chain predecessor's shift where they coincide
        int h = j;
        while (h > a && lam[h] - lam[h - 1] <= ortol) --h;
        double lm = -1e308;
        for (int t = h; t <= j; ++t) {
            const double lt = lam[t], sep = 10.0 * EPS * fmax(fabs(lt), 1e-3 * tn);
            lm = (t > h && lt < lm + sep) ? lm + sep : lt;
        }
        int rk = 0;
        for (int i = 0; i < n; ++i) rk += (lam[i] < lam[j]) || (lam[i] == lam[j] && i < j);
        g.rank[eo + j] = rk;
        g.E[eo + rk] = lam[j];
        double* z = Zb + (long)rk * n;
        bool ok = true;
        if (a == b) {
            for (int i = 0; i < n; ++i) z[i] = (i == a) ? 1.0 : 0.0;
        } else {
            for (int i = a; i <= b; ++i) zt[(long)i * st] = start_entry(j, i);
            for (int t = 0; t < INV_ITERS && ok; ++t) {
                lu_solve(d, e, a, b, lm, pfloor, zt, u1, u2, u3, st);
                ok = normalize(zt, a, b, st);
            }
            for (int i = 0; i < n; ++i) z[i] = (i >= a && i <= b) ? zt[(long)i * st] : 0.0;
        }
        if (!ok) atomicExch(g.status, PGX_ERR_NUMERIC);
    }
}

// The CTA's warp orthogonalises each chain whose head lies in its range:
// modified Gram-Schmidt (two passes) of every member against its close
// predecessors, the dot products and updates spread over the lanes (a chain
// of a symmetry multiplet can hold dozens of vectors of thousands of states).
__global__ void __launch_bounds__(TRI_THREADS) ortho_kernel(TriArgs g) {
    extern __shared__ double sh[];
    const TriItem it = g.items[blockIdx.x];
    const int n = g.dims[it.block];
    const long eo = g.eoff[it.block], mo = g.moff[it.block];
    double* d = sh;
    double* e = sh + n;
    double* lam = sh + 2 * n;
    const double tn = load_tri(g.tri, eo, n, d, e);
    for (int i = threadIdx.x; i < n; i += blockDim.x) lam[i] = g.lam[eo + i];
    __syncthreads();
    const int lane = threadIdx.x;
    const double ortol = CHAIN_TOL * tn;
    const int* sa = g.sb + 2 * eo;
    const int* sbe = sa + n;
    const int* rank = g.rank + eo;
    double* Zb = (n > BT_MAX_DIM ? g.Zq : g.Z) + mo;
    for (int j = it.j0; j < it.j1; ++j) {
        const int a = sa[j], b = sbe[j];
        if (j > a && lam[j] - lam[j - 1] <= ortol) continue;  // not the head of a chain
        bool ok = true;
        for (int jj = j + 1; jj <= b && lam[jj] - lam[jj - 1] <= ortol; ++jj) {
            double* z = Zb + (long)rank[jj] * n;
            for (int pass = 0; pass < 2 && ok; ++pass) {
                for (int pp = jj - 1; pp >= j && lam[jj] - lam[pp] <= ortol; --pp) {
                    const double* qv = Zb + (long)rank[pp] * n;
                    double dot = 0.0;
                    for (int i = a + lane; i <= b; i += TRI_THREADS) dot = fma(qv[i], z[i], dot);
                    dot = warp_sum(dot);
                    for (int i = a + lane; i <= b; i += TRI_THREADS) z[i] = fma(-dot, qv[i], z[i]);
                }
                double nn = 0.0;
                for (int i = a + lane; i <= b; i += TRI_THREADS) nn = fma(z[i], z[i], nn);
                nn = warp_sum(nn);
                if (!(nn > 0.0) || !isfinite(nn)) {
                    ok = false;
                } else {
                    const double inv = rsqrt(nn);
                    for (int i = a + lane; i <= b; i += TRI_THREADS) z[i] *= inv;
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicExch(g.status, PGX_ERR_NUMERIC);
    }
}

// ----------------------------------------------------------------------------
// Complex Hermitian blocks.  H = R + iI (R symmetric, I antisymmetric) has the
// real symmetric embedding [[R, -I], [I, R]] of twice the size; every
// eigenvalue of H appears twice in it, and for a real eigenvector [a; b] of
// the pair, a + ib is an eigenvector of H (unit norm).  The embedding is
// diagonalised by the real stages above; cx_extract_kernel then forms the
// complex eigenvectors.

// block b of H (complex, row-major n x n) -> block b of the embedding (2n x 2n)
__global__ void cx_embed_kernel(const int* dims, const long* moff, const long* moff2, const double* H, double* H2) {
    const int b = blockIdx.y, n = dims[b];
    const cd* Hb = reinterpret_cast<const cd*>(H) + moff[b];
    double* E = H2 + moff2[b];
    const long nn = (long)n * n, n2 = 2L * n;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < nn; e += (long)gridDim.x * blockDim.x) {
        const int i = (int)(e / n), j = (int)(e % n);
        const cd h = Hb[e];
        E[i * n2 + j] = h.x;
        E[i * n2 + n + j] = -h.y;
        E[(n + i) * n2 + j] = h.y;
        E[(n + i) * n2 + n + j] = h.x;
    }
}

// One thread per cluster of equal eigenvalues of the embedding (2m values):
// the m complex eigenvectors of H are taken from the 2m candidates a + ib by
// modified Gram-Schmidt (twice), keeping those with a residual norm above 1/2.
// A cluster is a run of consecutive eigenvalues closer than tol.
__global__ void cx_extract_kernel(const int* dims, const long* moff, const long* eoff, const long* moff2,
                                  const long* eoff2, const double* E2, const double* U2, double* E, cd* U, double tol,
                                  int* status) {
    const int b = blockIdx.x, n = dims[b];
    const long n2 = 2L * n;
    const double* Eb2 = E2 + eoff2[b];
    const double* Ub2 = U2 + moff2[b];
    double* Eb = E + eoff[b];
    cd* Ub = U + moff[b];
    for (int j = threadIdx.x; j < 2 * n; j += blockDim.x) {
        if (j > 0 && Eb2[j] - Eb2[j - 1] <= tol) continue;  // not the start of a cluster
        int jend = j;
        while (jend + 1 < 2 * n && Eb2[jend + 1] - Eb2[jend] <= tol) ++jend;
        const int sz = jend - j + 1, m = sz / 2, c0 = j / 2;
        if ((sz & 1) || (j & 1)) {
            atomicExch(status, PGX_ERR_NUMERIC);
            continue;
        }
        int acc = 0;
        for (int k = 0; k < sz && acc < m; ++k) {
            cd* v = Ub + (c0 + acc);  // column c0 + acc, stride n
            for (int i = 0; i < n; ++i) v[(long)i * n] = cd{Ub2[i * n2 + j + k], Ub2[(n + i) * n2 + j + k]};
            for (int pass = 0; pass < 2; ++pass)
                for (int q = 0; q < acc; ++q) {
                    const cd* u = Ub + (c0 + q);
                    double px = 0.0, py = 0.0;  // u^H v
                    for (int i = 0; i < n; ++i) {
                        const cd a = u[(long)i * n], c = v[(long)i * n];
                        px += a.x * c.x + a.y * c.y;
                        py += a.x * c.y - a.y * c.x;
                    }
                    for (int i = 0; i < n; ++i) {
                        const cd a = u[(long)i * n];
                        v[(long)i * n].x -= px * a.x - py * a.y;
                        v[(long)i * n].y -= px * a.y + py * a.x;
                    }
                }
            double nn = 0.0;
            for (int i = 0; i < n; ++i) nn += abs2(v[(long)i * n]);
            if (nn > 0.25) {
                const double inv = rsqrt(nn);
                for (int i = 0; i < n; ++i) v[(long)i * n] = v[(long)i * n] * inv;
                Eb[c0 + acc] = Eb2[j + 2 * acc];
                ++acc;
            }
        }
        if (acc < m) atomicExch(status, PGX_ERR_NUMERIC);
    }
}

}  // namespace

static long total_dim(const std::vector<int>& dims) {
    long s = 0;
    for (int n : dims) s += n;
    return s;
}

// Work items, largest blocks first: vector_kernel takes TRI_THREADS
// eigen-indices per CTA, bisect_kernel BIS_THREADS / bisect_lanes; both lists
// go into one descriptor upload (vector items, then bisection items).
static void tri_plan(const std::vector<int>& dims, std::vector<TriItem>& items, size_t* n_vec = nullptr) {
    std::vector<int> order(dims.size());
    for (size_t b = 0; b < dims.size(); ++b) order[b] = (int)b;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dims[x] > dims[y]; });
    long soff = 0;
    for (int b : order)
        for (int j0 = 0; j0 < dims[b]; j0 += TRI_THREADS) {
            items.push_back(TriItem{b, j0, std::min(dims[b], j0 + TRI_THREADS), 0, soff});
            soff += 4L * dims[b] * TRI_THREADS;
        }
    if (n_vec) *n_vec = items.size();
    const int per = BIS_THREADS / bisect_lanes(total_dim(dims));
    for (int b : order)
        for (int j0 = 0; j0 < dims[b]; j0 += per) items.push_back(TriItem{b, j0, std::min(dims[b], j0 + per), 0, 0});
}

constexpr int CL_NCLS = 5;
constexpr int CL_SIZES[CL_NCLS] = {1, 2, 4, 8, 16};
constexpr size_t CL_SMEM_MAX = 226 * 1024;  // dynamic shared memory per CTA (the static part is small)

// The cluster class of an n x n block, or -1 (the block then takes the
// large-block path): the smallest cluster whose shared memory holds the
// block.  16 CTAs (a non-portable cluster size) only where 8 do not suffice
// (453 to 513 states): at 400 states the per-step cost is set by the cluster
// barriers, and 16-CTA clusters were measured slower than 8-CTA ones there.
static int cluster_class(int n) {
    if (n > CL_MAX_DIM) return -1;
    for (int i = 0; i < CL_NCLS; ++i)
        if (cluster_smem_doubles(n, CL_SIZES[i]) * sizeof(double) <= CL_SMEM_MAX) return i;
    return -1;
}

// Whether a block may take the large-block path: beyond the clusters, or of a
// size that needs 16 CTAs, which not every device can schedule.
static bool maybe_big(int n) { return cluster_class(n) < 0 || CL_SIZES[cluster_class(n)] > 8; }

// Back-transformation plan: the T factors' items (one per panel), then the
// column slabs of each class, largest blocks first.  first[q] is where list q
// starts (0: T factors, 1 + c: class c), first[BT_NCLS + 1] the total; nmax[c]
// the largest block of class c.
struct BtPlan {
    std::vector<BtItem> items;
    size_t first[BT_NCLS + 2];
    int nmax[BT_NCLS];
};
static BtPlan bt_plan(const std::vector<int>& dims) {
    std::vector<int> order(dims.size());
    std::vector<long> moff(dims.size()), toff(dims.size());
    long m = 0, t = 0;
    for (size_t b = 0; b < dims.size(); ++b) {
        order[b] = (int)b;
        moff[b] = m;
        toff[b] = t;
        m += (long)dims[b] * dims[b];
        if (bt_class(dims[b]) >= 0) t += (long)bt_panels(dims[b]) * BT_NB * BT_NB;
    }
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dims[x] > dims[y]; });
    BtPlan p;
    auto add = [&](int b, int at) {
        p.items.push_back(BtItem{b, at, dims[b], 0, moff[b], toff[b]});
    };
    p.first[0] = 0;
    for (int b : order)
        if (bt_class(dims[b]) >= 0)
            for (int q = 0; q < bt_panels(dims[b]); ++q) add(b, q);
    for (int c = 0; c < BT_NCLS; ++c) {
        p.first[c + 1] = p.items.size();
        p.nmax[c] = 0;
        for (int b : order) {
            if (bt_class(dims[b]) != c) continue;
            p.nmax[c] = std::max(p.nmax[c], dims[b]);
            for (int j = 0; j < dims[b]; j += BT_COLS[c]) add(b, j);
        }
    }
    p.first[BT_NCLS + 1] = p.items.size();
    return p;
}
template <int C>
static void launch_bt_apply(const BtItem* items, size_t n, int nmax, const double* V, const double* T, const double* Z,
                            double* U, cudaStream_t st) {
    const size_t smem = bt_smem_doubles(nmax, C) * sizeof(double);
    PGX_CUDA(cudaFuncSetAttribute(bt_apply_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BT_SMEM_MAX));
    bt_apply_kernel<C><<<(unsigned)n, BT_THREADS, smem, st>>>(items, V, T, Z, U);
    check_launch("bt_apply_kernel");
}

// doubles of vector_kernel scratch (EighDev::S); the large-block path uses
// the same buffer before the vector stage (one scratch per large block)
size_t eigh_vec_scratch_doubles(const std::vector<int>& dims) {
    size_t s = 0, big = 0;
    for (int n : dims) {
        // the vectors' scratch, later the T factors
        s += std::max(4 * (size_t)n * TRI_THREADS * ((n + TRI_THREADS - 1) / TRI_THREADS),
                      (size_t)bt_panels(n) * BT_NB * BT_NB);
        if (maybe_big(n)) big += (size_t)bhh_scratch_doubles(n);
    }
    return std::max<size_t>(std::max(s, big), 1);
}


// Householder stage plan: the block list of each cluster size (largest
// blocks first) and the blocks left to the large-block path.
struct HhPlan {
    std::vector<int> cls[CL_NCLS];
    std::vector<int> global;
};

static HhPlan hh_plan(const std::vector<int>& dims) {
    std::vector<int> order(dims.size());
    for (size_t b = 0; b < dims.size(); ++b) order[b] = (int)b;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dims[x] > dims[y]; });
    HhPlan h;
    for (int b : order) {
        const int q = cluster_class(dims[b]);
        if (q < 0) h.global.push_back(b);
        else h.cls[q].push_back(b);
    }
    return h;
}

// the blocks that may take the large-block path, largest first
static std::vector<int> big_blocks(const std::vector<int>& dims) {
    std::vector<int> big;
    for (size_t b = 0; b < dims.size(); ++b)
        if (maybe_big(dims[b])) big.push_back((int)b);
    std::stable_sort(big.begin(), big.end(), [&](int x, int y) { return dims[x] > dims[y]; });
    return big;
}

// descriptor bytes: bisection items, one int per block (Householder lists);
// with large blocks also their descriptors
static size_t big_desc_bytes(const std::vector<int>& dims) {
    const size_t nb = big_blocks(dims).size();
    if (nb == 0) return 0;
    return 8 + nb * sizeof(BigBlk);
}
size_t eigh_item_bytes(const std::vector<int>& dims) {
    std::vector<TriItem> items;
    tri_plan(dims, items);
    return items.size() * sizeof(TriItem) + bt_plan(dims).items.size() * sizeof(BtItem) + dims.size() * sizeof(int) +
           big_desc_bytes(dims);
}

size_t eigh_gemm_bytes(const std::vector<int>& dims, size_t* tiles_bytes) {
    size_t np = dims.size();
    size_t panels = 0;
    for (int b : big_blocks(dims)) panels += (size_t)bhh_panels(dims[b]);
    np = std::max(np, panels);
    if (tiles_bytes) *tiles_bytes = gemm_index_bytes(np);
    return std::max<size_t>(np, 1) * sizeof(GemmProblem<double, double, double>);
}

// The large-block Householder path (see bhh_col_kernel) on stream st.
// big: the blocks, largest first; d_blk: their device list (uploaded by the
// caller).
static void launch_big(const EighDev& d, const std::vector<int>& dims, const std::vector<long>& moff,
                       const std::vector<int>& big, const BigBlk* d_blk, cudaStream_t st) {
    const int nbig = (int)big.size();
    std::vector<long> boff(nbig);
    long o = 0;
    for (int i = 0; i < nbig; ++i) {
        boff[i] = o;
        o += bhh_scratch_doubles(dims[big[i]]);
    }
    const int nmax = dims[big[0]];
    // blocks with a reflector in column j: a prefix of the list
    auto nact = [&](int j) {
        int c = 0;
        while (c < nbig && dims[big[c]] - 2 > j) ++c;
        return c;
    };
    BigArgs a{};
    a.blk = d_blk;
    a.A = d.A;
    a.Zc = d.Zc;
    a.S = d.S;
    a.tri = d.tri;
    a.slots = 0;
    double fl = 0.0, by = 0.0;
    for (int b : big) {
        const double n = dims[b];
        fl += 8.0 / 3.0 * n * n * n;
        by += 16.0 * n * n + 16.0 * n;
    }
    ProfRange pr("eigh_blocked_householder", st, fl, by);
    for (int b : big)
        PGX_CUDA(cudaMemcpyAsync(d.A + moff[b], d.H + moff[b], (size_t)dims[b] * dims[b] * sizeof(double),
                                 cudaMemcpyDeviceToDevice, st));
    // The column and product kernels alternate, each launched while the one
    // before it drains (it waits for that one's results itself).
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.stream = st;
    auto col_step = [&]() {
        // CTAs per block: eight rows a warp, as long as all blocks are
        // resident at once (two CTAs per SM)
        const int lo = (a.fin >= 0 ? a.fin + 1 : a.col) & ~7;
        int cs = std::max(1, (int)ceil_div(nmax - lo, BHH_COL_THREADS / 4));
        while (cs > 1 && a.nact * cs > (a.slots ? 1 : 2) * 148) cs = (cs + 1) / 2;
        cfg.gridDim = dim3((unsigned)cs, (unsigned)a.nact);
        cfg.blockDim = dim3(BHH_COL_THREADS);
        ProfRange r1("bhh_col_kernel", st, 0.0, 0.0);
        PGX_CUDA(cudaLaunchKernelEx(&cfg, a.slots ? bhh_col_kernel<true> : bhh_col_kernel<false>, a));
        check_launch("bhh_col_kernel");
    };
    auto symv_step = [&](int rows, long all_rows, double bytes) {
        if (a.slots) {
            cfg.gridDim = dim3((unsigned)(a.ntri + ceil_div(2 * (a.col - a.k), SYT_THREADS / 32)), (unsigned)a.nact);
            cfg.blockDim = dim3(SYT_THREADS);
            ProfRange r2("bhh_symv_tri_kernel", st, 0.0, 0.5 * bytes);
            PGX_CUDA(cudaLaunchKernelEx(&cfg, bhh_symv_tri_kernel, a));
            check_launch("bhh_symv_tri_kernel");
            return;
        }
        // rows per warp: 24 warps per SM where there are that many rows
        const int rw = all_rows >= 4L * 148 * 24 ? 4 : all_rows >= 2L * 148 * 24 ? 2 : 1;
        cfg.gridDim = dim3((unsigned)ceil_div(rows, rw * (BHH_SYMV_THREADS / 32)), (unsigned)a.nact);
        cfg.blockDim = dim3(BHH_SYMV_THREADS);
        ProfRange r2("bhh_symv_kernel", st, 0.0, bytes);
        PGX_CUDA(cudaLaunchKernelEx(&cfg, rw == 4 ? bhh_symv_kernel<4> : rw == 2 ? bhh_symv_kernel<2> : bhh_symv_kernel<1>, a));
        check_launch("bhh_symv_kernel");
    };
    PGX_CUDA(cudaFuncSetAttribute(bhh_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)UPD_SMEM));
    // ---- tridiagonalisation
    for (int k = 0; k < nmax - 2; k += BHH_NB) {
        a.k = k;
        const int jend = std::min(k + BHH_NB, nmax - 2);  // columns k .. jend - 1 of the largest block
        for (int j = k; j < jend; ++j) {
            a.fin = (j > k) ? j - 1 : -1;
            a.col = j;
            a.nact = nact(j > k ? j - 1 : j);
            col_step();
            a.fin = -1;
            a.nact = nact(j);
            double bytes = 0.0;
            long all_rows = 0;
            for (int i = 0; i < a.nact; ++i) {
                const double m = dims[big[i]] - j - 1;
                bytes += 8.0 * m * m;
                all_rows += dims[big[i]] - j - 1 + 2 * (j - k);
            }
            a.slots = bytes > SYT_BYTES;
            a.ntri = (int)(bhh_slots(nmax - j - 1) * (bhh_slots(nmax - j - 1) + 1) / 2);
            symv_step(nmax - j - 1 + 2 * (j - k), all_rows, bytes);
        }
        a.fin = jend - 1;
        a.col = -1;
        a.nact = nact(jend - 1);
        col_step();
        a.nact = nact(k);
        const long nt = ceil_div(nmax - jend, UPD_T);  // of the largest block
        double ufl = 0.0, uby = 0.0;
        for (int i = 0; i < a.nact; ++i) {
            const double p = std::min(BHH_NB, dims[big[i]] - 2 - k), m = dims[big[i]] - k - p;
            ufl += 2.0 * p * m * m;
            uby += 12.0 * m * m;
        }
        ProfRange ru("bhh_update_kernel", st, ufl, uby);
        bhh_update_kernel<<<dim3((unsigned)(nt * (nt + 1) / 2), (unsigned)a.nact), UPD_THREADS, UPD_SMEM, st>>>(a);
        check_launch("bhh_update_kernel");
    }
    // blocks beyond the direct back-transformation, a prefix of the list
    int nwide = 0;
    while (nwide < nbig && bt_class(dims[big[nwide]]) < 0) ++nwide;
    a.nact = nwide;
    bhh_finish_kernel<<<(unsigned)nbig, 256, 0, st>>>(a);
    check_launch("bhh_finish_kernel");
    if (nwide == 0) return;
    // ---- Q: Gram matrices and -T of every panel, then the panels from the last
    std::vector<GemmProblem<double, double, double>> probs;
    size_t tiles_cap = 0;
    const size_t probs_cap = eigh_gemm_bytes(dims, &tiles_cap);
    long npan_total = 0;
    long npan_max = 0;
    for (int i = 0; i < nwide; ++i) {
        const int n = dims[big[i]];
        const long np = bhh_panels(n);
        npan_max = std::max(npan_max, np);
        npan_total += np;
        for (long q = 0; q < np; ++q) {
            const int k = (int)q * BHH_NB, p = std::min(BHH_NB, n - 2 - k), m = n - k - 1;
            const double* Vp = d.A + moff[big[i]] + (long)k * n + (k + 1);  // V^T, p x m
            GemmProblem<double, double, double> g{};
            g.A = Vp;
            g.B = Vp;
            g.C = d.S + boff[i] + 2L * BHH_NB * n + 2L * n + q * BHH_NB * BHH_NB;
            g.M = p;
            g.N = p;
            g.K = m;
            g.sa_i = n;
            g.sa_k = 1;
            g.sb_k = 1;
            g.sb_j = n;
            g.sc_i = BHH_NB;
            g.sc_j = 1;
            probs.push_back(g);
        }
    }
    launch_gemm_batch(probs, d.gemm_probs, probs_cap, d.gemm_tiles, tiles_cap, st);
    bhh_tfactor_kernel<<<(unsigned)npan_total, 32, 0, st>>>(a);
    check_launch("bhh_tfactor_kernel");
    for (long q = npan_max - 1; q >= 0; --q) {
        const int k = (int)q * BHH_NB;
        std::vector<GemmProblem<double, double, double>> py, pt, pu;
        for (int i = 0; i < std::min(nwide, nact(k)); ++i) {
            const int n = dims[big[i]];
            const int p = std::min(BHH_NB, n - 2 - k), m = n - k - 1;
            const double* Vp = d.A + moff[big[i]] + (long)k * n + (k + 1);  // V^T, p x m
            double* Qs = d.Zc + moff[big[i]] + (long)(k + 1) * n + (k + 1);
            double* Y = d.S + boff[i];
            double* Y2 = Y + (long)BHH_NB * n;
            const double* nT = d.S + boff[i] + 2L * BHH_NB * n + 2L * n + (bhh_panels(n) + q) * BHH_NB * BHH_NB;
            GemmProblem<double, double, double> g{};
            g.A = Vp;  // Y = V^T Q
            g.sa_i = n;
            g.sa_k = 1;
            g.B = Qs;
            g.sb_k = 1;
            g.sb_j = n;
            g.C = Y;
            g.sc_i = n;
            g.sc_j = 1;
            g.M = p;
            g.N = m;
            g.K = m;
            py.push_back(g);
            GemmProblem<double, double, double> h{};  // Y2 = (-T) Y
            h.A = nT;
            h.sa_i = BHH_NB;
            h.sa_k = 1;
            h.B = Y;
            h.sb_k = n;
            h.sb_j = 1;
            h.C = Y2;
            h.sc_i = n;
            h.sc_j = 1;
            h.M = p;
            h.N = m;
            h.K = p;
            pt.push_back(h);
            GemmProblem<double, double, double> u{};  // Q += V Y2
            u.A = Vp;
            u.sa_i = 1;
            u.sa_k = n;
            u.B = Y2;
            u.sb_k = n;
            u.sb_j = 1;
            u.C = Qs;
            u.sc_i = 1;
            u.sc_j = n;
            u.M = m;
            u.N = m;
            u.K = p;
            u.accumulate = 1;
            pu.push_back(u);
        }
        launch_gemm_batch(py, d.gemm_probs, probs_cap, d.gemm_tiles, tiles_cap, st);
        launch_gemm_batch(pt, d.gemm_probs, probs_cap, d.gemm_tiles, tiles_cap, st);
        launch_gemm_batch(pu, d.gemm_probs, probs_cap, d.gemm_tiles, tiles_cap, st);
    }
}

// All eigensolver stages on caller-provided device buffers (no allocation),
// enqueued on stream st (asynchronous).
void launch_eigh_raw(const EighDev& d, const std::vector<int>& dims, const std::vector<long>& moff,
                     cudaStream_t st) {
    int dmax = 1;
    for (int x : dims) dmax = std::max(dmax, x);
    // descriptors: bisection items and the Householder block lists, one upload
    std::vector<TriItem> items;
    size_t n_vec = 0;
    tri_plan(dims, items, &n_vec);
    const size_t n_bis = items.size() - n_vec;
    HhPlan hp = hh_plan(dims);
    // blocks of a 16-CTA cluster take the large-block path where the device
    // cannot schedule one (a partition of a GPU, say)
    ClusterArgs ca;
    ca.dims = d.dims;
    ca.moff = d.moff;
    ca.eoff = d.eoff;
    ca.H = d.H;
    ca.V = d.A;
    ca.tri = d.tri;
    size_t cl_smem[CL_NCLS] = {0, 0, 0, 0, 0};
    PGX_CUDA(cudaFuncSetAttribute(eigh_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM_MAX));
    PGX_CUDA(cudaFuncSetAttribute(eigh_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (int q = CL_NCLS - 1; q >= 0; --q) {
        if (hp.cls[q].empty()) continue;
        for (int b : hp.cls[q]) cl_smem[q] = std::max(cl_smem[q], cluster_smem_doubles(dims[b], CL_SIZES[q]) * sizeof(double));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL_SIZES[q];
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)CL_SIZES[q]);
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = cl_smem[q];
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, eigh_cluster_kernel, &cfg) != cudaSuccess || nclusters < 1) {
            cudaGetLastError();
            PGX_CHECK(CL_SIZES[q] > 8, PGX_ERR_CUDA,
                      "the eigensolver's thread-block clusters cannot be scheduled on this device");
            hp.global.insert(hp.global.end(), hp.cls[q].begin(), hp.cls[q].end());  // smaller than those there
            hp.cls[q].clear();
            cl_smem[q] = 0;
        }
    }
    std::vector<int> lists(hp.global);
    size_t cl_off[CL_NCLS];
    for (int q = 0; q < CL_NCLS; ++q) {
        cl_off[q] = lists.size();
        lists.insert(lists.end(), hp.cls[q].begin(), hp.cls[q].end());
    }
    const BtPlan bt = bt_plan(dims);
    const size_t lists_at = items.size() * sizeof(TriItem) + bt.items.size() * sizeof(BtItem);
    // large blocks: scratch offsets (doubles into S)
    const std::vector<int>& big = hp.global;
    const size_t lists_end = lists_at + lists.size() * sizeof(int);
    const size_t boff_at = (lists_end + 7) & ~size_t(7);
    size_t host_bytes = lists_end;
    std::vector<BigBlk> blk;
    if (!big.empty()) {
        std::vector<long> eoff(dims.size() + 1, 0);
        for (size_t b = 0; b < dims.size(); ++b) eoff[b + 1] = eoff[b] + dims[b];
        long o = 0;
        for (int b : big) {
            blk.push_back(BigBlk{moff[b], eoff[b], o, dims[b], 0});
            o += bhh_scratch_doubles(dims[b]);
        }
        host_bytes = boff_at + blk.size() * sizeof(BigBlk);
        PGX_CHECK(host_bytes <= eigh_item_bytes(dims), PGX_ERR_ARG, "eigensolver descriptor layout overflow");
    }
    std::vector<char> host(host_bytes);
    std::memcpy(host.data(), items.data(), items.size() * sizeof(TriItem));
    if (!bt.items.empty())
        std::memcpy(host.data() + items.size() * sizeof(TriItem), bt.items.data(), bt.items.size() * sizeof(BtItem));
    std::memcpy(host.data() + lists_at, lists.data(), lists.size() * sizeof(int));
    if (!big.empty()) std::memcpy(host.data() + boff_at, blk.data(), blk.size() * sizeof(BigBlk));
    h2d(d.items, host.data(), host.size(), st);
    const BtItem* d_bt = reinterpret_cast<const BtItem*>(static_cast<const TriItem*>(d.items) + items.size());
    const int* d_lists = reinterpret_cast<const int*>(static_cast<const char*>(d.items) + lists_at);
    const BigBlk* d_blk = reinterpret_cast<const BigBlk*>(static_cast<const char*>(d.items) + boff_at);

    // LAPACK operation counts: tridiagonalisation 4/3 n^3, forming Q 4/3 n^3;
    // minimum DRAM traffic: read H, write Q and the tridiagonal
    auto hh_work = [&](const std::vector<int>& bl, double& fl, double& by) {
        fl = by = 0.0;
        for (int b : bl) {
            const double n = dims[b];
            fl += 8.0 / 3.0 * n * n * n;
            by += 16.0 * n * n + 16.0 * n;
        }
    };
    // the launches are independent: with side streams, cluster class q > 0 runs
    // on aux[q - 1] while the main stream runs the large blocks and class 0
    const bool fork = d.aux[0] && d.aux[1] && d.aux[2] && d.aux[3] && d.fork;
    if (fork) {
        PGX_CUDA(cudaEventRecord(d.fork, st));
        for (int i = 0; i < 4; ++i) PGX_CUDA(cudaStreamWaitEvent(d.aux[i], d.fork, 0));
    }
    if (!big.empty()) launch_big(d, dims, moff, big, d_blk, st);
    for (int q = 0; q < CL_NCLS; ++q) {
        if (hp.cls[q].empty()) continue;
        const cudaStream_t sq = (fork && q > 0) ? d.aux[q - 1] : st;
        ca.blocks = d_lists + cl_off[q];
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = CL_SIZES[q];
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(hp.cls[q].size() * CL_SIZES[q]));
        cfg.blockDim = dim3(CL_THREADS);
        cfg.dynamicSmemBytes = cl_smem[q];
        cfg.stream = sq;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        double fl, by;
        hh_work(hp.cls[q], fl, by);
        static const char* names[CL_NCLS] = {"eigh_cluster_kernel<1>", "eigh_cluster_kernel<2>", "eigh_cluster_kernel<4>",
                                       "eigh_cluster_kernel<8>", "eigh_cluster_kernel<16>"};
        ProfRange pr(names[q], sq, fl, by);
        PGX_CUDA(cudaLaunchKernelEx(&cfg, eigh_cluster_kernel, ca));
        check_launch("eigh_cluster_kernel");
    }
    if (fork) {
        for (int i = 0; i < 4; ++i) {
            PGX_CUDA(cudaEventRecord(d.join[i], d.aux[i]));
            PGX_CUDA(cudaStreamWaitEvent(st, d.join[i], 0));
        }
    }

    TriArgs t;
    t.items = static_cast<const TriItem*>(d.items);
    t.dims = d.dims;
    t.moff = d.moff;
    t.eoff = d.eoff;
    t.tri = d.tri;
    t.lam = d.lam;
    t.sb = d.sb;
    t.rank = d.rank;
    t.Z = d.Zc;
    t.Zq = d.A;  // the reflectors are in Q
    t.S = d.S;
    t.E = d.E;
    t.status = d.status;
    const size_t smem_b = 2 * sizeof(double) * (size_t)dmax, smem_v = 3 * sizeof(double) * (size_t)dmax;
    const TriItem* bis_items = static_cast<const TriItem*>(d.items) + n_vec;
    PGX_CUDA(cudaFuncSetAttribute(bisect_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_b));
    PGX_CUDA(cudaFuncSetAttribute(vector_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_v));
    PGX_CUDA(cudaFuncSetAttribute(ortho_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_v));
    double esum = 0.0, msum = 0.0;
    for (int n : dims) {
        esum += n;
        msum += (double)n * n;
    }
    {
        ProfRange pr("bisect_kernel", st, 0.0, 16.0 * esum + 8.0 * esum + 8.0 * esum);
        bisect_kernel<<<(unsigned)n_bis, BIS_THREADS, smem_b, st>>>(t, bis_items, bisect_lanes(total_dim(dims)));
        check_launch("bisect_kernel");
    }
    {
        ProfRange pr("vector_kernel", st, 0.0, 8.0 * msum + 48.0 * esum);
        vector_kernel<<<(unsigned)n_vec, TRI_THREADS, smem_v, st>>>(t);
        check_launch("vector_kernel");
    }
    {
        ProfRange pr("ortho_kernel", st, 0.0, 0.0);
        ortho_kernel<<<(unsigned)n_vec, TRI_THREADS, smem_v, st>>>(t);
        check_launch("ortho_kernel");
    }

    // the reflectors (A) applied to Z (Zc); the T factors take the vector stage's scratch
    if (bt.first[1] > 0) {
        ProfRange pr("bt_tfactor_kernel", st, 0.0, 0.0);
        bt_tfactor_kernel<<<(unsigned)bt.first[1], BT_THREADS, 0, st>>>(d_bt, d.A, d.S);
        check_launch("bt_tfactor_kernel");
    }
    for (int c = 0; c < BT_NCLS; ++c) {
        const size_t nit = bt.first[c + 2] - bt.first[c + 1];
        if (nit == 0) continue;
        double fl = 0.0, by = 0.0;
        for (int n : dims)
            if (bt_class(n) == c) {
                fl += 2.0 * n * (double)n * n;
                by += 24.0 * n * (double)n;
            }
        ProfRange pr("bt_apply_kernel", st, fl, by);
        const BtItem* q = d_bt + bt.first[c + 1];
        if (BT_COLS[c] == 32) launch_bt_apply<32>(q, nit, bt.nmax[c], d.A, d.S, d.Zc, d.U, st);
        else if (BT_COLS[c] == 16) launch_bt_apply<16>(q, nit, bt.nmax[c], d.A, d.S, d.Zc, d.U, st);
        else launch_bt_apply<8>(q, nit, bt.nmax[c], d.A, d.S, d.Zc, d.U, st);
    }
    // wider blocks: U = Q Z, Q column-major (Zc), Z column-major (A), U row-major
    std::vector<GemmProblem<double, double, double>> probs;
    for (size_t b = 0; b < dims.size(); ++b) {
        const int n = dims[b];
        if (bt_class(n) >= 0) continue;
        GemmProblem<double, double, double> g{};
        g.A = d.Zc + moff[b];
        g.B = d.A + moff[b];
        g.C = d.U + moff[b];
        g.M = n;
        g.N = n;
        g.K = n;
        g.sa_i = 1;
        g.sa_k = n;
        g.sb_k = 1;
        g.sb_j = n;
        g.sc_i = n;
        g.sc_j = 1;
        probs.push_back(g);
    }
    size_t tiles_cap = 0;
    const size_t probs_cap = eigh_gemm_bytes(dims, &tiles_cap);
    launch_gemm_batch(probs, d.gemm_probs, probs_cap, d.gemm_tiles, tiles_cap, st);
}

// Complex Hermitian blocks: embedding, real eigensolve of the embedding,
// extraction of the complex eigenvectors (see cx_extract_kernel).
static void launch_eigh_complex(pgx_ctx* c) {
    Problem& P = c->P;
    cudaStream_t st = c->stream;
    const int nb = P.nblocks;
    std::vector<int> d2(nb);
    std::vector<long> m2(nb), e2(nb);
    long msz2 = 0, esz2 = 0;
    for (int b = 0; b < nb; ++b) {
        d2[b] = 2 * P.dims[b];
        m2[b] = msz2;
        e2[b] = esz2;
        msz2 += (long)d2[b] * d2[b];
        esz2 += d2[b];
    }
    // dims | moff | eoff of the embedding, on the device
    const size_t off_m = (nb * sizeof(int) + 15) & ~size_t(15);
    P.cx_meta.reserve(off_m + 2 * nb * sizeof(long));
    int* dd2 = P.cx_meta.as<int>();
    long* dm2 = reinterpret_cast<long*>(P.cx_meta.as<char>() + off_m);
    long* de2 = dm2 + nb;
    h2d(dd2, d2.data(), nb * sizeof(int), st);
    h2d(dm2, m2.data(), nb * sizeof(long), st);
    h2d(de2, e2.data(), nb * sizeof(long), st);
    P.cx_H.reserve(msz2 * sizeof(double));
    P.cx_A.reserve(msz2 * sizeof(double));
    P.cx_Zc.reserve(msz2 * sizeof(double));
    P.cx_U.reserve(msz2 * sizeof(double));
    P.cx_E.reserve(esz2 * sizeof(double));
    P.cx_tri.reserve((3 * esz2) * sizeof(double) + 3 * esz2 * sizeof(int) + 64);
    P.cx_S.reserve(eigh_vec_scratch_doubles(d2) * sizeof(double));
    P.cx_items.reserve(eigh_item_bytes(d2));
    size_t tiles_b = 0;
    const size_t probs_b = eigh_gemm_bytes(d2, &tiles_b);
    P.cx_gemm.reserve(((probs_b + 255) & ~size_t(255)) + tiles_b);
    int dmax = 1;
    for (int x : P.dims) dmax = std::max(dmax, x);
    {
        dim3 g(std::min(ceil_div((long)dmax * dmax, 256), 1024), (unsigned)nb);
        cx_embed_kernel<<<g, 256, 0, st>>>(P.d_dims, P.d_moff, dm2, P.d_H, P.cx_H.as<double>());
        check_launch("cx_embed_kernel");
    }
    EighDev d;
    d.dims = dd2;
    d.moff = dm2;
    d.eoff = de2;
    d.H = P.cx_H.as<double>();
    d.A = P.cx_A.as<double>();
    d.Zc = P.cx_Zc.as<double>();
    d.tri = P.cx_tri.as<double>();
    d.lam = d.tri + 2 * esz2;
    d.sb = reinterpret_cast<int*>(d.lam + esz2);
    d.rank = d.sb + 2 * esz2;
    d.S = P.cx_S.as<double>();
    d.items = P.cx_items.p;
    d.gemm_probs = P.cx_gemm.p;
    d.gemm_tiles = P.cx_gemm.as<char>() + ((probs_b + 255) & ~size_t(255));
    d.U = P.cx_U.as<double>();
    d.E = P.cx_E.as<double>();
    d.status = P.d_status;
    for (int i = 0; i < 4; ++i) {
        d.aux[i] = c->aux[i];
        d.join[i] = c->join[i];
    }
    d.fork = c->fork;
    launch_eigh_raw(d, d2, m2, st);
    // pairs of the embedding agree to the eigensolver's accuracy, far inside
    // this clustering tolerance; distinct eigenvalues of H closer than it are
    // orthonormalised together
    std::vector<double> e(esz2);
    PGX_CUDA(cudaMemcpyAsync(e.data(), d.E, esz2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    PGX_CUDA(cudaStreamSynchronize(st));
    double emax = 1.0;
    for (double x : e) emax = std::max(emax, std::fabs(x));
    cx_extract_kernel<<<nb, 128, 0, st>>>(P.d_dims, P.d_moff, P.d_eoff, dm2, de2, d.E, d.U, P.d_E,
                                          reinterpret_cast<cd*>(P.d_U), 1e-10 * emax, P.d_status);
    check_launch("cx_extract_kernel");
}

void ensure_side_streams(pgx_ctx* c) {
    if (c->fork) return;
    PGX_CUDA(cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming));
    for (int i = 0; i < 4; ++i) {
        PGX_CUDA(cudaStreamCreateWithFlags(&c->aux[i], cudaStreamNonBlocking));
        PGX_CUDA(cudaEventCreateWithFlags(&c->join[i], cudaEventDisableTiming));
    }
}

void launch_eigh(pgx_ctx* c) {
    Problem& P = c->P;
    cudaStream_t st = c->stream;
    ensure_side_streams(c);
    if (P.is_complex) {
        launch_eigh_complex(c);
        return;
    }
    // tri (2 sum d) | lam (sum d) | sb (2 sum d ints) | rank (sum d ints)
    const long e = std::max<long>(P.esize, 1);
    P.tri.reserve((2 * e + e) * sizeof(double) + 3 * e * sizeof(int) + 64);
    P.tri_items.reserve(eigh_item_bytes(P.dims));
    size_t tiles_b = 0;
    const size_t probs_b = eigh_gemm_bytes(P.dims, &tiles_b);
    P.eigh_gemm.reserve(((probs_b + 255) & ~size_t(255)) + tiles_b);
    P.eigh_scratch.reserve(eigh_vec_scratch_doubles(P.dims) * sizeof(double));
    EighDev d;
    d.dims = P.d_dims;
    d.moff = P.d_moff;
    d.eoff = P.d_eoff;
    d.H = P.d_H;
    d.A = P.d_work;
    d.Zc = P.d_work2;
    d.tri = P.tri.as<double>();
    d.lam = d.tri + 2 * e;
    d.sb = reinterpret_cast<int*>(d.lam + e);
    d.rank = d.sb + 2 * e;
    d.S = P.eigh_scratch.as<double>();
    d.items = P.tri_items.p;
    d.gemm_probs = P.eigh_gemm.p;
    d.gemm_tiles = P.eigh_gemm.as<char>() + ((probs_b + 255) & ~size_t(255));
    d.U = P.d_U;
    d.E = P.d_E;
    d.status = P.d_status;
    for (int i = 0; i < 4; ++i) {
        d.aux[i] = c->aux[i];
        d.join[i] = c->join[i];
    }
    d.fork = c->fork;
    launch_eigh_raw(d, P.dims, P.moff, st);
}

}  // namespace pgx
