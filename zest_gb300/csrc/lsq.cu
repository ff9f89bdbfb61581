// Least-squares fits of expansions to data at scattered points:
//   st::LSQTransformer::transform   lsq_transformer.hpp:57-110 (RealSHGenerator::generate,
//                                   sh_generator.hpp:69-120; LinearMultifit, src/linearfit.cpp)
//   zt::LSQTransformer::transform   lsq_transformer.hpp:119-187 (ZernikeGenerator::generate,
//                                   zernike_generator.hpp:64-140)
//
// The reference builds the design matrix (one row per point, one column per
// real basis function) and solves it with LAPACK's dgels (Householder QR).
// Here the design matrix is built on the device from the P_lm and R_nl
// tables at the points (the same table kernels as everywhere else) and
// cos/sin(m lon) -- the reference's generators take std::cos/std::sin of
// m * lon -- and solved by the method of dgels, written here in FP64 kernels
// of this file: blocked Householder QR (panels of 32 columns, the reflectors
// of a panel applied to the trailing columns in the compact WY form
// I - V T V^T), the right-hand sides carried as extra trailing columns so
// that they receive Q^T, and back substitution with R.  `batch` data vectors
// at the same points are the right-hand sides of one factorisation.  As
// dgels, no rank check: the points must determine the expansion (at least as
// many points as unknowns).
//
// SH basis: P_lm(z) cos(m lon), P_lm(z) sin(m lon) with z = sin(latitude),
// as RealSHGenerator::generate (it evaluates P_lm at the sine of its angle
// argument, which LSQTransformer passes latitudes to).  Zernike basis:
// R_nl(r) P_lm(cos colatitude) {cos, sin}(m lon), as ZernikeGenerator
// evaluates it.  (The reference's Zernike fit passes its arguments to the
// generator in another order and regroups the solution by l alone; the fit
// here is the one its interface describes.)
#include <algorithm>
#include <cmath>
#include <vector>

#include "context.cuh"
#include "lsq.cuh"
#include "tables.cuh"

namespace zgpu {

struct LsqState {
    DevBuf A, b, cols, P, R, z, r, lon;
    DevBuf part, T, W;  // QR: reduction partials, the panel's T, the panel's T^T V^T C
    DevBuf order, off;  // design columns by m
    DevBuf sync;        // arrivals of the panels' exchanges, error flag
};
void destroy_lsq(LsqState* s) { delete s; }

namespace {

// A[col][i] (column-major, lda = npts): block row m fills the columns of one m,
// entries {n, l, c, col} at [off[m], off[m + 1]) (n < 0: SH), so that a point's
// sincos(m lon) is taken once for all of them (about 60 FP64 operations against
// one product per entry): 1.08 -> 0.11 ms for 1,024 columns of 20,000 points.
__global__ void design_kernel(int npts, const int4* __restrict__ entries, const int* __restrict__ off,
                              const double* __restrict__ P, const double* __restrict__ R,
                              const double* __restrict__ lon, double* __restrict__ A) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npts) return;
    const int m = blockIdx.y;
    double sn, cs;
    sincos(double(m) * lon[i], &sn, &cs);
    for (int j = off[m]; j < off[m + 1]; ++j) {
        const int4 c = entries[j];
        double v = P[tri_idx(c.y, m) * npts + i] * (c.z ? sn : cs);
        if (c.x >= 0) v *= R[((((long long)c.x + 1) * (c.x + 1)) >> 2) * npts + (c.y >> 1) * (long long)npts + i];
        A[(long long)c.w * npts + i] = v;
    }
}

// coeffs[b][k][c] = x[b][col(k, c)] (the first ncol entries of right-hand side b)
__global__ void scatter_kernel(int ncol, int batch, const int4* __restrict__ cols, const int* __restrict__ pair,
                               const double* __restrict__ X, long long ldx, double* __restrict__ coeffs,
                               long long cstride) {
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= (long long)ncol * batch) return;
    const int b = int(t / ncol), j = int(t - (long long)b * ncol);
    coeffs[b * cstride + 2 * (long long)pair[j] + cols[j].w] = X[b * ldx + j];
}


// ---------------------------------------------------------------------------
// Householder QR least squares in FP64 (the method of LAPACK dgels).  The
// m x n matrix A (column-major, lda = m, m >= n) is factored in panels of
// QR_NB columns; reflector k is H_k = I - tau_k v_k v_k^T with v_k[k] = 1,
// v_k[i] = 0 for i < k and v_k[i > k] stored below the diagonal of A, as
// dgeqrf stores it; R is left in the upper triangle.  After each panel its
// reflectors are applied to the trailing columns of A and to the nrhs
// right-hand sides B (m x nrhs, ldb = m) at once, as
// C <- (I - V T V^T)^T C = C - V (T^T (V^T C)).  Every reduction is summed in
// a fixed order (per-block partials, then one pass over the blocks), so the
// result does not depend on the launch.
constexpr int QR_NB = 32;           // panel width
constexpr int QR_CCOLS = 64;        // columns per block of V^T C and of the update

// column c of the trailing part: columns of A from a0 on, then those of B
struct QrCols {
    double* A;
    long long lda;
    int na;  // trailing columns of A
    double* B;
    long long ldb;
    __device__ double* col(int c) const { return c < na ? A + (long long)c * lda : B + (long long)(c - na) * ldb; }
};

// ---------------------------------------------------------------------------
// One panel in one cooperative launch: columns j0 .. j0 + jb - 1, every CTA
// keeping its rows of them in shared memory (or, above SMEM_ROWS rows per CTA, in
// place in A).  A reflector needs one exchange between the CTAs: each sums, over
// its rows below the pivot, the products of the pivot column with all columns of
// the panel -- those to the right give the norm and the update, those to the
// left (the earlier reflectors) the next column of T -- and writes the 32 sums;
// after a grid barrier every CTA adds the sums of all CTAs in the same order and
// goes on alone.  The columns of earlier reflectors stay unscaled in the panel
// (u = x, v = scale u) until the end.  Reflectors as dlarfg: tau = 0 (H = I) when
// the column below the diagonal is zero.  T of the compact WY form (dlarft,
// forward, columnwise): T[k][k] = tau_k, T[0:k][k] = -tau_k T[0:k][0:k] V^T v_k,
// formed by block 0 while it waits for the next exchange.
//
// What bounds it is the chain of a reflector: partial sums, the exchange, a
// square root and two quotients.  With one launch per reflector and the panel
// read from L2 each time it took 20 us a reflector, 9.2 so (20,000 rows).  Every
// wait is bounded (2 s): then the error flag is set and all blocks leave.
constexpr int QR_SMEM = 200 * 1024;  // shared memory of a CTA's panel rows
constexpr long long QR_TIMEOUT_NS = 2000000000LL;

struct QrPanel {
    double* A;
    long long lda;
    int m, j0, jb, rpb;  // rows per block, from row j0 on
    double* part;        // [2][blocks][QR_NB] sums, then [2][QR_NB] pivot rows
    double* tau;
    double* T;           // QR_NB x QR_NB row-major
    unsigned* bar;       // arrivals of all exchanges so far in this solve
    unsigned base;       // its value before this launch
    int* err;
};

// Sum over the warp's lanes of four values per lane: every group of 8 lanes
// (lane >> 3) ends up with value lane >> 3 (six additions instead of twenty).
__device__ __forceinline__ double warp_sum4(const double (&v)[4], int lane) {
    const bool h1 = lane & 16, h2 = lane & 8;
    const double a0 = (h1 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[2], 16);
    const double a1 = (h1 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h1 ? v[1] : v[3], 16);
    double t = (h2 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, h2 ? a0 : a1, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

template <bool SMEM>
__global__ void __launch_bounds__(256) qr_panel(const QrPanel Q) {
    extern __shared__ double panel_s[];
    __shared__ double red[8][QR_NB], w[QR_NB], z[QR_NB], scale_s[QR_NB], tau_s[QR_NB];
    __shared__ double Ts[QR_NB][QR_NB + 1];
    __shared__ int ok_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, jb = Q.jb;
    const int r0 = Q.j0 + int(blockIdx.x) * Q.rpb, nr = max(0, min(Q.m - r0, Q.rpb));
    double* const pbase = SMEM ? panel_s : Q.A + (long long)Q.j0 * Q.lda + r0;
    const long long ps = SMEM ? (long long)Q.rpb : Q.lda;
    auto col = [&](int c) { return pbase + c * ps; };
    if constexpr (SMEM) {
        for (int c = warp; c < jb; c += 8)
            for (int i = lane; i < nr; i += 32) col(c)[i] = Q.A[(long long)(Q.j0 + c) * Q.lda + r0 + i];
    }
    for (int e = tid; e < QR_NB * (QR_NB + 1); e += 256) (&Ts[0][0])[e] = 0.0;
    __syncthreads();
    // column k of T from z = V^T v_k; lane a: row a
    auto t_column = [&](int k) {
        double t0 = 0.0, t1 = 0.0;
        if (lane < k) {
            int q = lane;
            for (; q + 1 < k; q += 2) {
                t0 = fma(Ts[lane][q], z[q], t0);
                t1 = fma(Ts[lane][q + 1], z[q + 1], t1);
            }
            if (q < k) t0 = fma(Ts[lane][q], z[q], t0);
        }
        __syncwarp();
        if (lane < k) Ts[lane][k] = -tau_s[k] * (t0 + t1);
        if (lane == k) Ts[k][k] = tau_s[k];
        __syncwarp();
    };
    bool ok = true;
    for (int k = 0; k < jb; ++k) {
        const int pk = Q.j0 + k - r0;  // the pivot row within this block's rows (may lie outside)
        double* part = Q.part + (size_t)(k & 1) * G * QR_NB;
        double* rowk = Q.part + (size_t)2 * G * QR_NB + (k & 1) * QR_NB;
        {
            double acc[4] = {0.0, 0.0, 0.0, 0.0};
            const double* x = col(k);
            const int c0 = 4 * warp;
            for (int i = max(0, pk + 1) + lane; i < nr; i += 32) {
                const double xi = x[i];
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (c0 + q < jb) acc[q] = fma(xi, col(c0 + q)[i], acc[q]);
            }
            const double t = warp_sum4(acc, lane);
            if ((lane & 7) == 0) __stcg(part + (size_t)blockIdx.x * QR_NB + c0 + (lane >> 3), t);
        }
        if (pk >= 0 && pk < nr && tid < jb) __stcg(rowk + tid, col(tid)[pk]);
        __syncthreads();
        if (tid == 0) {  // exchange: arrive, wait for the other blocks
            __threadfence();
            atomicAdd(Q.bar, 1u);
            const unsigned want = Q.base + unsigned(k + 1) * unsigned(G);
            unsigned long long t0 = 0;
            int good = 1;
            for (unsigned it = 1;; ++it) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(Q.bar) : "memory");
                if (int(v - want) >= 0) break;
                if ((it & 1023) == 0) {
                    unsigned long long now;
                    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                    if (t0 == 0) t0 = now;
                    if (*(volatile int*)Q.err || now - t0 > (unsigned long long)QR_TIMEOUT_NS) {
                        atomicCAS(Q.err, 0, 1);
                        good = 0;
                        break;
                    }
                }
            }
            ok_s = good;
        }
        if (blockIdx.x == 0 && warp == 7 && k > 0) t_column(k - 1);
        __syncthreads();
        ok = ok_s != 0;
        if (!ok) break;  // uniform
        {
            double v = 0.0;
            for (int b0 = warp; b0 < G; b0 += 8 * 20) {  // 20 loads in flight: all of 152 blocks' share
                double t[20];
#pragma unroll
                for (int u = 0; u < 20; ++u) {
                    const int b = b0 + 8 * u;
                    t[u] = b < G ? __ldcg(part + (size_t)b * QR_NB + lane) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 20; ++u)
                    if (b0 + 8 * u < G) v += t[u];
            }
            red[warp][lane] = v;
        }
        __syncthreads();
        if (warp == 0) {
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q) sum += red[q][lane];
            const double row = lane < jb ? __ldcg(rowk + lane) : 0.0;
            const double alpha = __shfl_sync(0xffffffffu, row, k), ss = __shfl_sync(0xffffffffu, sum, k);
            double t = 0.0, scale = 0.0, beta = alpha;
            if (ss > 0.0) {
                beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
                t = (beta - alpha) / beta;
                scale = 1.0 / (alpha - beta);
            }
            // tau v^T a_c = tau (a_c[k] + scale d_c); V^T v_k for the earlier reflectors
            const double vd = fma(scale, sum, row);
            if (lane > k) w[lane] = t * vd;
            else if (lane < k) z[lane] = scale_s[lane] * vd;
            else {
                w[lane] = beta;
                scale_s[lane] = scale;
                tau_s[lane] = t;
            }
        }
        __syncthreads();
        // apply H_k to the columns right of k on this block's rows
        const double scale = scale_s[k];
        const double* x = col(k);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = 4 * warp + q;
            if (c <= k || c >= jb) continue;
            double* a = col(c);
            const double wc = w[c], sw = scale * wc;
            for (int i = max(0, pk) + lane; i < nr; i += 32) a[i] = i == pk ? a[i] - wc : fma(-x[i], sw, a[i]);
        }
        __syncthreads();
        if (tid == 0 && pk >= 0 && pk < nr) col(k)[pk] = w[k];
        // (the pivot element is read again only by the write-back: later reflectors sum the rows below)
    }
    __syncthreads();
    if (!ok) return;
    for (int c = warp; c < jb; c += 8) {
        const double sc = scale_s[c];
        const int d = Q.j0 + c - r0;  // the diagonal's row
        for (int i = lane; i < nr; i += 32) {
            const double v = i > d ? col(c)[i] * sc : col(c)[i];
            Q.A[(long long)(Q.j0 + c) * Q.lda + r0 + i] = v;
        }
    }
    if (blockIdx.x == 0) {
        if (warp == 7) t_column(jb - 1);
        __syncthreads();
        for (int e = tid; e < QR_NB * QR_NB; e += 256) Q.T[e] = Ts[e / QR_NB][e % QR_NB];
        if (tid < jb) Q.tau[Q.j0 + tid] = tau_s[tid];
    }
}

// v_a[i] of a panel starting at column j0 (v_a[j0 + a] = 1, 0 above)
__device__ __forceinline__ double qr_v(const double* __restrict__ A, long long lda, int j0, int a, int i) {
    const int d = j0 + a;
    return i < d ? 0.0 : (i == d ? 1.0 : A[(long long)d * lda + i]);
}

// Per-block partials of V^T C over rows j0 .. m-1: part[blk][a][c] for the
// block's QR_CCOLS trailing columns (a < jb).  Thread (ty, tx): rows a =
// 4 ty .. 4 ty + 3 of V^T, columns tx and tx + 32 of the tile (the second half
// only where the tile has more than 32 columns).  `crows` rows per block: enough
// blocks that the last wave's idle SMs cost little (the FP64 pipe is the bound).
__global__ void __launch_bounds__(256) qr_vtc(const double* __restrict__ A, long long lda, int m, int j0, int jb,
                                              QrCols C, int ncols, int crows, double* __restrict__ part) {
    __shared__ double Vs[32][QR_NB + 1];
    __shared__ double Cs[32][QR_CCOLS + 1];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c0 = blockIdx.x * QR_CCOLS;
    double acc[4][2] = {};
    const int r0 = j0 + blockIdx.y * crows, r1 = min(m, r0 + crows);
    const bool both = c0 + 32 < ncols;
    for (int q0 = r0; q0 < r1; q0 += 32) {
        for (int e = threadIdx.x; e < 32 * QR_NB; e += blockDim.x) {
            const int i = e & 31, a = e >> 5;
            Vs[i][a] = (q0 + i < r1 && a < jb) ? qr_v(A, lda, j0, a, q0 + i) : 0.0;
        }
        for (int e = threadIdx.x; e < 32 * QR_CCOLS; e += blockDim.x) {
            const int i = e & 31, c = e >> 5;
            Cs[i][c] = (q0 + i < r1 && c0 + c < ncols) ? C.col(c0 + c)[q0 + i] : 0.0;
        }
        __syncthreads();
#pragma unroll 8
        for (int i = 0; i < 32; ++i) {
            double va[4];
#pragma unroll
            for (int p = 0; p < 4; ++p) va[p] = Vs[i][4 * ty + p];
            const double cb = Cs[i][tx];
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[p][0] = fma(va[p], cb, acc[p][0]);
            if (both) {
                const double cc = Cs[i][tx + 32];
#pragma unroll
                for (int p = 0; p < 4; ++p) acc[p][1] = fma(va[p], cc, acc[p][1]);
            }
        }
        __syncthreads();
    }
    double* out = part + (long long)blockIdx.y * QR_NB * ncols;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int a = 4 * ty + p;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int c = c0 + tx + 32 * q;
            if (a < jb && c < ncols) out[(long long)a * ncols + c] = acc[p][q];
        }
    }
}

// W = T^T (sum over the row blocks of V^T C).  A block of 8 x 32 x 4 threads takes
// 8 trailing columns (enough blocks for all SMs at 1,000 columns): thread (c, a,
// y) sums entry (a, c) over the row blocks of slice y, the four slices are added
// in order, and thread (c, a, 0) forms (T^T u)_a = sum_{q <= a} T[q][a] u_q.
// 216 us a panel with 32 blocks of 32 columns, 30 so.
__global__ void __launch_bounds__(1024) qr_wmat(const double* __restrict__ part, int nblk, int jb, int ncols,
                                                const double* __restrict__ T, double* __restrict__ W) {
    __shared__ double Ts[QR_NB][QR_NB + 1];
    __shared__ double u[4][QR_NB][8];
    const int cl = threadIdx.x, a = threadIdx.y, y = threadIdx.z;
    const int tid = (y * 32 + a) * 8 + cl;
    Ts[tid / QR_NB][tid % QR_NB] = T[tid];
    const int c = blockIdx.x * 8 + cl;
    double v = 0.0;
    if (c < ncols && a < jb) {
        const int per = (nblk + 3) / 4, b1 = min(nblk, (y + 1) * per);
        const double* p = part + (long long)a * ncols + c;
        const long long st = (long long)QR_NB * ncols;
#pragma unroll 8
        for (int b = y * per; b < b1; ++b) v += p[b * st];
    }
    u[y][a][cl] = v;
    __syncthreads();
    if (y == 0) u[0][a][cl] = ((v + u[1][a][cl]) + u[2][a][cl]) + u[3][a][cl];
    __syncthreads();
    if (y || c >= ncols || a >= jb) return;
    double w = 0.0;
    for (int q = 0; q <= a; ++q) w = fma(Ts[q][a], u[0][q][cl], w);  // T upper triangular
    W[(long long)a * ncols + c] = w;
}

// C[i][c] -= sum_a v_a[i] W[a][c] for rows j0 .. m-1: 64 x 64 tiles; thread
// (tx, ty) updates rows i0 + tx + 32 p (p < 2) of columns c0 + ty + 8 q
// (q < 8), so that the lanes of a warp touch 32 consecutive rows of a column.
__global__ void __launch_bounds__(256) qr_update(const double* __restrict__ A, long long lda, int m, int j0, int jb,
                                                 QrCols C, int ncols, const double* __restrict__ W) {
    __shared__ double Vs[QR_NB][64 + 1];
    __shared__ double Ws[QR_NB][64 + 1];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i0 = j0 + blockIdx.y * 64, c0 = blockIdx.x * 64;
    for (int e = threadIdx.x; e < 64 * QR_NB; e += blockDim.x) {
        const int i = e & 63, a = e >> 6;
        Vs[a][i] = (i0 + i < m && a < jb) ? qr_v(A, lda, j0, a, i0 + i) : 0.0;
        Ws[a][i] = (c0 + i < ncols && a < jb) ? W[(long long)a * ncols + c0 + i] : 0.0;
    }
    const int nq = min(8, (ncols - c0 - ty + 7) / 8);
    double acc[2][8];  // C itself, so that no addition is left for the end
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const double* col = q < nq ? C.col(c0 + ty + 8 * q) : nullptr;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int i = i0 + tx + 32 * p;
            acc[p][q] = (q < nq && i < m) ? col[i] : 0.0;
        }
    }
    __syncthreads();
#pragma unroll 4
    for (int a = 0; a < QR_NB; ++a) {
        double vv[2], ww[8];
#pragma unroll
        for (int p = 0; p < 2; ++p) vv[p] = Vs[a][tx + 32 * p];
#pragma unroll
        for (int q = 0; q < 8; ++q) ww[q] = Ws[a][ty + 8 * q];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (q < nq) {  // uniform over the warp: no products for columns past the end
#pragma unroll
                for (int p = 0; p < 2; ++p) acc[p][q] = fma(-vv[p], ww[q], acc[p][q]);
            }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if (q >= nq) continue;
        double* col = C.col(c0 + ty + 8 * q);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int i = i0 + tx + 32 * p;
            if (i < m) col[i] = acc[p][q];
        }
    }
}

// Back substitution R x = y for each right-hand side (one block each): y =
// B[0:n][r] (the first n entries of Q^T b), R the upper triangle of A; x
// overwrites y.  Blocks of 32 unknowns from the end: one warp solves the 32 x 32
// triangle (x_j = y_j / R_jj, then y_i -= R_ij x_j, j descending), then every
// thread takes the block's 32 products off its rows above, in the same order.
// Two barriers per 32 unknowns instead of two per unknown: 2.1 -> 0.8 ms at 1,024 unknowns.
__global__ void __launch_bounds__(1024) qr_backsub(const double* __restrict__ A, long long lda, int n,
                                                   double* __restrict__ B, long long ldb) {
    extern __shared__ double y[];
    __shared__ double Rs[32][33], xs[32];
    double* b = B + (long long)blockIdx.x * ldb;
    for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = b[i];
    for (int j1 = n; j1 > 0;) {
        const int j0 = (j1 - 1) / 32 * 32, nb = j1 - j0;
        const int ti = threadIdx.x & 31, tj = threadIdx.x >> 5;
        if (ti < nb && tj < nb) Rs[tj][ti] = A[(long long)(j0 + tj) * lda + j0 + ti];  // [column][row]
        __syncthreads();
        if (threadIdx.x < 32) {
            double yi = ti < nb ? y[j0 + ti] : 0.0;
            for (int j = nb - 1; j >= 0; --j) {
                const double q = ti == j ? yi / Rs[j][j] : 0.0;
                const double xj = __shfl_sync(0xffffffffu, q, j);
                if (ti == j) yi = xj;
                else if (ti < j) yi = fma(-Rs[j][ti], xj, yi);
            }
            if (ti < nb) y[j0 + ti] = xs[ti] = yi;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < j0; i += blockDim.x) {
            double v = y[i];
#pragma unroll 8
            for (int j = nb - 1; j >= 0; --j) v = fma(-A[(long long)(j0 + j) * lda + i], xs[j], v);
            y[i] = v;
        }
        __syncthreads();
        j1 = j0;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) b[i] = y[i];
}

// Least-squares solution of A x = B (m x n, m >= n, nrhs right-hand sides):
// A is overwritten by its QR factors, B's first n rows by the solutions.
int qr_solve(zest_gpu_context* ctx, LsqState& Q, double* A, int m, int n, double* B, int nrhs) {
    cudaStream_t s = ctx->stream;
    const long long lda = m;
    int dev = 0, sms = 0;
    ZG_CUDA_TRY(cudaGetDevice(&dev));
    ZG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int ncol_max = n + nrhs;
    // row blocks of V^T C: 32 blocks per SM over the column tiles, 64 to 512 rows each
    auto vtc_rows = [&](int rows, int ntrail) {
        const int ct = (ntrail + QR_CCOLS - 1) / QR_CCOLS;
        const long long want = (long long)rows * ct / (32LL * sms);
        return int(std::min<long long>(512, std::max<long long>(64, (want + 31) / 32 * 32)));
    };
    size_t part_n = (size_t)2 * sms * QR_NB + 2 * QR_NB;
    for (int j0 = 0; j0 < n; j0 += QR_NB) {
        const int nt = std::max(0, n - j0 - QR_NB) + nrhs, cr = vtc_rows(m - j0, nt);
        part_n = std::max(part_n, (size_t)((m - j0 + cr - 1) / cr) * QR_NB * nt);
    }
    ZG_TRY(Q.part.ensure((part_n + 8) * sizeof(double)));
    ZG_TRY(Q.T.ensure((QR_NB * QR_NB + n + 8) * sizeof(double)));
    ZG_TRY(Q.W.ensure((size_t)QR_NB * ncol_max * sizeof(double)));
    ZG_TRY(Q.sync.ensure(2 * sizeof(unsigned)));
    ZG_CUDA_TRY(cudaMemsetAsync(Q.sync.p, 0, 2 * sizeof(unsigned), s));
    double* part = Q.part.as<double>();
    double* T = Q.T.as<double>();
    double* tau = T + QR_NB * QR_NB;
    double* W = Q.W.as<double>();
    unsigned arrivals = 0;
    ZG_CUDA_TRY(cudaFuncSetAttribute(qr_panel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, QR_SMEM));
    for (int j0 = 0; j0 < n; j0 += QR_NB) {
        const int jb = std::min(QR_NB, n - j0);
        // one CTA per SM, at least 64 rows each
        const int G = std::max(1, std::min(sms, (m - j0 + 63) / 64));
        const int rpb = (m - j0 + G - 1) / G;
        const size_t psmem = (size_t)rpb * jb * sizeof(double);
        QrPanel P{A, lda, m, j0, jb, rpb, part, tau, T, Q.sync.as<unsigned>(), arrivals, Q.sync.as<int>() + 1};
        arrivals += unsigned(G) * unsigned(jb);
        void* args[] = {&P};
        const bool in_smem = psmem <= size_t(QR_SMEM);
        const void* kern = in_smem ? reinterpret_cast<const void*>(qr_panel<true>)
                                   : reinterpret_cast<const void*>(qr_panel<false>);
        ZG_CUDA_TRY(cudaLaunchCooperativeKernel(kern, dim3(G), dim3(256), args, in_smem ? psmem : 0, s));
        ZG_TRY(launch_check("qr_panel"));
        const int ntrail = (n - j0 - jb) + nrhs;
        if (ntrail == 0) continue;
        const QrCols C{A + (long long)(j0 + jb) * lda, lda, n - j0 - jb, B, lda};
        const int crows = vtc_rows(m - j0, ntrail), vb = (m - j0 + crows - 1) / crows;
        qr_vtc<<<dim3((ntrail + QR_CCOLS - 1) / QR_CCOLS, vb), 256, 0, s>>>(A, lda, m, j0, jb, C, ntrail, crows, part);
        ZG_TRY(launch_check("qr_vtc"));
        qr_wmat<<<(ntrail + 7) / 8, dim3(8, 32, 4), 0, s>>>(part, vb, jb, ntrail, T, W);
        ZG_TRY(launch_check("qr_wmat"));
        qr_update<<<dim3((ntrail + 63) / 64, (m - j0 + 63) / 64), 256, 0, s>>>(A, lda, m, j0, jb, C, ntrail, W);
        ZG_TRY(launch_check("qr_update"));
    }
    const size_t ysmem = (size_t)n * sizeof(double);
    if (ysmem > 200 * 1024) return fail(ZEST_GPU_ERR_UNSUPPORTED, "least-squares fit: more than 25600 unknowns");
    if (ysmem > 48 * 1024)
        ZG_CUDA_TRY(cudaFuncSetAttribute(qr_backsub, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ysmem));
    qr_backsub<<<nrhs, 1024, ysmem, s>>>(A, lda, n, B, lda);
    return launch_check("qr_backsub");
}

}  // namespace

int lsq_dev(zest_gpu_context* ctx, int kind, int zn, int sn, int sp, int L, int npts, int batch, const double* data,
            const std::vector<double>& z, const std::vector<double>& lon, const std::vector<double>& r,
            double* coeffs) {
    if (batch == 0 || L == 0) return ZEST_GPU_OK;
    cudaStream_t s = ctx->stream;
    if (!ctx->lsq) ctx->lsq.reset(new LsqState());
    LsqState& Q = *ctx->lsq;
    // columns: every (n, l, m) cos term, and the sin term for m > 0
    std::vector<int4> cols;
    std::vector<int> pair;
    if (kind == 0) {
        for (int n = 0; n < L; ++n)
            for (int l = n & 1; l <= n; l += 2)
                for (int m = 0; m <= l; ++m)
                    for (int c = 0; c < (m ? 2 : 1); ++c) {
                        cols.push_back(make_int4(n, l, m, c));
                        pair.push_back(int(zidx(n, l, m)));
                    }
    } else {
        for (int l = 0; l < L; ++l)
            for (int m = 0; m <= l; ++m)
                for (int c = 0; c < (m ? 2 : 1); ++c) {
                    cols.push_back(make_int4(-1, l, m, c));
                    pair.push_back(int(tri_idx(l, m)));
                }
    }
    const int ncol = int(cols.size());
    if (npts < ncol)
        return fail(ZEST_GPU_ERR_UNSUPPORTED, "least-squares fit: fewer points (" + std::to_string(npts) +
                                                  ") than unknowns (" + std::to_string(ncol) + ")");
    std::vector<int4> order;  // {n, l, c, column} by m
    std::vector<int> off((size_t)L + 1, 0);
    for (const int4& c : cols) ++off[(size_t)c.z + 1];
    for (int m = 0; m < L; ++m) off[(size_t)m + 1] += off[(size_t)m];
    {
        order.resize(cols.size());
        std::vector<int> fill(off.begin(), off.end() - 1);
        for (int j = 0; j < ncol; ++j)
            order[(size_t)fill[(size_t)cols[(size_t)j].z]++] = make_int4(cols[(size_t)j].x, cols[(size_t)j].y, cols[(size_t)j].w, j);
    }
    DevBuf dpair;
    ZG_TRY(upload(Q.cols, cols, s));
    ZG_TRY(upload(Q.order, order, s));
    ZG_TRY(upload(Q.off, off, s));
    ZG_TRY(upload(dpair, pair, s));
    ZG_TRY(upload(Q.z, z, s));
    ZG_TRY(upload(Q.lon, lon, s));
    ZG_TRY(Q.P.ensure((size_t)tri_size(L) * npts * sizeof(double)));
    ZG_TRY(launch_plm_ref(s, L, sn, sp, npts, Q.z.as<double>(), Q.P.as<double>()));
    if (kind == 0) {
        ZG_TRY(upload(Q.r, r, s));
        ZG_TRY(Q.R.ensure((size_t)((((size_t)L + 1) * (L + 1)) >> 2) * npts * sizeof(double)));
        ZG_TRY(launch_radial_ref(s, L, zn, npts, Q.r.as<double>(), Q.R.as<double>()));
    }
    ZG_TRY(Q.A.ensure((size_t)ncol * npts * sizeof(double)));
    {
        StageScope sc(ctx, ST_EVAL_TABLES);
        design_kernel<<<dim3((npts + 127) / 128, L), 128, 0, s>>>(npts, Q.order.as<int4>(), Q.off.as<int>(),
                                                                  Q.P.as<double>(),
                                                                  kind == 0 ? Q.R.as<double>() : nullptr,
                                                                  Q.lon.as<double>(), Q.A.as<double>());
        ZG_TRY(launch_check("design_kernel"));
    }
    // right-hand sides: the data vectors, npts each (overwritten by Q^T b)
    ZG_TRY(Q.b.ensure((size_t)npts * batch * sizeof(double)));
    ZG_CUDA_TRY(cudaMemcpyAsync(Q.b.p, data, (size_t)npts * batch * sizeof(double), cudaMemcpyDeviceToDevice, s));
    {
        StageScope sc(ctx, ST_EVAL_LEG);
        ZG_TRY(qr_solve(ctx, Q, Q.A.as<double>(), npts, ncol, Q.b.as<double>(), batch));
    }
    double* b = Q.b.as<double>();
    const long long csz = 2 * (kind == 0 ? zsize(L) : tri_size(L));
    ZG_CUDA_TRY(cudaMemsetAsync(coeffs, 0, (size_t)csz * batch * sizeof(double), s));
    const long long n = (long long)ncol * batch;
    scatter_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(ncol, batch, Q.cols.as<int4>(), dpair.as<int>(), b, npts,
                                                            coeffs, csz);
    ZG_TRY(launch_check("scatter_kernel"));
    int late = 0;
    ZG_CUDA_TRY(cudaMemcpyAsync(&late, Q.sync.as<int>() + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    ZG_CUDA_TRY(cudaStreamSynchronize(s));  // dpair is local
    if (late) return fail(ZEST_GPU_ERR_TIMEOUT, "least-squares fit: bounded wait expired");
    return ZEST_GPU_OK;
}

}  // namespace zgpu
