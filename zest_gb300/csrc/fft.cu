// Batched real DFT along the longitude axis, FP64, in shared memory.
//
// Replaces pocketfft::r2c / c2r as called by the reference transformers
// (zernike_glq_transformer.hpp:710-720 and 943-949, sh_glq_transformer.hpp:
// 757-765 and 1195-1201).  The longitude count is odd (2L-1: 39, 199, 399,
// 2047, ...) or a multiple of 8 (LatLon layout).
//
// GB300 retires two FP64 multiply-adds per clock and SM, so only the number
// of FP64 operations counts; integer work, shared-memory traffic and index
// arithmetic hide behind them.  The plan of a length N keeps them few:
//   * N = product of coprime prime powers: a multi-dimensional DFT by the
//     prime-factor (Good-Thomas) index maps, which needs no twiddle factors
//     between the dimensions.  The maps are applied where the columns are
//     loaded and stored;
//   * a dimension p^a: Stockham stages of radix p (4 and 2 for p = 2), the
//     first without twiddles;
//   * a dimension that is a large prime p with a smooth p - 1: Rader's
//     algorithm, a cyclic convolution of length p - 1 done by two DFTs of that
//     length (themselves prime-factor transforms) and a product with the
//     transformed roots.  Its index permutation is part of the same maps, and
//     its second DFT is a forward one too: the reversed output order is the
//     order of the powers of the generator.
// FP64 operations per complex point: N = 199 (order 100) 59 against 198 of
// the direct radix, N = 399 (order 200) 36 against 46 with twiddled stages,
// N = 2047 (order 1024) 81 against 126.  Measured, one direction: order 100 x
// 32 12.8 -> 4.4 ms (its 61 operations per point take 3.4 ms at the FP64 rate),
// SH order 1024 x 8 2.1 -> 1.3 ms.
//
// Each CTA transforms 2*NC real columns packed as NC complex columns
// (z = x_a + i x_b); the real spectra are separated at the end.  Columns are
// the contiguous (lat, rad) points of one longitude row, so every global load
// and store is coalesced.
//
// Forward output  F[b][m][col][2] = conj(X_m(col)), m < nm (no scaling; the
//                 quadrature prefactor lives in the Legendre tables).
// Inverse input   F[b][m][col][2] = Hermitian coefficients of m < nm; output
//                 x_i = Re F_0 + 2 sum_{m>0} Re(F_m e^{+2 pi i im/N}) -- the
//                 c2r semantics with factor 1.  It is the forward DFT of the
//                 conjugated spectra, conjugated.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <utility>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "spectra.cuh"

namespace zgpu {

namespace {

__device__ __forceinline__ double2 cmul_tw(double2 a, double2 w) {
    return make_double2(fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x));
}

// x / 2 by the exponent field (exact like the product, but no FP64 operation)
__device__ __forceinline__ double halve(double x) {
    const int hi = __double2hiint(x), e = hi & 0x7FF00000;
    if (e > 0x00100000 && e != 0x7FF00000) return __hiloint2double(hi - 0x00100000, __double2loint(x));
    return 0.5 * x;  // zero, subnormal results, infinities, NaN
}

// R-point DFT of a small odd R in registers: y_q and y_{R-q} from the sums and
// differences s_r = t_r + t_{R-r}, d_r = t_r - t_{R-r}:
//     y_q = a - i b,  y_{R-q} = a + i b,  a = t_0 + sum_r s_r cos(2 pi r q/R),
//     b = sum_r d_r sin(2 pi r q/R)
// (R - 1 multiply-adds per output instead of 4 R).  w[wR m] = W_R^m.
template <int R>
__device__ __forceinline__ void dft_odd(const double2 (&t)[R], const double2* __restrict__ w, int wR,
                                        double2* __restrict__ y, size_t ys) {
    constexpr int h = R / 2;
    double2 s[h], d[h];
    double2 y0 = t[0];
#pragma unroll
    for (int r = 0; r < h; ++r) {
        s[r] = make_double2(t[r + 1].x + t[R - 1 - r].x, t[r + 1].y + t[R - 1 - r].y);
        d[r] = make_double2(t[r + 1].x - t[R - 1 - r].x, t[r + 1].y - t[R - 1 - r].y);
        y0.x += s[r].x;
        y0.y += s[r].y;
    }
    y[0] = y0;
#pragma unroll
    for (int q = 1; q <= h; ++q) {
        double2 a = t[0], b = make_double2(0.0, 0.0);
#pragma unroll
        for (int r = 1; r <= h; ++r) {
            const double2 c = w[wR * ((r * q) % R)];  // cos, -sin
            a.x = fma(s[r - 1].x, c.x, a.x);
            a.y = fma(s[r - 1].y, c.x, a.y);
            if (h == 1) {  // R = 3: one term, added and subtracted by multiply-adds
                y[ys] = make_double2(fma(-d[0].y, c.y, a.x), fma(d[0].x, c.y, a.y));
                y[2 * ys] = make_double2(fma(d[0].y, c.y, a.x), fma(-d[0].x, c.y, a.y));
            } else if (r == 1) {
                b = make_double2(-d[0].x * c.y, -d[0].y * c.y);
            } else {
                b.x = fma(-d[r - 1].x, c.y, b.x);
                b.y = fma(-d[r - 1].y, c.y, b.y);
            }
        }
        if (h > 1) {
            y[q * ys] = make_double2(a.x + b.y, a.y - b.x);
            y[(R - q) * ys] = make_double2(a.x - b.y, a.y + b.x);
        }
    }
}

// One butterfly of a stage of small odd radix R: load, twiddle, DFT, store.
template <int R>
__device__ __forceinline__ void butterfly(const double2* __restrict__ x, size_t xs, double2* __restrict__ y, size_t ys,
                                          const double2* __restrict__ tw, int tstep, int wR) {
    double2 t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = x[r * xs];
    if (tstep) {
#pragma unroll
        for (int r = 1; r < R; ++r) t[r] = cmul_tw(t[r], tw[r * tstep]);
    }
    dft_odd<R>(t, tw, wR, y, ys);
}

// One Stockham pass of radix R along one dimension of the array: elements
// (o, k, i) at base + o ostride + k inner + i, k < Nd, twiddle table tw (size
// Nd, W_t = e^{-2 pi i t/Nd}).  Butterfly j takes x_r = src[j + r Nd/R],
// twiddles it, t_r = x_r W^{r jm Nd/(Ns R)} with jm = j mod Ns (jm = 0 needs
// none: all butterflies of a first stage), and stores its R-point DFT to
// dst[(j/Ns) Ns R + jm + q Ns].  Radices up to 13 are done per butterfly in
// registers; a larger odd radix in two phases: phase A (per butterfly)
// twiddles and writes the sums s_r and differences d_r back in place -- every
// src element belongs to exactly one butterfly -- and stores y_0; phase B
// computes the output pairs, one (butterfly, q) per thread.
__device__ __forceinline__ void fft_stage(double2* __restrict__ src, double2* __restrict__ dst,
                                          const double2* __restrict__ tw, const FftOp& op, int NC) {
    const int R = op.R, Ns = op.Ns;
    const unsigned NR = unsigned(op.Nd / R), in = unsigned(op.inner * NC);
    const int step = op.Nd / (Ns * R);
    const int wR = op.Nd / R;  // W_R^m = tw[wR m]
    const size_t xs = (size_t)NR * in, ys = (size_t)Ns * in, os = (size_t)op.ostride * NC, b0 = (size_t)op.base * NC;
    const unsigned nb = unsigned(op.outer) * NR * in;
    for (unsigned o = threadIdx.x; o < nb; o += blockDim.x) {
        const unsigned t = o / in, i = o - t * in;
        const unsigned ou = t / NR, j = t - ou * NR;
        const unsigned jq = j / unsigned(Ns), jm = j - jq * unsigned(Ns);
        double2* x = src + b0 + ou * os + (size_t)j * in + i;
        double2* y = dst + b0 + ou * os + (size_t)(jq * unsigned(Ns * R) + jm) * in + i;
        const int tstep = int(jm) * step;
        switch (R) {
        case 2: {
            const double2 a = x[0];
            double2 b = x[xs];
            if (tstep) b = cmul_tw(b, tw[tstep]);
            y[0] = make_double2(a.x + b.x, a.y + b.y);
            y[ys] = make_double2(a.x - b.x, a.y - b.y);
            break;
        }
        case 4: {
            const double2 a = x[0];
            double2 b = x[xs], c = x[2 * xs], d = x[3 * xs];
            if (tstep) {
                b = cmul_tw(b, tw[tstep]);
                c = cmul_tw(c, tw[2 * tstep]);
                d = cmul_tw(d, tw[3 * tstep]);
            }
            const double2 s0 = make_double2(a.x + c.x, a.y + c.y), d0 = make_double2(a.x - c.x, a.y - c.y);
            const double2 s1 = make_double2(b.x + d.x, b.y + d.y), d1 = make_double2(b.x - d.x, b.y - d.y);
            y[0] = make_double2(s0.x + s1.x, s0.y + s1.y);
            y[ys] = make_double2(d0.x + d1.y, d0.y - d1.x);  // d0 - i d1
            y[2 * ys] = make_double2(s0.x - s1.x, s0.y - s1.y);
            y[3 * ys] = make_double2(d0.x - d1.y, d0.y + d1.x);
            break;
        }
        case 3: butterfly<3>(x, xs, y, ys, tw, tstep, wR); break;
        case 5: butterfly<5>(x, xs, y, ys, tw, tstep, wR); break;
        case 7: butterfly<7>(x, xs, y, ys, tw, tstep, wR); break;
        case 11: butterfly<11>(x, xs, y, ys, tw, tstep, wR); break;
        case 13: butterfly<13>(x, xs, y, ys, tw, tstep, wR); break;
        default: {
            if (tstep) {
                int t2 = tstep;
                for (int r = 1; r < R; ++r) {
                    x[r * xs] = cmul_tw(x[r * xs], tw[t2]);
                    t2 += tstep;
                }
            }
            const int h = R >> 1;
            double2 y0 = x[0];
            for (int r = 1; r <= h; ++r) {
                const double2 a = x[r * xs], b = x[(R - r) * xs];
                const double2 sr = make_double2(a.x + b.x, a.y + b.y);
                x[r * xs] = sr;
                x[(R - r) * xs] = make_double2(a.x - b.x, a.y - b.y);
                y0.x += sr.x;
                y0.y += sr.y;
            }
            y[0] = y0;
        }
        }
    }
    if (R <= 13) return;
    __syncthreads();
    const unsigned h = unsigned(R) >> 1;
    const unsigned np = nb * h;
    for (unsigned o = threadIdx.x; o < np; o += blockDim.x) {
        const unsigned bq = o / h;
        const int q = int(o - bq * h) + 1;
        const unsigned t = bq / in, i = bq - t * in;
        const unsigned ou = t / NR, j = t - ou * NR;
        const unsigned jq = j / unsigned(Ns), jm = j - jq * unsigned(Ns);
        const double2* x = src + b0 + ou * os + (size_t)j * in + i;
        double2* y = dst + b0 + ou * os + (size_t)(jq * unsigned(Ns * R) + jm) * in + i;
        double2 a = x[0], b = make_double2(0.0, 0.0);
        int m = q;
        for (unsigned r = 1; r <= h; ++r) {
            const double2 w = tw[wR * m];  // cos(2 pi m/R), -sin(2 pi m/R)
            const double2 sr = x[r * xs], dr = x[(R - r) * xs];
            a.x = fma(sr.x, w.x, a.x);
            a.y = fma(sr.y, w.x, a.y);
            b.x = fma(dr.x, -w.y, b.x);
            b.y = fma(dr.y, -w.y, b.y);
            m += q;
            if (m >= R) m -= R;
        }
        y[q * ys] = make_double2(a.x + b.y, a.y - b.x);        // a - i b
        y[(R - q) * ys] = make_double2(a.x - b.y, a.y + b.x);  // a + i b
    }
}

// The middle of a Rader dimension: rows 1 .. p-1 of each outer slice hold the
// DFT X of the permuted inputs (in `cur`); row 0 holds x_0, in `home`, the
// buffer the dimension started in.  y_0 = x_0 + X_0 goes back to `home`, and
// the rows become X_k B_k (B: the transformed roots over p - 1), with x_0 added
// to k = 0, so that the second DFT adds it to every output.
__device__ __forceinline__ void rader_product(double2* __restrict__ cur, double2* home, const double2* __restrict__ B,
                                              const FftOp& op, int NC) {
    const unsigned in = unsigned(op.inner * NC), n = unsigned(op.Nd);  // Nd = p - 1
    const size_t os = (size_t)op.ostride * NC, b0 = (size_t)op.base * NC;
    const unsigned total = unsigned(op.outer) * n * in;
    for (unsigned o = threadIdx.x; o < total; o += blockDim.x) {
        const unsigned t = o / in, i = o - t * in;
        const unsigned ou = t / n, k = t - ou * n;
        double2* c = cur + b0 + ou * os + (size_t)k * in + i;
        const double2 X = *c;
        double2 v = cmul_tw(X, B[k]);
        if (k == 0) {
            double2* z = home + b0 - in + ou * os + i;  // row 0 is the row before `base`
            const double2 x0 = *z;
            *z = make_double2(x0.x + X.x, x0.y + X.y);
            v.x += x0.x;
            v.y += x0.y;
        }
        *c = v;
    }
}

// All operations of the plan; the result's buffer is returned.
__device__ __forceinline__ double2* run_plan(double2* a, double2* b, const double2* tab, const FftPlan& plan, int NC) {
    for (int s = 0; s < plan.nops; ++s) {
        const FftOp& op = plan.ops[s];
        if (op.R > 0) {
            fft_stage(a, b, tab + op.tab, op, NC);
            double2* t = a;
            a = b;
            b = t;
        } else {
            // Ns: whether an odd number of stages lies behind the permuted rows
            rader_product(a, op.Ns ? b : a, tab + op.tab, op, NC);
        }
        __syncthreads();
    }
    return a;
}

// x(b, i, col) = x + b*xb + i*si + col*sc ; lon_fast: i is the contiguous axis
__global__ void __launch_bounds__(256) rfft_fwd_kernel(const __grid_constant__ FftPlan plan,
                                                       const double* __restrict__ x, long long xb, long long si,
                                                       long long sc, int C, int nm, int NC, int lon_fast,
                                                       double* __restrict__ F) {
    extern __shared__ double2 smem[];
    const int N = plan.N;
    double2* tab = smem;
    double2* A = smem + plan.ntab;
    double2* Bf = A + (size_t)N * NC;
    const int b = blockIdx.y;
    const int col0 = blockIdx.x * 2 * NC;
    for (int t = threadIdx.x; t < plan.ntab; t += blockDim.x) tab[t] = plan.tab[t];
    const double* xbp = x + (long long)b * xb;
    double* Ad = reinterpret_cast<double*>(A);
    const int W = 2 * NC;
    for (int e = threadIdx.x; e < N * W; e += blockDim.x) {
        int i, cl;
        if (lon_fast) { i = e % N; cl = e / N; }
        else { cl = e % W; i = e / W; }
        const int col = col0 + cl;
        const double v = (col < C) ? xbp[(long long)i * si + (long long)col * sc] : 0.0;
        Ad[(plan.in_row[i] * NC + (cl >> 1)) * 2 + (cl & 1)] = v;
    }
    __syncthreads();
    const double2* Z = run_plan(A, Bf, tab, plan, NC);
    // separate the two real spectra and store conj(X_m), m < nm
    for (int e = threadIdx.x; e < nm * NC; e += blockDim.x) {
        const int cp = e % NC;
        const int m = e / NC;
        const double2 z = Z[plan.out_row[m] * NC + cp];
        const double2 zn = Z[plan.out_row[m ? N - m : 0] * NC + cp];
        // X_a = (Z_m + conj Z_{N-m}) / 2,  X_b = (Z_m - conj Z_{N-m}) / (2i)
        const int col = col0 + 2 * cp;
        double* out = F + (((long long)b * nm + m) * C + col) * 2;
        if (col < C) {
            out[0] = halve(z.x + zn.x);
            out[1] = halve(zn.y - z.y);
        }
        if (col + 1 < C) {
            out[2] = halve(z.y + zn.y);
            out[3] = halve(z.x - zn.x);
        }
    }
}

template <class In>
__global__ void __launch_bounds__(256) rfft_inv_kernel(const __grid_constant__ FftPlan plan, const In src, int C,
                                                       int nm, int NC, int lon_fast, double* __restrict__ x,
                                                       long long xb, long long si, long long sc) {
    extern __shared__ double2 smem[];
    const int N = plan.N;
    double2* tab = smem;
    double2* A = smem + plan.ntab;
    double2* Bf = A + (size_t)N * NC;
    const int b = blockIdx.y;
    const int col0 = blockIdx.x * 2 * NC;
    for (int t = threadIdx.x; t < plan.ntab; t += blockDim.x) tab[t] = plan.tab[t];
    // Hermitian completion of the two packed spectra F_a + i F_b, conjugated
    for (int e = threadIdx.x; e < N * NC; e += blockDim.x) {  // orders the spectra do not hold
        const int m = e / NC;
        if (m >= nm && N - m >= nm) A[plan.in_row[m] * NC + e - m * NC] = make_double2(0.0, 0.0);
    }
    for (int e = threadIdx.x; e < nm * NC; e += blockDim.x) {
        const int cp = e % NC;
        const int m = e / NC;
        const int col = col0 + 2 * cp;
        const double2 fa = (col < C) ? src.get(b, m, col) : make_double2(0.0, 0.0);
        const double2 fb = (col + 1 < C) ? src.get(b, m, col + 1) : make_double2(0.0, 0.0);
        if (m == 0) {
            A[plan.in_row[0] * NC + cp] = make_double2(fa.x, -fb.x);
        } else {
            A[plan.in_row[m] * NC + cp] = make_double2(fa.x - fb.y, -(fa.y + fb.x));
            A[plan.in_row[N - m] * NC + cp] = make_double2(fa.x + fb.y, fa.y - fb.x);
        }
    }
    __syncthreads();
    const double2* Z = run_plan(A, Bf, tab, plan, NC);
    const double* Zd = reinterpret_cast<const double*>(Z);
    double* xbp = x + (long long)b * xb;
    const int W = 2 * NC;
    for (int e = threadIdx.x; e < N * W; e += blockDim.x) {
        int i, cl;
        if (lon_fast) { i = e % N; cl = e / N; }
        else { cl = e % W; i = e / W; }
        const int col = col0 + cl;
        const double v = Zd[(plan.out_row[i] * NC + (cl >> 1)) * 2 + (cl & 1)];
        // the second column is the imaginary part, conjugated
        if (col < C) xbp[(long long)i * si + (long long)col * sc] = (cl & 1) ? -v : v;
    }
}

// ---- plan ---------------------------------------------------------------------

// FP64 operations per complex point of the transforms above
double dft_cost(int R) { return R == 2 ? 2.0 : R == 3 ? 4.0 : R == 4 ? 4.0 : (R - 1.0) * (R + 4.0) / R; }

struct PrimePower {
    int p, a, n;  // n = p^a
};
std::vector<PrimePower> factors(int N) {
    std::vector<PrimePower> f;
    for (int q = 2; N > 1; ++q) {
        if ((long long)q * q > N) q = N;
        PrimePower w{q, 0, 1};
        while (N % q == 0) {
            N /= q;
            ++w.a;
            w.n *= q;
        }
        if (w.a) f.push_back(w);
    }
    return f;
}
// radices of the stages of a dimension p^a
std::vector<int> stages_of(const PrimePower& w) {
    std::vector<int> r;
    if (w.p == 2) {
        for (int k = 0; k + 1 < w.a; k += 2) r.push_back(4);
        if (w.a & 1) r.push_back(2);
    } else {
        r.assign(size_t(w.a), w.p);
    }
    return r;
}
double direct_cost(const PrimePower& w) {
    double c = 0.0;
    bool first = true;
    for (int R : stages_of(w)) {
        c += dft_cost(R) + (first ? 0.0 : 4.0 * (R - 1.0) / R);
        first = false;
    }
    return c;
}
// Rader where it saves a tenth of the direct radix's operations
bool use_rader(const PrimePower& w) {
    if (w.a != 1 || w.p < 17) return false;
    double sub = 0.0;
    for (const PrimePower& v : factors(w.p - 1)) sub += direct_cost(v);
    return (w.p - 1.0) / w.p * (2.0 * sub + 4.0) + 4.0 / w.p < 0.9 * direct_cost(w);
}

int inverse_mod(int a, int n) {
    for (int x = 1; x < n; ++x)
        if ((long long)(a % n) * x % n == 1) return x;
    return 0;  // n = 1
}
int power_mod(int g, int e, int p) {
    long long r = 1, b = g;
    for (; e; e >>= 1, b = b * b % p)
        if (e & 1) r = r * b % p;
    return int(r);
}
int generator_of(int p) {
    const std::vector<PrimePower> f = factors(p - 1);
    for (int g = 2;; ++g) {
        bool ok = true;
        for (const PrimePower& v : f) ok = ok && power_mod(g, (p - 1) / v.p, p) != 1;
        if (ok) return g;
    }
}

// e^{-2 pi i t / n} with the angle reduced to an eighth of a turn
void root(long long t, long long n, double* re, double* im) {
    t %= n;
    // eighths: 8 t = o n + rest, angle = (o + rest / n) pi / 4
    const double pi4 = 0.785398163397448309615660845819875721;
    const long long o = 8 * t / n, rest = 8 * t - o * n;
    const bool odd = o & 1;
    const double a = pi4 * (double(odd ? n - rest : rest) / double(n));
    double c = std::cos(a), s = std::sin(a);
    if (odd) std::swap(c, s);  // pi/4 < angle < pi/2 within the quadrant
    const long long quad = o >> 1;
    double C = c, Sn = s;
    if (quad == 1) { C = -s; Sn = c; }
    if (quad == 2) { C = -c; Sn = -s; }
    if (quad == 3) { C = s; Sn = -c; }
    *re = C;
    *im = -Sn;
}

// Position of index v (0 <= v < product of the dimensions) by the Good map:
// coordinate v (N / N_d)^{-1} mod N_d along each dimension, row-major.
struct GoodMap {
    std::vector<PrimePower> f;
    std::vector<int> inv, stride;
    int N = 1;
    explicit GoodMap(std::vector<PrimePower> dims) : f(std::move(dims)) {
        for (const PrimePower& w : f) N *= w.n;
        stride.assign(f.size(), 1);
        for (size_t d = f.size(); d-- > 1;) stride[d - 1] = stride[d] * f[d].n;
        for (const PrimePower& w : f) inv.push_back(w.n == 1 ? 0 : inverse_mod(N / w.n, w.n));
    }
};

}  // namespace

int build_fft_plan(int N, FftPlan& plan, std::vector<double>& tab, std::vector<int>& rows, bool allow_rader) {
    plan = FftPlan{};
    plan.N = N;
    tab.clear();
    auto add_roots = [&](int n) {
        const int at = int(tab.size() / 2);
        for (int t = 0; t < n; ++t) {
            double c, s;
            root(t, n, &c, &s);
            tab.push_back(c);
            tab.push_back(s);
        }
        return at;
    };
    auto add_op = [&](FftOp op) {
        if (plan.nops == kFftMaxOps) return false;
        auto rcp = [](long long d) { return d == 1 ? 0u : unsigned((1ll << 32) / d + 1); };
        op.nr = op.R ? op.Nd / op.R : 1;
        op.step = op.R ? op.nr / op.Ns : 0;
        op.rcp_inner = rcp(op.inner);
        op.rcp_nr = rcp(op.nr);
        op.rcp_ns = rcp(op.Ns ? op.Ns : 1);
        for (int k = 0; k < 4; ++k) op.rcp_nb[k] = rcp(((long long)op.outer * op.nr * op.inner) << k);
        plan.ops[plan.nops++] = op;
        return true;
    };
    bool fits = true;
    // the largest prime that pays as a Rader dimension becomes the outermost one
    std::vector<PrimePower> dims = factors(N);
    size_t rader = dims.size();
    for (size_t d = 0; allow_rader && d < dims.size(); ++d)
        if (use_rader(dims[d])) rader = d;
    if (rader < dims.size()) {
        std::swap(dims[0], dims[rader]);
        rader = 0;
    }
    // the stages of a dimension of `n` rows of `inner`, `outer` slices `ostride` rows apart from row `base`
    auto add_dim = [&](const PrimePower& w, int base, int outer, int ostride, int inner, int at) {
        int Ns = 1;
        for (int R : stages_of(w)) {
            fits = add_op(FftOp{R, w.n, Ns, base, outer, ostride, inner, at}) && fits;
            Ns *= R;
        }
        return int(stages_of(w).size());
    };
    const GoodMap top(dims);
    rows.assign(2 * (size_t)N, 0);
    int* in_row = rows.data();
    int* out_row = rows.data() + N;
    for (size_t d = 0; d < top.f.size(); ++d) {
        const PrimePower& w = top.f[d];
        const int stride = top.stride[d], outer = N / (w.n * stride), ostride = w.n * stride;
        std::vector<int> perm(w.n);  // index along the dimension -> row of the dimension
        for (int v = 0; v < w.n; ++v) perm[v] = v;
        if (d == rader) {
            const int p = w.p, g = generator_of(p);
            const GoodMap sub(factors(p - 1));
            auto good = [&](int r) {
                int at = 0;
                for (size_t e = 0; e < sub.f.size(); ++e)
                    at += int((long long)r * sub.inv[e] % sub.f[e].n) * sub.stride[e];
                return at;
            };
            auto crt = [&](int k) {
                int at = 0;
                for (size_t e = 0; e < sub.f.size(); ++e) at += k % sub.f[e].n * sub.stride[e];
                return at;
            };
            // rows: 0, then the powers g^r at 1 + good(r)
            std::vector<int> pw(p - 1);
            long long x = 1;
            for (int r = 0; r < p - 1; ++r, x = x * g % p) {
                pw[r] = int(x);
                perm[x] = 1 + good(r);
            }
            // transformed roots: B_k = 1/(p-1) sum_r w_p^{g^{-r}} w_{p-1}^{k r}
            std::vector<double> wp(2 * (size_t)p), wn(2 * (size_t)(p - 1));
            for (int t = 0; t < p; ++t) root(t, p, &wp[2 * t], &wp[2 * t + 1]);
            for (int t = 0; t < p - 1; ++t) root(t, p - 1, &wn[2 * t], &wn[2 * t + 1]);
            std::vector<int> at(sub.f.size());
            for (size_t e = 0; e < sub.f.size(); ++e) at[e] = add_roots(sub.f[e].n);
            const int bt = int(tab.size() / 2);
            tab.resize(tab.size() + 2 * (size_t)(p - 1));
            for (int k = 0; k < p - 1; ++k) {
                double re = 0.0, im = 0.0;
                int t = 0;
                for (int r = 0; r < p - 1; ++r) {
                    const int q = pw[r ? p - 1 - r : 0];
                    re += wp[2 * q] * wn[2 * t] - wp[2 * q + 1] * wn[2 * t + 1];
                    im += wp[2 * q] * wn[2 * t + 1] + wp[2 * q + 1] * wn[2 * t];
                    t += k;
                    if (t >= p - 1) t -= p - 1;
                }
                tab[2 * (size_t)(bt + crt(k))] = re / (p - 1);
                tab[2 * (size_t)(bt + crt(k)) + 1] = im / (p - 1);
            }
            int ns = 0;
            for (int pass = 0; pass < 2; ++pass) {
                for (size_t e = 0; e < sub.f.size(); ++e) {
                    const int si = sub.stride[e] * stride, so = (p - 1) / (sub.f[e].n * sub.stride[e]);
                    const int k = add_dim(sub.f[e], stride, so, sub.f[e].n * si, si, at[e]);
                    if (pass == 0) ns += k;
                }
                if (pass == 0) fits = add_op(FftOp{0, p - 1, ns & 1, stride, 1, N, stride, bt}) && fits;
            }
        } else {
            add_dim(w, 0, outer, ostride, stride, add_roots(w.n));
        }
        for (int v = 0; v < N; ++v) {
            in_row[v] += perm[(long long)v * top.inv[d] % w.n] * stride;
            out_row[v] += perm[v % w.n] * stride;
        }
    }
    plan.ntab = int(tab.size() / 2);
    return fits ? ZEST_GPU_OK : ZEST_GPU_ERR_UNSUPPORTED;
}

size_t fft_smem_bytes(const FftPlan& plan, int NC) { return 16 * ((size_t)plan.ntab + 2 * (size_t)plan.N * NC); }

namespace {

// Columns per CTA: two ping-pong buffers and the tables within ~110 KB keep two
// CTAs per SM; fewer where the whole transform would leave SMs without a CTA.
int choose_nc(const FftPlan& plan, long long cols) {
    int nc = 8;
    while (nc > 1 && fft_smem_bytes(plan, nc) > 110 * 1024) --nc;
    while (nc > 2 && cols < 2LL * nc * 152) nc /= 2;
    return nc;
}

// Threads per CTA: small blocks with several CTAs per SM run 128, whose stages
// leave fewer warps idle at the barriers (order 100 x 32: 4.4 ms against 4.7
// with 256); the two CTAs per SM of long transforms need 256 (order 1024: 1.32
// against 1.35 ms), and so does a grid that gives an SM a CTA or two (order 20 x
// 1: 2 us less for both directions).
int threads_for(size_t smem, long long ctas) { return smem <= 56 * 1024 && ctas > 4 * 152 ? 128 : 256; }

// Opens the shared memory that the kernel may use, once per kernel and device.
int set_smem_limit() {
    static std::mutex mu;
    static std::set<int> done;
    int dev = 0;
    ZG_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (done.count(dev)) return ZEST_GPU_OK;
    ZG_CUDA_TRY(cudaFuncSetAttribute(rfft_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    ZG_CUDA_TRY(cudaFuncSetAttribute(rfft_inv_kernel<SpectraIn>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    ZG_CUDA_TRY(cudaFuncSetAttribute(rfft_inv_kernel<ParityIn>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    done.insert(dev);
    return ZEST_GPU_OK;
}

}  // namespace

int launch_rfft_fwd(cudaStream_t s, const FftPlan& plan, const double* x, long long xb, long long si, long long sc,
                    int C, int nm, int batch, int lon_fast, double* F) {
    if (batch <= 0 || C <= 0 || nm <= 0) return ZEST_GPU_OK;
    ZG_TRY(set_smem_limit());
    const int NC = choose_nc(plan, (long long)C * batch);
    const size_t smem = fft_smem_bytes(plan, NC);
    dim3 grid((C + 2 * NC - 1) / (2 * NC), batch);
    rfft_fwd_kernel<<<grid, threads_for(smem, (long long)grid.x * batch), smem, s>>>(plan, x, xb, si, sc, C, nm, NC, lon_fast, F);
    return launch_check("rfft_fwd_kernel");
}

namespace {

template <class In>
int launch_inv(cudaStream_t s, const FftPlan& plan, const In& src, int C, int nm, int batch, int lon_fast, double* x,
               long long xb, long long si, long long sc) {
    if (batch <= 0 || C <= 0) return ZEST_GPU_OK;
    ZG_TRY(set_smem_limit());
    const int NC = choose_nc(plan, (long long)C * batch);
    const size_t smem = fft_smem_bytes(plan, NC);
    dim3 grid((C + 2 * NC - 1) / (2 * NC), batch);
    rfft_inv_kernel<<<grid, threads_for(smem, (long long)grid.x * batch), smem, s>>>(plan, src, C, nm, NC, lon_fast, x, xb, si, sc);
    return launch_check("rfft_inv_kernel");
}

}  // namespace

int launch_rfft_inv(cudaStream_t s, const FftPlan& plan, const double* F, int C, int nm, int batch, int lon_fast,
                    double* x, long long xb, long long si, long long sc) {
    return launch_inv(s, plan, SpectraIn{F, C, nm}, C, nm, batch, lon_fast, x, xb, si, sc);
}

int launch_rfft_inv_parity(cudaStream_t s, const FftPlan& plan, const double* E, int nlat, int nrad, int kh, int j0u,
                           int j0d, int nm, int ms, int batch, int lon_fast, double* x, long long xb, long long si,
                           long long sc) {
    return launch_inv(s, plan, ParityIn{E, ms, nm, nrad, kh, j0u, j0d, batch}, nlat * nrad, nm, batch, lon_fast, x, xb,
                      si, sc);
}

}  // namespace zgpu
