// Batched real DFT along the longitude axis in 64-bit fixed point: the longitude
// transforms of the split-precision SH path on LonLat grids, and of its Zernike path
// above order 256.  (LatLon grids keep the FP64 transform of fft.cu.)
//
// The FP64 pipe of GB300 retires two operations per clock and SM; the tensor
// cores need the data cut into slices (20 bytes of traffic per value) and a dense
// product with the whole DFT matrix, whose cost per value grows with N.  The
// integer pipe multiplies 32 x 32 -> 64 bits for 32 lanes per clock and SM, so
// three such products -- one term of a 64-bit fixed-point sum -- cost a fifth of
// an FP64 multiply-add, and the transform runs there: every column is scaled by
// its largest value to as many bits as the transform's growth leaves room for, and
// the plan of fft.cu (prime-factor dimensions, Rader, no twiddles between coprime
// factors) is evaluated on (re, im) pairs of 64-bit integers.
//
// Numbers.  A column is held as round(x 2^{hb - e}), |x| < 2^e; the DFT of N
// points grows by at most N sqrt(2) in either component of a packed pair of
// columns (and every partial sum inside a stage, the Rader product included, by
// Cauchy-Schwarz), so hb = 62 - ceil(log2(N sqrt 2)), at most 52, forward, and with
// twice the growth for the inverse, whose packed spectra are twice as large: 52 bits
// forward and 51 inverse at N = 399, 50 and 49 at N = 2047, 49 and 48 at N = 4093,
// against the 48 bits less one or two of headroom of a tensor product's slices.  A
// value x = xh 2^31 + xl and a root c 2^60 = ch 2^31 + cl (xl, cl
// balanced) are multiplied as xh ch, xh cl + xl ch; the dropped xl cl is at most
// one unit of the result.  Sums of products are kept in two 64-bit accumulators
// (at most 10 terms each, bounded by 2^63) and shifted once.  Results become FP64
// by integer operations (i64_ldexp).  A column with an infinity or a NaN gives
// NaN.
//
// What bounds it: the integer pipes (multiply and ALU about 60% busy each).
// Measured, SH order 1024 x 8 (N = 2047), forward 0.45 ms, inverse 0.48; 0.65 as
// K-chunked tensor products with their slicing, 1.3 in FP64.  At N = 399 (Zernike
// order 200 x 64) it takes 16 ms against 13.4 of the tensor products, whose sums
// are short there: orders up to 256 of the Zernike path stay on the tensor cores.
//
// Layout, packing and the meaning of forward and inverse are those of fft.cu.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <set>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.cuh"
#include "spectra.cuh"

namespace zgpu {

namespace {

constexpr int CBITS = 60;   // fraction bits of the roots
constexpr int LIMB = 31;    // bits of the low limb
constexpr int MAXTERM = 10;  // products per accumulator pair: 10 2^30 2^29 + 2^31 2^30 < 2^63

constexpr int IN_REGS = 7;  // largest odd radix done per butterfly in registers
template <int NC>
constexpr int LOG2 = NC == 8 ? 3 : NC == 4 ? 2 : NC == 2 ? 1 : 0;

using Z = longlong2;  // re, im

__device__ __forceinline__ Z zadd(Z a, Z b) { return make_longlong2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ Z zsub(Z a, Z b) { return make_longlong2(a.x - b.x, a.y - b.y); }

using Acc = FixedAcc<CBITS>;  // sum of products value * root
// a W for a root w = {ch, cl of the real part, of the imaginary part}
__device__ __forceinline__ Z zmul(Z a, int4 w) {
    const Limbs x = limbs(a.x), y = limbs(a.y);
    Acc re, im;
    re.add(x, w.x, w.y);
    re.add(y, -w.z, -w.w);
    im.add(x, w.z, w.w);
    im.add(y, w.x, w.y);
    return make_longlong2(re.value(), im.value());
}

// R-point DFT of a small odd R in registers (as dft_odd of fft.cu)
template <int R>
__device__ __forceinline__ void dft_odd(const Z (&t)[R], const int4* __restrict__ w, int wR, Z* __restrict__ y,
                                        int ys) {
    constexpr int h = R / 2;
    Limbs sx[h], sy[h], dx[h], dy[h];
    Z y0 = t[0];
#pragma unroll
    for (int r = 0; r < h; ++r) {
        const Z s = zadd(t[r + 1], t[R - 1 - r]), d = zsub(t[r + 1], t[R - 1 - r]);
        sx[r] = limbs(s.x);
        sy[r] = limbs(s.y);
        dx[r] = limbs(d.x);
        dy[r] = limbs(d.y);
        y0 = zadd(y0, s);
    }
    y[0] = y0;
#pragma unroll
    for (int q = 1; q <= h; ++q) {
        Acc ax, ay, bx, by;  // b: sum of d sin with the table's -sin, so -b
#pragma unroll
        for (int r = 1; r <= h; ++r) {
            const int4 c = w[wR * ((r * q) % R)];
            ax.add(sx[r - 1], c.x, c.y);
            ay.add(sy[r - 1], c.x, c.y);
            bx.add(dx[r - 1], c.z, c.w);
            by.add(dy[r - 1], c.z, c.w);
        }
        const Z a = make_longlong2(t[0].x + ax.value(), t[0].y + ay.value());
        const Z b = make_longlong2(bx.value(), by.value());
        y[q * ys] = make_longlong2(a.x - b.y, a.y + b.x);
        y[(R - q) * ys] = make_longlong2(a.x + b.y, a.y - b.x);
    }
}

template <int R>
__device__ __forceinline__ void butterfly(const Z* __restrict__ x, int xs, Z* __restrict__ y, int ys,
                                          const int4* __restrict__ tw, int tstep, int wR) {
    Z t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) t[r] = x[r * xs];
    if (tstep) {
#pragma unroll
        for (int r = 1; r < R; ++r) t[r] = zmul(t[r], tw[r * tstep]);
    }
    dft_odd<R>(t, tw, wR, y, ys);
}

// Sums and differences of the large radices are written back as limbs.
__device__ __forceinline__ Z pack(Z v) {
    const Limbs a = limbs(v.x), b = limbs(v.y);
    return make_longlong2((long long)(((unsigned long long)unsigned(a.h) << 32) | unsigned(a.l)),
                          (long long)(((unsigned long long)unsigned(b.h) << 32) | unsigned(b.l)));
}
__device__ __forceinline__ Limbs unpack(long long v) { return Limbs{int(v >> 32), int(unsigned(v))}; }

// n / d for n d < 2^32 by the operation's reciprocal (0 stands for d = 1)
__device__ __forceinline__ int divide(int n, unsigned rcp) { return rcp ? int(__umulhi(unsigned(n), rcp)) : n; }

// Butterfly b of an operation: column pair b mod NC, then position within the
// inner rows, butterfly j of the dimension and outer slice.
struct Place {
    int x, y, jm;  // first input and output element, twiddle index
};
template <int NC>
__device__ __forceinline__ Place place(const FftOp& op, int b) {
    const int cp = b & (NC - 1), o = b / NC;
    const int t = divide(o, op.rcp_inner), i = o - t * op.inner;
    const int ou = divide(t, op.rcp_nr), j = t - ou * op.nr;
    const int jq = divide(j, op.rcp_ns), jm = j - jq * op.Ns;
    const int slice = op.base + ou * op.ostride + i;
    return Place{(slice + j * op.inner) * NC + cp, (slice + (jq * op.Ns * op.R + jm) * op.inner) * NC + cp, jm};
}

// One Stockham pass (as fft_stage of fft.cu).
template <int NC>
__device__ __forceinline__ void fixed_stage(Z* __restrict__ src, Z* __restrict__ dst, const int4* __restrict__ tw,
                                            const FftOp& op) {
    const int R = op.R;
    const int step = op.step;
    const int wR = op.nr;  // W_R^m = tw[wR m]
    const int in = op.inner * NC, xs = op.nr * in, ys = op.Ns * in;
    const int nb = op.outer * op.nr * in;
    for (int o = threadIdx.x; o < nb; o += blockDim.x) {
        const Place at = place<NC>(op, o);
        Z* x = src + at.x;
        Z* y = dst + at.y;
        const int tstep = at.jm * step;
        switch (R) {
        case 2: {
            const Z a = x[0];
            Z b = x[xs];
            if (tstep) b = zmul(b, tw[tstep]);
            y[0] = zadd(a, b);
            y[ys] = zsub(a, b);
            break;
        }
        case 4: {
            const Z a = x[0];
            Z b = x[xs], c = x[2 * xs], d = x[3 * xs];
            if (tstep) {
                b = zmul(b, tw[tstep]);
                c = zmul(c, tw[2 * tstep]);
                d = zmul(d, tw[3 * tstep]);
            }
            const Z s0 = zadd(a, c), d0 = zsub(a, c), s1 = zadd(b, d), d1 = zsub(b, d);
            y[0] = zadd(s0, s1);
            y[ys] = make_longlong2(d0.x + d1.y, d0.y - d1.x);  // d0 - i d1
            y[2 * ys] = zsub(s0, s1);
            y[3 * ys] = make_longlong2(d0.x - d1.y, d0.y + d1.x);
            break;
        }
        case 3: butterfly<3>(x, xs, y, ys, tw, tstep, wR); break;
        case 5: butterfly<5>(x, xs, y, ys, tw, tstep, wR); break;
        case 7: butterfly<7>(x, xs, y, ys, tw, tstep, wR); break;
        default: {
            if (tstep) {
                int t2 = tstep;
                for (int r = 1; r < R; ++r) {
                    x[r * xs] = zmul(x[r * xs], tw[t2]);
                    t2 += tstep;
                }
            }
            const int h = R >> 1;
            Z y0 = x[0];
            Z *lo = x + xs, *hi = x + (R - 1) * xs;
            for (int r = 1; r <= h; ++r, lo += xs, hi -= xs) {
                const Z a = *lo, b = *hi;
                const Z s = zadd(a, b);
                *lo = pack(s);
                *hi = pack(zsub(a, b));
                y0 = zadd(y0, s);
            }
            y[0] = y0;
        }
        }
    }
    if (R <= IN_REGS) return;
    __syncthreads();
    // one (butterfly, q) per thread, q slowest, so that the lanes of a warp share roots
    const int h = R >> 1;
    for (int o = threadIdx.x; o < nb * h; o += blockDim.x) {
        const int g = divide(o, op.rcp_nb[LOG2<NC>]), q = g + 1;
        const Place at = place<NC>(op, o - g * nb);
        const Z* x = src + at.x;
        Z* y = dst + at.y;
        const int dm = wR * q;
        int m = dm;
        Z a = x[0], b = make_longlong2(0, 0);
        const Z *lo = x + xs, *hi = x + (R - 1) * xs;
        for (int r0 = 0; r0 < h; r0 += MAXTERM) {
            Acc ax, ay, bx, by;
            const int n = min(h - r0, MAXTERM);
#pragma unroll 4
            for (int r = 0; r < n; ++r, lo += xs, hi -= xs) {
                const Z s = *lo, d = *hi;
                const int4 c = tw[m];
                ax.add(unpack(s.x), c.x, c.y);
                ay.add(unpack(s.y), c.x, c.y);
                bx.add(unpack(d.x), c.z, c.w);
                by.add(unpack(d.y), c.z, c.w);
                m += dm;
                if (m >= op.Nd) m -= op.Nd;
            }
            a = make_longlong2(a.x + ax.value(), a.y + ay.value());
            b = make_longlong2(b.x + bx.value(), b.y + by.value());
        }
        y[q * ys] = make_longlong2(a.x - b.y, a.y + b.x);
        y[(R - q) * ys] = make_longlong2(a.x + b.y, a.y - b.x);
    }
}

// The middle of a Rader dimension (as rader_product of fft.cu).
template <int NC>
__device__ __forceinline__ void fixed_rader(Z* __restrict__ cur, Z* home, const int4* __restrict__ B, const FftOp& op) {
    const int in = op.inner * NC, total = op.Nd * in, b0 = op.base * NC;
    for (int o = threadIdx.x; o < total; o += blockDim.x) {
        const int k = divide(o / NC, op.rcp_inner), i = o - k * in;
        Z* c = cur + b0 + o;
        const Z X = *c;
        Z v = zmul(X, B[k]);
        if (k == 0) {
            Z* z = home + b0 - in + i;
            const Z x0 = *z;
            *z = zadd(x0, X);
            v = zadd(v, x0);
        }
        *c = v;
    }
}

template <int NC>
__device__ __forceinline__ Z* run_plan(Z* a, Z* b, const int4* tab, const FftPlan& plan) {
    for (int s = 0; s < plan.nops; ++s) {
        const FftOp& op = plan.ops[s];
        if (op.R > 0) {
            fixed_stage<NC>(a, b, tab + op.tab, op);
            Z* t = a;
            a = b;
            b = t;
        } else {
            fixed_rader<NC>(a, op.Ns ? b : a, tab + op.tab, op);
        }
        __syncthreads();
    }
    return a;
}

// x(b, i, col) = x + b*xb + i*si + col*sc.
// F: `ms` orders per item, of which m < nm are written.
template <int NC>
__global__ void __launch_bounds__(256) fixed_fwd_kernel(const __grid_constant__ FftPlan plan, int hb,
                                                           const double* __restrict__ x, long long xb, long long si,
                                                           long long sc, int C, int nm, int ms,
                                                           double* __restrict__ F) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int W = 2 * NC;
    __shared__ unsigned top[W];  // largest magnitude's high word per column
    const int N = plan.N;
    int4* tab = reinterpret_cast<int4*>(smem);
    Z* A = reinterpret_cast<Z*>(tab + plan.ntab);
    Z* Bf = A + N * NC;
    const int b = blockIdx.y;
    const int col0 = blockIdx.x * W;
    for (int t = threadIdx.x; t < plan.ntab; t += blockDim.x) tab[t] = plan.itab[t];
    if (threadIdx.x < W) top[threadIdx.x] = 0;
    __syncthreads();
    const double* xbp = x + (long long)b * xb;
    long long* Al = reinterpret_cast<long long*>(A);
    auto high = [](double v) { return unsigned(__double2hiint(v)) & 0x7FFFFFFFu; };
    // a thread keeps one column: rows i0, i0 + rs, ..  Blocks with all their columns
    // load without a check; with one loop for both the compiler needs registers that
    // cost the third CTA per SM (SH order 1024 x 8 0.45 against 0.53 ms; 0.48 with the
    // loads unrolled by 8 instead of 2)
    auto load = [&](auto whole) {
        const int cl = threadIdx.x & (W - 1), i0 = threadIdx.x / W, rs = 256 / W;
        const bool in = decltype(whole)::value || col0 + cl < C;
        const double* p = xbp + (long long)(col0 + cl) * sc + (long long)i0 * si;
        const long long dp = (long long)rs * si;
        unsigned mx = 0;
#pragma unroll 2
        for (int i = i0; i < N; i += rs, p += dp) {
            const double v = in ? *p : 0.0;
            mx = max(mx, high(v));
            Al[plan.in_row[i] * W + cl] = __double_as_longlong(v);
        }
        if (mx) atomicMax(&top[cl], mx);
        __syncthreads();
        const unsigned h = top[cl];
        const int c = 1074 + fixed_scale(h) - hb;
        const bool bad = not_finite(h);
#pragma unroll 4
        for (int i = i0; i < N; i += rs) {
            long long* q = Al + plan.in_row[i] * W + cl;
            *q = bad ? 0 : to_fixed_c(__longlong_as_double(*q), c);
        }
    };
    if (col0 + W <= C) load(std::true_type{});
    else load(std::false_type{});
    __syncthreads();
    const Z* Zr = run_plan<NC>(A, Bf, tab, plan);
    // separate the two real spectra and store conj(X_m), m < nm (twice them: hb + 1)
    const int cp = threadIdx.x & (NC - 1), col = col0 + 2 * cp;
    const unsigned ha = top[2 * cp], hc = top[2 * cp + 1];
    const int sa = fixed_scale(ha) - hb - 1, sb = fixed_scale(hc) - hb - 1;
    const bool bad_a = not_finite(ha), bad_b = not_finite(hc);
    const int m0 = threadIdx.x / NC, dm = blockDim.x / NC;
    double2* out = reinterpret_cast<double2*>(F) + ((long long)b * ms + m0) * C + col;
    const long long dout = (long long)dm * C;
    for (int m = m0; m < nm; m += dm, out += dout) {
        const Z z = Zr[plan.out_row[m] * NC + cp];
        const Z zn = Zr[plan.out_row[m ? N - m : 0] * NC + cp];
        if (col < C)
            out[0] = make_double2(bad_a ? nan64() : i64_ldexp(z.x + zn.x, sa),
                                  bad_a ? nan64() : i64_ldexp(zn.y - z.y, sa));
        if (col + 1 < C)
            out[1] = make_double2(bad_b ? nan64() : i64_ldexp(z.y + zn.y, sb),
                                  bad_b ? nan64() : i64_ldexp(z.x - zn.x, sb));
    }
}

template <int NC>
__global__ void __launch_bounds__(256) fixed_inv_kernel(const __grid_constant__ FftPlan plan, int hb, const ParityIn src,
                                                           int C, int nm, double* __restrict__ x,
                                                           long long xb, long long si, long long sc) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int W = 2 * NC;
    __shared__ unsigned top[W];
    const int N = plan.N;
    int4* tab = reinterpret_cast<int4*>(smem);
    Z* A = reinterpret_cast<Z*>(tab + plan.ntab);
    Z* Bf = A + N * NC;
    const int b = blockIdx.y;
    const int col0 = blockIdx.x * W;
    for (int t = threadIdx.x; t < plan.ntab; t += blockDim.x) tab[t] = plan.itab[t];
    if (threadIdx.x < W) top[threadIdx.x] = 0;
    __syncthreads();
    auto high = [](double v) { return unsigned(__double2hiint(v)) & 0x7FFFFFFFu; };
    double2* Ad = reinterpret_cast<double2*>(A);
    // a thread keeps one pair of columns: orders m0, m0 + dm, ..
    const int cp = threadIdx.x & (NC - 1), colp = col0 + 2 * cp;
    const int m0 = threadIdx.x / NC, dm = blockDim.x / NC;
    unsigned ma = 0, mb = 0;
    for (int m = nm + m0; m <= N - nm; m += dm)  // orders the spectra do not hold
        Ad[plan.in_row[m] * NC + cp] = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int m = m0; m < nm; m += dm) {
        double2 fa = make_double2(0.0, 0.0), fb = fa;
        if (colp < C) fa = src.get(b, m, colp);
        if (colp + 1 < C) fb = src.get(b, m, colp + 1);
        if (m == 0) {  // real
            fa.y = fb.x;
            ma = max(ma, high(fa.x));
            mb = max(mb, high(fb.x));
        } else {
            ma = max(ma, max(high(fa.x), high(fa.y)));
            mb = max(mb, max(high(fb.x), high(fb.y)));
            Ad[plan.in_row[N - m] * NC + cp] = fb;
        }
        Ad[plan.in_row[m] * NC + cp] = fa;
    }
    if (ma) atomicMax(&top[2 * cp], ma);
    if (mb) atomicMax(&top[2 * cp + 1], mb);
    __syncthreads();
    {
        // Hermitian completion of the packed spectra F_a + i F_b, conjugated
        const unsigned ha = top[2 * cp], hc = top[2 * cp + 1];
        const int ca = 1074 + fixed_scale(ha) - hb, cb = 1074 + fixed_scale(hc) - hb;
        const bool bad_a = not_finite(ha), bad_b = not_finite(hc);
        auto fix = [](double v, int c, bool bad) { return bad ? 0ll : to_fixed_c(v, c); };
#pragma unroll 2
        for (int m = m0; m < nm; m += dm) {
            Z* p = A + plan.in_row[m] * NC + cp;
            const double2 fa = *reinterpret_cast<const double2*>(p);
            if (m == 0) {
                *p = make_longlong2(fix(fa.x, ca, bad_a), -fix(fa.y, cb, bad_b));
            } else {
                Z* n = A + plan.in_row[N - m] * NC + cp;
                const double2 fb = *reinterpret_cast<const double2*>(n);
                const long long ax = fix(fa.x, ca, bad_a), ay = fix(fa.y, ca, bad_a);
                const long long bx = fix(fb.x, cb, bad_b), by = fix(fb.y, cb, bad_b);
                *p = make_longlong2(ax - by, -(ay + bx));
                *n = make_longlong2(ax + by, ay - bx);
            }
        }
    }
    __syncthreads();
    const Z* Zr = run_plan<NC>(A, Bf, tab, plan);
    const long long* Zl = reinterpret_cast<const long long*>(Zr);
    double* xbp = x + (long long)b * xb;
    // the second column of a pair is the imaginary part, conjugated
    auto value = [&](int i, int cl, unsigned h) {
        const long long v = Zl[plan.out_row[i] * W + cl];
        return not_finite(h) ? nan64() : i64_ldexp((cl & 1) ? -v : v, fixed_scale(h) - hb);
    };
    const int cl = threadIdx.x & (W - 1), i0 = threadIdx.x / W, rs = blockDim.x / W;
    if (col0 + cl >= C) return;
    const unsigned h = top[cl];
    double* p = xbp + (long long)(col0 + cl) * sc + (long long)i0 * si;
    const long long dp = (long long)rs * si;
#pragma unroll 2
    for (int i = i0; i < N; i += rs, p += dp) *p = value(i, cl, h);
}

// bits of a column's largest value: the growth by N sqrt(2) (`wide`: twice that,
// two spectra in one packed one) stays below 2^62
int headroom_bits(int N, bool wide) {
    const double grow = std::log2(double(N)) + (wide ? 1.5 : 0.5);
    return std::max(1, std::min(52, 62 - int(std::ceil(grow))));
}

// Columns per CTA (a power of two): four CTAs per SM where N allows it, two
// otherwise; fewer where the whole transform would leave SMs without a CTA.
int choose_nc(const FftPlan& plan, long long cols) {
    int nc = 8;
    while (nc > 4 && fft_smem_bytes(plan, nc) > 56 * 1024) nc /= 2;
    while (nc > 1 && fft_smem_bytes(plan, nc) > 110 * 1024) nc /= 2;
    while (nc > 2 && cols < 2LL * nc * 152) nc /= 2;
    return nc;
}

template <class Kern>
int allow_smem(Kern kern) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    ZG_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    const std::pair<const void*, int> key(reinterpret_cast<const void*>(kern), dev);
    if (done.count(key)) return ZEST_GPU_OK;
    ZG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 222 * 1024));
    done.insert(key);
    return ZEST_GPU_OK;
}

// Calls go(integral constant NC, shared memory, grid) for the column count of the size.
template <class Go>
int with_nc(const FftPlan& plan, int C, int batch, Go&& go) {
    const int nc = choose_nc(plan, (long long)C * batch);
    const size_t smem = fft_smem_bytes(plan, nc);
    const dim3 grid((C + 2 * nc - 1) / (2 * nc), batch);
    switch (nc) {
    case 8: return go(std::integral_constant<int, 8>{}, smem, grid);
    case 4: return go(std::integral_constant<int, 4>{}, smem, grid);
    case 2: return go(std::integral_constant<int, 2>{}, smem, grid);
    default: return go(std::integral_constant<int, 1>{}, smem, grid);
    }
}

}  // namespace

void fixed_fft_table(const std::vector<double>& tab, std::vector<int4>& itab) {
    auto limbs_of = [](double c, int& h, int& l) {
        const long long v = std::llrint(std::ldexp(c, CBITS));
        l = int((unsigned)(v & 0x7FFFFFFFll) << 1) >> 1;
        h = int((v - l) >> LIMB);
    };
    itab.resize(tab.size() / 2);
    for (size_t t = 0; t < itab.size(); ++t) {
        limbs_of(tab[2 * t], itab[t].x, itab[t].y);
        limbs_of(tab[2 * t + 1], itab[t].z, itab[t].w);
    }
}

int launch_fixed_fft_fwd(cudaStream_t s, const FftPlan& plan, const double* x, long long xb, long long si,
                         long long sc, int C, int nm, int ms, int batch, double* F) {
    if (batch <= 0 || C <= 0 || nm <= 0) return ZEST_GPU_OK;
    return with_nc(plan, C, batch, [&](auto nc, size_t smem, dim3 grid) -> int {
        constexpr int NC = decltype(nc)::value;
        ZG_TRY(allow_smem(fixed_fwd_kernel<NC>));
        fixed_fwd_kernel<NC><<<grid, 256, smem, s>>>(plan, headroom_bits(plan.N, false), x, xb, si, sc, C, nm, ms, F);
        return launch_check("fixed_fwd_kernel");
    });
}

int launch_fixed_fft_inv_parity(cudaStream_t s, const FftPlan& plan, const double* E, int nlat, int nrad, int kh,
                                int j0u, int j0d, int nm, int ms, int batch, double* x, long long xb, long long si,
                                long long sc) {
    const int C = nlat * nrad;
    if (batch <= 0 || C <= 0) return ZEST_GPU_OK;
    const ParityIn src{E, ms, nm, nrad, kh, j0u, j0d, batch};
    return with_nc(plan, C, batch, [&](auto nc, size_t smem, dim3 grid) -> int {
        constexpr int NC = decltype(nc)::value;
        ZG_TRY(allow_smem(fixed_inv_kernel<NC>));
        fixed_inv_kernel<NC><<<grid, 256, smem, s>>>(plan, headroom_bits(plan.N, true), src, C, nm, x, xb, si, sc);
        return launch_check("fixed_inv_kernel");
    });
}

}  // namespace zgpu
