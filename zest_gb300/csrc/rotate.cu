// Rotations of real Zernike and SH expansions, FP64 (Rotor::rotate and
// Rotor::polar_rotate, include/rotor.hpp:121-378).
//
// Per expansion and per (n, l) vector of l+1 complex coefficients:
//   real -> complex   m > 0: {a, b} -> {a/sqrt2, -b/sqrt2}    zernike_expansion.hpp:484-575
//   rotate_l          e^{-im g'} X(pi/2) e^{-im b'} X(-pi/2) e^{-im a'}
//                                                             wignerd_collection.hpp:122-296
//   complex -> real   m > 0: {a, b} -> {a sqrt2, -b sqrt2}    zernike_expansion.hpp:577-634
// with (a', b', g') = detail::convert(euler, type), rotor.hpp:68-81.
//
// X(pi/2) in the reference uses the parity structure of d^l(pi/2) and of the
// complex coefficients of a real function: output m with q = (l+m) & 1 takes
//   Re <- 1/2 d(m,0) Re v_0 + sum_{m' >= 1, m'+q even} d(m,m') Re v_m'
//   Im <-                     sum_{m' >= 1, m'+q odd } d(m,m') Im v_m'
// (times 2), and X(-pi/2) the same with d transposed.  d(m,m') is read as
// (-1)^(m+m') d(m',m) so that consecutive lanes read consecutive addresses; the
// sign is the same for all terms of a sum and goes on the result.
//
// Bound: the FP64 pipe (two multiply-adds per clock and SM), so every lane of
// every FP64 instruction has to do work and no operation is spent on scaling.
//   * A CTA takes a tile of vectors of one degree l, from any items.  A thread
//     owns one output row m and TV vectors, so one table element read from L1
//     feeds TV products, and the (m, vector group) pairs are dealt to the
//     threads in one sequence: lanes idle only at its end.  (One warp per
//     vector, lane = m, left 40% of the lanes of the mean l idle.)
//   * The coefficients are kept sqrt(2) times larger than the complex ones:
//     (a, -b) as they are for m > 0, and sqrt(2) a for m = 0 alone.  The factor
//     2 of the sums is an exponent increment on the stored operand.
// Measured, order 64 x 256, rotation and both gradients: 9.93 -> 2.99 ms.
//
// Zernike vectors are n >= 1 and l in the parity range of n starting at 0
// for even n (the reference's indices(1) rounds down, so l = 0 is "rotated",
// which zeroes Im c_{n00}); SH vectors are l >= 1.
#include "common.cuh"
#include "kernels.cuh"
#include "rotate.cuh"

namespace zgpu {

namespace {

constexpr int MAXL = 2048;  // longest vector (order) supported

// phases[b][k][m] = e^{-i m angle_k}, k = alpha, beta, gamma
__global__ void phase_kernel(int L, int batch, const double* __restrict__ euler, int type, double2* __restrict__ ph) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (m >= L || b >= batch) return;
    double ang[3];
    convert_angles(euler + 3 * b, type, ang[0], ang[1], ang[2]);
    for (int k = 0; k < 3; ++k) {
        double s, c;
        sincos(-double(m) * ang[k], &s, &c);
        ph[((long long)b * 3 + k) * L + m] = make_double2(c, s);
    }
}

__device__ __forceinline__ double2 cmul(double2 c, double2 r) {
    return make_double2(c.x * r.x - c.y * r.y, c.x * r.y + c.y * r.x);
}

// 2 x by the exponent field: exact like the product, no FP64 operation
__device__ __forceinline__ double twice(double x) {
    const int hi = __double2hiint(x), e = hi & 0x7FF00000;
    if (e != 0 && e < 0x7FE00000) return __hiloint2double(hi + 0x00100000, __double2loint(x));
    return x + x;
}
__device__ __forceinline__ double flip(double x, int sign) {  // sign: 0 or the sign bit
    return __hiloint2double(__double2hiint(x) ^ sign, __double2loint(x));
}
__device__ __forceinline__ double2 conjugate(double2 z) { return make_double2(z.x, -z.y); }

// The operand of the sums for component m of a vector: doubled for m > 0 (the
// sums are 2 (1/2 d(m,0) v_0 + ..)).
__device__ __forceinline__ double2 operand(double2 v, int m) {
    return m ? make_double2(twice(v.x), twice(v.y)) : v;
}

template <int TV>
__device__ __forceinline__ void load_row(const double* __restrict__ p, double (&v)[TV]) {
    if constexpr (TV == 1) {
        v[0] = p[0];
    } else {
#pragma unroll
        for (int j = 0; j < TV; j += 2) {
            const double2 x = *reinterpret_cast<const double2*>(p + j);
            v[j] = x.x;
            v[j + 1] = x.y;
        }
    }
}

// X(+-pi/2) rows m of TV vectors of each of NS sets: r[s][j] + i w[s][j].
// vr[s], vi[s]: the operands [m'][vector], at the thread's first vector.
template <int TV, int NS>
__device__ __forceinline__ void xsum(const double* const (&vr)[NS], const double* const (&vi)[NS], int VS,
                                     const double* __restrict__ d, int l, int m, bool transpose,
                                     double (&re)[NS][TV], double (&im)[NS][TV]) {
    const int ld = l + 1, q = (l + m) & 1;
    const double d0 = d[m];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        double v[TV];
        load_row<TV>(vr[s], v);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            re[s][j] = d0 * v[j];
            im[s][j] = 0.0;
        }
    }
    auto term = [&](int mp, const double* const (&v)[NS], double (&acc)[NS][TV]) {
        const double x = d[ld * mp + m];
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            double w[TV];
            load_row<TV>(v[s] + (size_t)mp * VS, w);
#pragma unroll
            for (int j = 0; j < TV; ++j) acc[s][j] = fma(x, w[j], acc[s][j]);
        }
    };
    int a = q ? 1 : 2, b = q ? 2 : 1;  // m' of the real and of the imaginary sum
#pragma unroll 2
    for (; max(a, b) <= l; a += 2, b += 2) {
        term(a, vr, re);
        term(b, vi, im);
    }
    if (a <= l) term(a, vr, re);
    if (b <= l) term(b, vi, im);
    if (!transpose) {
        // d(m, m') = (-1)^(m+m') d(m', m): m + m' = l + q + m' is of the parity of
        // l in the real sum (d(m, 0) = 0 where it is not), of the other in the
        // imaginary one
        const int sr = (l & 1) ? int(0x80000000u) : 0, si = sr ^ int(0x80000000u);
#pragma unroll
        for (int s = 0; s < NS; ++s)
#pragma unroll
            for (int j = 0; j < TV; ++j) {
                re[s][j] = flip(re[s][j], sr);
                im[s][j] = flip(im[s][j], si);
            }
    }
}

constexpr double kSqrt2 = 1.41421356237309504880168872420969808;

// sqrt(2) times the complex coefficient m of a real vector, and back
__device__ __forceinline__ double2 to_complex(const double* __restrict__ c, int m) {
    return m ? make_double2(c[2 * m], -c[2 * m + 1]) : make_double2(kSqrt2 * c[0], kSqrt2 * c[1]);
}
__device__ __forceinline__ void to_real(double* __restrict__ c, int m, double2 v) {
    c[2 * m] = m ? v.x : v.x * (1.0 / kSqrt2);
    c[2 * m + 1] = m ? -v.y : v.y * (1.0 / kSqrt2);
}

template <int TV>
__global__ void __launch_bounds__(256) rotate_kernel(RotSet S, int elems, double* __restrict__ coeffs,
                                                     const double* __restrict__ wig, const double2* __restrict__ ph) {
    extern __shared__ __align__(16) double rbuf[];
    __shared__ long long off[128];
    __shared__ int item[128];
    const int l = S.L - 1 - int(blockIdx.y);
    const int V = rot_tile(l, elems, TV), VS = rot_stride(V);
    const long long cnt = S.count(l), first = (long long)blockIdx.x * V;
    if (first >= cnt) return;
    const int nv = int(min((long long)V, cnt - first)), ld = l + 1, L = S.L;
    const double* d = wig + wig_off(l);
    double* vr = rbuf;
    double* vi = vr + (size_t)ld * VS;
    double* tr = vi + (size_t)ld * VS;
    double* ti = tr + (size_t)ld * VS;
    for (int v = threadIdx.x; v < V; v += blockDim.x) {
        item[v] = -1;
        if (v < nv) S.vector(l, first + v, &item[v], &off[v]);
    }
    __syncthreads();
    // real -> complex, gamma phase
    for (int e = threadIdx.x; e < ld * V; e += blockDim.x) {
        const int v = e / ld, m = e - v * ld;
        double2 x = make_double2(0.0, 0.0);
        if (v < nv) x = operand(cmul(to_complex(coeffs + off[v], m), ph[((long long)item[v] * 3 + 2) * L + m]), m);
        vr[m * VS + v] = x.x;
        vi[m * VS + v] = x.y;
    }
    __syncthreads();
    const int items = ld * ((nv + TV - 1) / TV);
    for (int e = threadIdx.x; e < items; e += blockDim.x) {  // X(pi/2), beta phase
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        const double* const pr[1] = {vr + v0};
        const double* const pi[1] = {vi + v0};
        double re[1][TV], im[1][TV];
        xsum<TV, 1>(pr, pi, VS, d, l, m, false, re, im);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            const double2 x = operand(cmul(make_double2(re[0][j], im[0][j]),
                                           ph[((long long)item[v0 + j] * 3 + 1) * L + m]), m);
            tr[m * VS + v0 + j] = x.x;
            ti[m * VS + v0 + j] = x.y;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < items; e += blockDim.x) {  // X(-pi/2), alpha phase, complex -> real
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        const double* const pr[1] = {tr + v0};
        const double* const pi[1] = {ti + v0};
        double re[1][TV], im[1][TV];
        xsum<TV, 1>(pr, pi, VS, d, l, m, true, re, im);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            to_real(coeffs + off[v0 + j], m, cmul(make_double2(re[0][j], im[0][j]),
                                                  ph[(long long)item[v0 + j] * 3 * L + m]));
        }
    }
}

// Gradient of <ybar, rotate(x)> with respect to the three converted angles
// (alpha', beta', gamma'), part[vector][k], and (xbar not null) the coefficient
// cotangent D^T ybar.  The rotation is E_a X(-pi/2) E_b X(pi/2) E_g on the real
// coefficients, with E_t = diag(e^{-i m t}) and every factor orthogonal, so
// with the states before and after each phase
//   v = E_g x,  w = E_b X(pi/2) v,  z = X(-pi/2) w
// and the cotangents carried back
//   u1 = E_a^T ybar,  u2 = X(pi/2) u1,  u4 = X(-pi/2) E_b^T u2,  xbar = E_g^T u4
// the derivatives are <u1, (-i m) z>, <u2, (-i m) w> and <u4, (-i m) v>: four
// products with d(pi/2) for all of it.  Carrying the three derivatives forward
// took five and the cotangent two more.  Same tiles as rotate_kernel, the two
// chains side by side as two sets of operands.
template <int TV>
__global__ void __launch_bounds__(256) rotate_grad_kernel(RotSet S, int elems, int nvec, const double* __restrict__ x,
                                                          const double* ybar, double* xbar,
                                                          const double* __restrict__ wig,
                                                          const double2* __restrict__ ph, double* __restrict__ part) {
    extern __shared__ __align__(16) double rbuf[];
    __shared__ long long off[128];
    __shared__ int item[128];
    const int l = S.L - 1 - int(blockIdx.y);
    const int V = rot_tile(l, elems, TV), VS = rot_stride(V);
    const long long cnt = S.count(l), first = (long long)blockIdx.x * V;
    if (first >= cnt) return;
    const int nv = int(min((long long)V, cnt - first)), ld = l + 1, L = S.L;
    const double* d = wig + wig_off(l);
    const size_t as = (size_t)ld * VS;
    double* f0r = rbuf;  // v (forward), u1 (cotangent), then w and E_b^T u2; pb: the beta terms
    double* f0i = f0r + as;
    double* b0r = f0i + as;
    double* b0i = b0r + as;
    double* f1r = b0i + as;
    double* f1i = f1r + as;
    double* b1r = f1i + as;
    double* b1i = b1r + as;
    double* pb = b1i + as;
    for (int v = threadIdx.x; v < V; v += blockDim.x) {
        item[v] = -1;
        if (v < nv) S.vector(l, first + v, &item[v], &off[v]);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ld * V; e += blockDim.x) {
        const int v = e / ld, m = e - v * ld;
        double2 a = make_double2(0.0, 0.0), b = a;
        if (v < nv) {
            const double2* p = ph + (long long)item[v] * 3 * L + m;
            a = operand(cmul(to_complex(x + off[v], m), p[2 * L]), m);
            b = operand(cmul(to_complex(ybar + off[v], m), conjugate(p[0])), m);
        }
        f0r[m * VS + v] = a.x;
        f0i[m * VS + v] = a.y;
        b0r[m * VS + v] = b.x;
        b0i[m * VS + v] = b.y;
    }
    __syncthreads();
    const int items = ld * ((nv + TV - 1) / TV);
    // m <u, -i v> of two components
    auto term = [](double2 u, double2 v, int m) { return double(m) * (u.x * v.y - u.y * v.x); };
    for (int e = threadIdx.x; e < items; e += blockDim.x) {
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        const double* const pr[2] = {f0r + v0, b0r + v0};
        const double* const pi[2] = {f0i + v0, b0i + v0};
        double re[2][TV], im[2][TV];
        xsum<TV, 2>(pr, pi, VS, d, l, m, false, re, im);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            const int at = m * VS + v0 + j;
            const double2 p = ph[((long long)item[v0 + j] * 3 + 1) * L + m];
            const double2 w = cmul(make_double2(re[0][j], im[0][j]), p);
            const double2 u2 = make_double2(re[1][j], im[1][j]);
            const double2 u3 = operand(cmul(u2, conjugate(p)), m), w2 = operand(w, m);
            // beta: the cotangent after E_b is u2, the state w
            pb[at] = term(u2, w, m);
            f1r[at] = w2.x;
            f1i[at] = w2.y;
            b1r[at] = u3.x;
            b1i[at] = u3.y;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < items; e += blockDim.x) {
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        const double* const pr[2] = {f1r + v0, b1r + v0};
        const double* const pi[2] = {f1i + v0, b1i + v0};
        double re[2][TV], im[2][TV];
        xsum<TV, 2>(pr, pi, VS, d, l, m, true, re, im);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            const int at = m * VS + v0 + j;
            const double2 z = make_double2(re[0][j], im[0][j]), u4 = make_double2(re[1][j], im[1][j]);
            // the stored u1 and v are doubled for m > 0; their own element is not
            // read again and takes the alpha and gamma terms (twice their value)
            const double pa = term(make_double2(b0r[at], b0i[at]), z, m);
            const double pg = term(u4, make_double2(f0r[at], f0i[at]), m);
            f0r[at] = pa;
            f0i[at] = pg;
            if (xbar) to_real(xbar + off[v0 + j], m, cmul(u4, conjugate(ph[((long long)item[v0 + j] * 3 + 2) * L + m])));
        }
    }
    __syncthreads();
    // sums over m, 4 lanes per (vector, angle), in a fixed order
    const int lane4 = threadIdx.x & 3;
    for (int s0 = threadIdx.x >> 2; s0 - int(threadIdx.x >> 2) < 3 * nv; s0 += blockDim.x >> 2) {
        const bool in = s0 < 3 * nv;
        const int v = in ? s0 / 3 : 0, k = in ? s0 - 3 * v : 0;
        const double* p = k == 0 ? f0r : k == 1 ? pb : f0i;
        double t = 0.0;
        for (int m = 1 + lane4; in && m < ld; m += 4) t += p[m * VS + v];
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        if (in && lane4 == 0) {
            const int c = vec_count(S.kind, L, l);
            const long long i = first + v, b = i / c;
            part[(b * nvec + vec_before(S.kind, L, l) + (i - b * c)) * 3 + k] = k == 1 ? t : 0.5 * t;
        }
    }
}

// Per expansion: the sum over its vectors of the angle partials (fixed order,
// so the result does not depend on scheduling), mapped back from the
// converted angles to the Euler angles of the call (rotor.hpp:68-81):
// object (a', b', g') = (a - pi/2, b, g + pi/2); coordinate (-g - pi/2, -b, -a + pi/2).
// xbar not null: the pair that no rotation touches (l = n = 0) is copied too.
__global__ void euler_grad_reduce_kernel(int nvec, const double* __restrict__ part, int type,
                                         double* __restrict__ grad, const double* ybar, double* xbar,
                                         long long cstride) {
    __shared__ double red[3][256];
    const int b = blockIdx.x;
    double s[3] = {0.0, 0.0, 0.0};
    for (int v = threadIdx.x; v < nvec; v += blockDim.x)
        for (int k = 0; k < 3; ++k) s[k] += part[((long long)b * nvec + v) * 3 + k];
    for (int k = 0; k < 3; ++k) red[k][threadIdx.x] = s[k];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w)
            for (int k = 0; k < 3; ++k) red[k][threadIdx.x] += red[k][threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (xbar) {
            xbar[b * cstride] = ybar[b * cstride];
            xbar[b * cstride + 1] = ybar[b * cstride + 1];
        }
        const double da = red[0][0], db = red[1][0], dg = red[2][0];
        double* g = grad + 3 * (long long)b;
        if (type == 0) {
            g[0] = da;
            g[1] = db;
            g[2] = dg;
        } else {
            g[0] = -dg;
            g[1] = -db;
            g[2] = -da;
        }
    }
}

// Euler angles of the inverse rotation, for either convention: (-g, -b, -a).
__global__ void invert_euler_kernel(int batch, const double* __restrict__ e, double* __restrict__ out) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    const double a = e[3 * b], be = e[3 * b + 1], g = e[3 * b + 2];
    out[3 * b] = -g;
    out[3 * b + 1] = -be;
    out[3 * b + 2] = -a;
}

__global__ void polar_kernel(int L, int nvec, int batch, double* __restrict__ coeffs, long long cstride, int kind,
                             const int2* __restrict__ vec_list, const double* __restrict__ angles, int type) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long vid = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
    if (vid >= (long long)nvec * batch) return;
    const int b = int(vid / nvec);
    const int2 nl = vec_list[vid - (long long)b * nvec];
    const int n = nl.x, l = nl.y;
    double* c = coeffs + b * cstride + 2 * vec_base(kind, n, l);
    const double ang = type == 0 ? angles[b] : -angles[b];
    const double isq2 = 1.0 / 1.41421356237309504880168872420969808;
    const double sq2 = 1.41421356237309504880168872420969808;
    for (int m = lane; m <= l; m += 32) {
        double2 x = make_double2(c[2 * m], c[2 * m + 1]);
        if (m > 0) { x.x *= isq2; x.y *= -isq2; }
        double s, co;
        sincos(-double(m) * ang, &s, &co);
        x = cmul(x, make_double2(co, s));
        if (m > 0) { x.x *= sq2; x.y *= -sq2; }
        c[2 * m] = x.x;
        c[2 * m + 1] = x.y;
    }
}

}  // namespace

namespace {

// (m, vector) pairs per CTA: 64 KB of the four arrays of a rotation (three
// CTAs per SM), 72 KB of the nine of the gradient
constexpr int ROT_ELEMS = 2048, GRAD_ELEMS = 1024;

template <class Count>
int launch_rotate(cudaStream_t s, const RotSet& S, Count&& count, double* coeffs, const double* wigner,
                  const double2* ph) {
    int elems, tv = 8;
    rot_shape(S.L, count, 4, ROT_ELEMS, &elems, &tv);
    return launch_tiles(S.L, tv, 4, elems, count, [&](dim3 grid, size_t smem) -> int {
        auto go = [&](auto kern) -> int {
            ZG_TRY(allow_smem(kern));
            kern<<<grid, 256, smem, s>>>(S, elems, coeffs, wigner, ph);
            return launch_check("rotate_kernel");
        };
        return tv == 8 ? go(rotate_kernel<8>) : tv == 4 ? go(rotate_kernel<4>) : go(rotate_kernel<2>);
    });
}

}  // namespace

int launch_rotate_vectors(cudaStream_t s, int kind, int L, int batch, double* coeffs, long long cstride,
                          const double* wigner, const double* euler, int type, double* phase_scratch) {
    if (batch <= 0 || L <= 0) return ZEST_GPU_OK;
    if (L > MAXL) return fail(ZEST_GPU_ERR_UNSUPPORTED, "rotation order above 2048");
    ZG_TRY(launch_phases(s, L, batch, euler, type, phase_scratch));
    const RotSet S{kind, L, batch, cstride, nullptr, nullptr, nullptr};
    return launch_rotate(s, S, [&](int l) { return (long long)batch * vec_count(kind, L, l); }, coeffs, wigner,
                         reinterpret_cast<const double2*>(phase_scratch));
}

int launch_rotate_euler_grad(cudaStream_t s, int kind, int L, int batch, const double* x, const double* ybar,
                             long long cstride, int nvec, const double* wigner, const double* euler, int type,
                             double* phase_scratch, double* part, double* grad, double* xbar) {
    if (batch <= 0) return ZEST_GPU_OK;
    if (L > 1024) return fail(ZEST_GPU_ERR_UNSUPPORTED, "rotation gradient: order above 1024");
    if (nvec <= 0) {
        ZG_CUDA_TRY(cudaMemsetAsync(grad, 0, (size_t)batch * 3 * sizeof(double), s));
        return ZEST_GPU_OK;
    }
    ZG_TRY(launch_phases(s, L, batch, euler, type, phase_scratch));
    const RotSet S{kind, L, batch, cstride, nullptr, nullptr, nullptr};
    const double2* ph = reinterpret_cast<const double2*>(phase_scratch);
    const auto count = [&](int l) { return (long long)batch * vec_count(kind, L, l); };
    int elems, tv = 4;
    rot_shape(L, count, 9, GRAD_ELEMS, &elems, &tv);
    ZG_TRY(launch_tiles(L, tv, 9, elems, count, [&](dim3 grid, size_t smem) -> int {
        auto go = [&](auto kern) -> int {
            ZG_TRY(allow_smem(kern));
            kern<<<grid, 256, smem, s>>>(S, elems, nvec, x, ybar, xbar, wigner, ph, part);
            return launch_check("rotate_grad_kernel");
        };
        return tv == 4 ? go(rotate_grad_kernel<4>) : go(rotate_grad_kernel<2>);
    }));
    euler_grad_reduce_kernel<<<batch, 256, 0, s>>>(nvec, part, type, grad, ybar, xbar, cstride);
    return launch_check("euler_grad_reduce_kernel");
}

int launch_rotate_ragged(cudaStream_t s, int Lmax, int items, double* coeffs, const long long* coff, const int4* vecs,
                         const std::vector<long long>& voff, const long long* voff_dev, const double* wigner,
                         const double* euler, int type, double* phase_scratch) {
    if (items <= 0 || Lmax <= 0 || voff.back() <= 0) return ZEST_GPU_OK;
    if (Lmax > MAXL) return fail(ZEST_GPU_ERR_UNSUPPORTED, "rotation order above 2048");
    ZG_TRY(launch_phases(s, Lmax, items, euler, type, phase_scratch));
    const RotSet S{0, Lmax, items, 0, vecs, voff_dev, coff};
    return launch_rotate(s, S, [&](int l) { return voff[size_t(l) + 1] - voff[size_t(l)]; }, coeffs, wigner,
                         reinterpret_cast<const double2*>(phase_scratch));
}

int launch_phases(cudaStream_t s, int Lmax, int items, const double* euler, int type, double* phase_scratch) {
    if (items <= 0 || Lmax <= 0) return ZEST_GPU_OK;
    phase_kernel<<<dim3((Lmax + 127) / 128, items), 128, 0, s>>>(Lmax, items, euler, type,
                                                                reinterpret_cast<double2*>(phase_scratch));
    return launch_check("phase_kernel");
}

int launch_invert_euler(cudaStream_t s, int batch, const double* euler, double* out) {
    if (batch <= 0) return ZEST_GPU_OK;
    invert_euler_kernel<<<(batch + 127) / 128, 128, 0, s>>>(batch, euler, out);
    return launch_check("invert_euler_kernel");
}

int launch_polar_vectors(cudaStream_t s, int kind, int L, int batch, double* coeffs, long long cstride,
                         const int2* vec_list, int nvec, const double* angles, int type) {
    if (batch <= 0 || nvec <= 0) return ZEST_GPU_OK;
    const long long total = (long long)nvec * batch;
    polar_kernel<<<(unsigned)((total + 7) / 8), 8 * 32, 0, s>>>(L, nvec, batch, coeffs, cstride, kind, vec_list,
                                                               angles, type);
    return launch_check("polar_kernel");
}

}  // namespace zgpu
