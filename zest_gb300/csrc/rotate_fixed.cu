// Rotations of real Zernike and SH expansions in 64-bit fixed point (the
// split-precision form of Rotor::rotate, include/rotor.hpp:121-243; rotate_l,
// wignerd_collection.hpp:122-296; the steps are those of rotate.cu).
//
// The d(pi/2) products of one vector are sums of l + 1 terms, too short and too
// many for the tensor cores (sliced operands are 24 bytes per coefficient and the
// intermediate vectors pass through memory three times), and the FP64 pipe retires
// two multiply-adds per clock and SM.  The integer pipe does a term in three
// 32 x 32 -> 64-bit multiply-adds at 32 lanes per clock and SM, five times as many
// terms, so a whole rotation runs in it: a CTA takes a tile of vectors of one
// degree (rotate.cuh), scales each vector by its largest coefficient to HB bits,
// and keeps it in shared memory between the three phases and the two products.
//
// Numbers.  |v| <= 2^(HB + 1/2) per component after the real -> complex step (all
// sqrt(2) times larger, as in rotate.cu), the rotations are orthogonal, so every
// later component is below 2^(HB + 1/2) sqrt(l + 1) <= 2^57.5 (l <= 255), its
// doubled operand below 2^58.5.  Operands are kept as two limbs, d(pi/2) and the
// phases with CB fraction bits.  A sum folds its accumulators every CHUNK terms:
// CHUNK 2^30 2^27 + 2^30 sum |xh| (Cauchy-Schwarz: 2^29.5 over a chunk) < 2^63.
// A dropped low product is below 4 units of 2^-HB of the vector's largest
// coefficient.  A vector with an infinity or a NaN becomes NaN, and so does one
// with an Euler angle whose multiples up to l are not all finite.
//
// Measured, order 64 x 256: 0.43 ms a call (0.40 the kernel); 0.80 as sliced
// tensor products per degree, with an error of 2.8e-14 against 4.5e-15 now; about 1
// in FP64.
#include <cmath>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.cuh"
#include "rotate.cuh"

namespace zgpu {

namespace {

constexpr int CB = 58;     // fraction bits of d(pi/2) and the phases
constexpr int HB = 53;     // bits of a vector's largest coefficient
constexpr int CHUNK = 30;  // terms per accumulator pair, and one more at each end
using Acc = FixedAcc<CB>;

__device__ __forceinline__ int2 constant(double c) {  // |c| <= 1
    const Limbs x = limbs(__double2ll_rn(c * double(1ll << CB)));
    return make_int2(x.h, x.l);
}

// d(pi/2) of all l < L as limbs
__global__ void fixed_wigner_kernel(long long n, const double* __restrict__ d, int2* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = constant(d[i]);
}

// phases[b][k][m] = e^{-i m angle_k} as limbs {re h, re l, im h, im l}; limbs hold no
// NaN, so the phase of a multiple that is not finite is zero
__global__ void fixed_phase_kernel(int L, int batch, const double* __restrict__ euler, int type, int4* __restrict__ ph) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (m >= L || b >= batch) return;
    double ang[3];
    convert_angles(euler + 3 * b, type, ang[0], ang[1], ang[2]);
    for (int k = 0; k < 3; ++k) {
        int4 w = make_int4(0, 0, 0, 0);
        const double x = -double(m) * ang[k];
        if (isfinite(x)) {
            double s, c;
            sincos(x, &s, &c);
            const int2 re = constant(c), im = constant(s);
            w = make_int4(re.x, re.y, im.x, im.y);
        }
        ph[((long long)b * 3 + k) * L + m] = w;
    }
}
// a phase has a part of at least 1 / sqrt(2), and with it a high limb
__device__ __forceinline__ bool is_phase(int4 w) { return (w.x | w.z) != 0; }

struct Z {
    long long x, y;
};
__device__ __forceinline__ Z zmul(Z a, int4 w) {
    const Limbs x = limbs(a.x), y = limbs(a.y);
    Acc re, im;
    re.add(x, w.x, w.y);
    re.add(y, -w.z, -w.w);
    im.add(x, w.z, w.w);
    im.add(y, w.x, w.y);
    return Z{re.value(), im.value()};
}
// a / sqrt(2)
__device__ __forceinline__ long long over_sqrt2(long long a) {
    constexpr long long c = 203809653520824722ll;  // 2^CB / sqrt(2)
    constexpr int cl = int(unsigned(c & 0x7FFFFFFF) << 1) >> 1;
    Acc t;
    t.add(limbs(a), int((c - cl) >> 31), cl);
    return t.value();
}
// the operand of the sums (doubled for m > 0), as limbs
__device__ __forceinline__ int2 operand(long long v, int m) {
    const Limbs x = limbs(m ? v + v : v);
    return make_int2(x.h, x.l);
}

template <int TV>
__device__ __forceinline__ void load_row(const int2* __restrict__ p, Limbs (&v)[TV]) {
#pragma unroll
    for (int j = 0; j < TV; j += 2) {
        const int4 x = *reinterpret_cast<const int4*>(p + j);
        v[j] = Limbs{x.x, x.y};
        v[j + 1] = Limbs{x.z, x.w};
    }
}

// X(+-pi/2) row m of TV vectors (as xsum of rotate.cu)
template <int TV>
__device__ __forceinline__ void xsum(const int2* __restrict__ vr, const int2* __restrict__ vi, int VS,
                                     const int2* __restrict__ d, int l, int m, bool transpose, Z (&r)[TV]) {
    const int ld = l + 1, q = (l + m) & 1;
    Acc re[TV], im[TV];
    auto term = [&](int mp, const int2* v, Acc(&acc)[TV]) {
        const int2 c = d[ld * mp + m];
        Limbs w[TV];
        load_row<TV>(v + mp * VS, w);
#pragma unroll
        for (int j = 0; j < TV; ++j) acc[j].add(w[j], c.x, c.y);
    };
#pragma unroll
    for (int j = 0; j < TV; ++j) r[j] = Z{0, 0};
    auto fold = [&]() {
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            r[j].x += re[j].value();
            r[j].y += im[j].value();
            re[j] = Acc();
            im[j] = Acc();
        }
    };
    term(0, vr, re);
    int a = q ? 1 : 2, b = q ? 2 : 1;  // m' of the real and of the imaginary sum
    int left = l >= 2 ? l / 2 : 0;     // pairs (a, b) with both at most l: max(a, b) = 2, 4, ..
    while (left > 0) {
        const int n = min(left, CHUNK);
#pragma unroll 2
        for (int k = 0; k < n; ++k, a += 2, b += 2) {
            term(a, vr, re);
            term(b, vi, im);
        }
        left -= n;
        if (left > 0) fold();
    }
    if (a <= l) term(a, vr, re);
    if (b <= l) term(b, vi, im);
    fold();
    if (!transpose) {  // d(m, m') = (-1)^(m+m') d(m', m): one sign for all terms of a sum
        const bool odd = l & 1;
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (odd) r[j].x = -r[j].x;
            else r[j].y = -r[j].y;
        }
    }
}

// (four CTAs per SM hide the latency of the multiply-add chains: 0.40 ms against
// 0.72 with the registers of one)
template <int TV>
__global__ void __launch_bounds__(256, 4) rotate_fixed_kernel(RotSet S, int elems, double* __restrict__ coeffs,
                                                           const int2* __restrict__ wig, const int4* __restrict__ ph) {
    extern __shared__ __align__(16) int2 fbuf[];
    __shared__ long long off[128];
    __shared__ int item[128];
    __shared__ unsigned top[128];  // high word of a vector's largest magnitude; an infinity's: it becomes NaN
    const int l = S.L - 1 - int(blockIdx.y);
    const int V = rot_tile(l, elems, TV), VS = rot_stride(V);
    const long long cnt = S.count(l), first = (long long)blockIdx.x * V;
    if (first >= cnt) return;
    const int nv = int(min((long long)V, cnt - first)), ld = l + 1, L = S.L;
    const int2* d = wig + wig_off(l);
    int2* vr = fbuf;
    int2* vi = vr + ld * VS;
    int2* tr = vi + ld * VS;
    int2* ti = tr + ld * VS;
    for (int v = threadIdx.x; v < V; v += blockDim.x) {
        item[v] = -1;
        if (v < nv) S.vector(l, first + v, &item[v], &off[v]);
    }
    __syncthreads();
    // one warp per vector: its scale, then real -> complex and the gamma phase
    const int lane = threadIdx.x & 31;
    for (int v = threadIdx.x >> 5; v < V; v += blockDim.x >> 5) {
        if (v >= nv) {
            for (int m = lane; m < ld; m += 32) vr[m * VS + v] = vi[m * VS + v] = make_int2(0, 0);
            continue;
        }
        const double* c = coeffs + off[v];
        auto high = [](double x) { return unsigned(__double2hiint(x)) & 0x7FFFFFFFu; };
        unsigned mx = 0;
        for (int m = lane; m < ld; m += 32) {
            // the sine part of m = 0 takes no part, unless it is not finite
            const unsigned im = high(c[2 * m + 1]);
            mx = max(mx, max(high(c[2 * m]), m || not_finite(im) ? im : 0u));
        }
        const int4* pa = ph + (long long)item[v] * 3 * L;
        const int4* pg = pa + 2 * L;
        if (lane < 3 && !is_phase(pa[lane * L + l])) mx = 0x7FF00000u;
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) top[v] = mx;
        const int cr = 1074 + fixed_scale(mx) - HB + 1;  // one bit more of the operand, dropped by the shift below
        for (int m = lane; m < ld; m += 32) {
            Z x{0, 0};
            if (!not_finite(mx)) {
                // 52 bits of the largest coefficient, at scale HB
                x = Z{to_fixed_c(c[2 * m], cr) * 2, m ? -to_fixed_c(c[2 * m + 1], cr) * 2 : 0};
                if (m == 0) x.x = 2 * over_sqrt2(x.x);
            }
            x = zmul(x, pg[m]);
            vr[m * VS + v] = operand(x.x, m);
            vi[m * VS + v] = operand(x.y, m);
        }
    }
    __syncthreads();
    const int items = ld * ((nv + TV - 1) / TV);
    for (int e = threadIdx.x; e < items; e += blockDim.x) {  // X(pi/2), beta phase
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        Z r[TV];
        xsum<TV>(vr + v0, vi + v0, VS, d, l, m, false, r);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            const Z x = zmul(r[j], ph[((long long)item[v0 + j] * 3 + 1) * L + m]);
            tr[m * VS + v0 + j] = operand(x.x, m);
            ti[m * VS + v0 + j] = operand(x.y, m);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < items; e += blockDim.x) {  // X(-pi/2), alpha phase, complex -> real
        const int g = e / ld, m = e - g * ld, v0 = g * TV;
        Z r[TV];
        xsum<TV>(tr + v0, ti + v0, VS, d, l, m, true, r);
#pragma unroll
        for (int j = 0; j < TV; ++j) {
            if (v0 + j >= nv) break;
            Z x = zmul(r[j], ph[(long long)item[v0 + j] * 3 * L + m]);
            if (m == 0) x = Z{over_sqrt2(x.x), 0};
            const int sc = fixed_scale(top[v0 + j]) - HB;
            const bool bad = not_finite(top[v0 + j]);
            double* c = coeffs + off[v0 + j] + 2 * m;
            c[0] = bad ? nan64() : i64_ldexp(x.x, sc);
            c[1] = bad ? nan64() : i64_ldexp(-x.y, sc);
        }
    }
}

template <class Count>
int launch_rotate(cudaStream_t s, const RotSet& S, Count&& count, double* coeffs, const int2* wigner, const int4* ph) {
    int elems, tv = 4;
    rot_shape(S.L, count, 4, 1024, &elems, &tv);
    return launch_tiles(S.L, tv, 4, elems, count, [&](dim3 grid, size_t smem) -> int {
        auto go = [&](auto kern) -> int {
            ZG_TRY(allow_smem(kern));
            kern<<<grid, 256, smem, s>>>(S, elems, coeffs, wigner, ph);
            return launch_check("rotate_fixed_kernel");
        };
        return tv == 4 ? go(rotate_fixed_kernel<4>) : go(rotate_fixed_kernel<2>);
    });
}

int launch_phases(cudaStream_t s, int L, int items, const double* euler, int type, int4* ph) {
    fixed_phase_kernel<<<dim3((L + 127) / 128, items), 128, 0, s>>>(L, items, euler, type, ph);
    return launch_check("fixed_phase_kernel");
}

}  // namespace

int launch_fixed_wigner(cudaStream_t s, int L, const double* wigner, int2* out) {
    const long long n = wig_off(L);
    if (n <= 0) return ZEST_GPU_OK;
    fixed_wigner_kernel<<<unsigned(std::min<long long>((n + 255) / 256, 4096)), 256, 0, s>>>(n, wigner, out);
    return launch_check("fixed_wigner_kernel");
}

int launch_rotate_fixed(cudaStream_t s, int kind, int L, int batch, double* coeffs, long long cstride,
                        const int2* wigner, const double* euler, int type, double* phase_scratch) {
    if (batch <= 0 || L <= 0) return ZEST_GPU_OK;
    if (L > kFixedRotateOrder) return fail(ZEST_GPU_ERR_UNSUPPORTED, "fixed-point rotation: orders up to 256");
    int4* ph = reinterpret_cast<int4*>(phase_scratch);
    ZG_TRY(launch_phases(s, L, batch, euler, type, ph));
    const RotSet S{kind, L, batch, cstride, nullptr, nullptr, nullptr};
    return launch_rotate(s, S, [&](int l) { return (long long)batch * vec_count(kind, L, l); }, coeffs, wigner, ph);
}

int launch_rotate_fixed_ragged(cudaStream_t s, int Lmax, int items, double* coeffs, const long long* coff,
                               const int4* vecs, const std::vector<long long>& voff, const long long* voff_dev,
                               const int2* wigner, const double* euler, int type, double* phase_scratch) {
    if (items <= 0 || Lmax <= 0 || voff.back() <= 0) return ZEST_GPU_OK;
    if (Lmax > kFixedRotateOrder) return fail(ZEST_GPU_ERR_UNSUPPORTED, "fixed-point rotation: orders up to 256");
    int4* ph = reinterpret_cast<int4*>(phase_scratch);
    ZG_TRY(launch_phases(s, Lmax, items, euler, type, ph));
    const RotSet S{0, Lmax, items, 0, vecs, voff_dev, coff};
    return launch_rotate(s, S, [&](int l) { return voff[size_t(l) + 1] - voff[size_t(l)]; }, coeffs, wigner, ph);
}

}  // namespace zgpu
