// What the inverse longitude transforms (fft.cu, fixed_fft.cu) read.
#pragma once

#include <cuda_runtime.h>

namespace zgpu {

// Spectra F[b][m][col] as fft.cu lays them out (ms orders per item).
struct SpectraIn {
    const double* F;
    int C, ms;
    __device__ double2 get(int b, int m, int col) const {
        return *reinterpret_cast<const double2*>(F + (((long long)b * ms + m) * C + col) * 2);
    }
};

// Spectra of nm orders formed from the parity sums E_p[b][m][j'][2 rad + {re, im}]
// of folded backward Legendre sums (p, b: B items): E_0 + E_1 at the north node
// lat = j0u + j', E_0 - E_1 at the south node lat = j0d - j' (the equator,
// j0u = j0d, is north).
struct ParityIn {
    const double* E;
    int ms, nm, nrad, kh, j0u, j0d, B;
    __device__ double2 get(int b, int m, int col) const {
        const int lat = col / nrad, rad = col - lat * nrad;
        const bool north = lat >= j0u;
        const int jf = north ? lat - j0u : j0d - lat;
        const double* p = E + ((((long long)b * ms + m) * kh + jf) * nrad + rad) * 2;
        const double2 e0 = *reinterpret_cast<const double2*>(p);
        double2 e1 = make_double2(0.0, 0.0);  // the last order has no degree of the odd parity
        if (m + 1 < nm) e1 = *reinterpret_cast<const double2*>(p + (long long)B * ms * kh * nrad * 2);
        return north ? make_double2(e0.x + e1.x, e0.y + e1.y) : make_double2(e0.x - e1.x, e0.y - e1.y);
    }
};

}  // namespace zgpu
