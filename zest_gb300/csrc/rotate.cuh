// What the FP64 (rotate.cu) and the fixed-point (rotate_fixed.cu) rotation kernels
// share: the rotated vectors of a launch and their tiles of one degree.
#pragma once

#include <algorithm>

#include "common.cuh"

namespace zgpu {

__device__ __forceinline__ void convert_angles(const double* e, int type, double& a, double& b, double& g) {
    const double pi = 3.14159265358979323846264338327950288;
    const double ar = e[0] - 0.5 * pi, br = e[1], gr = e[2] + 0.5 * pi;
    if (type == 0) { a = ar; b = br; g = gr; }
    else { a = -gr; b = -br; g = -ar; }
}

// First coefficient of vector (n, l): Zernike tetrahedral layout (kind 0),
// SH triangle (kind 1) or row-skipping triangle, floor(l^2 / 4) (kind 2).
__device__ __forceinline__ long long vec_base(int kind, int n, int l) {
    return kind == 0 ? zidx(n, l, 0) : kind == 1 ? tri_idx(l, 0) : ((long long)l * l) >> 2;
}

// Rotated vectors of degree l of one expansion of order L, and how many of lower
// degree come before them: Zernike n = l, l + 2, .. < L (l = 0 from n = 2), SH one
// for l >= 1, row-skipping one per l of the parity of L - 1.
__host__ __device__ inline int vec_count(int kind, int L, int l) {
    if (kind == 0) return l == 0 ? (L - 1) / 2 : (L - l + 1) / 2;
    if (kind == 1) return l >= 1 ? 1 : 0;
    return (l & 1) == ((L - 1) & 1) ? 1 : 0;
}
__device__ inline int vec_before(int kind, int L, int l) {  // Zernike and SH
    if (l == 0) return 0;
    return kind == 0 ? (L - 1) / 2 + (L * L / 4 - (L - l + 1) * (L - l + 1) / 4) : l - 1;
}

// The vectors a launch rotates: those of `batch` expansions of one order
// (vecs null), or the list vecs = {item, n, l, first pair} sorted by l, those of
// degree l at [voff[l], voff[l + 1]), item i's coefficients at coff[i].
struct RotSet {
    int kind, L, batch;
    long long cstride;
    const int4* vecs;
    const long long* voff;
    const long long* coff;
    __device__ long long count(int l) const {
        return vecs ? voff[l + 1] - voff[l] : (long long)batch * vec_count(kind, L, l);
    }
    __device__ void vector(int l, long long i, int* item, long long* off) const {
        if (vecs) {
            const int4 w = vecs[voff[l] + i];
            *item = w.x;
            *off = coff[w.x] + 2 * (long long)w.w;
            return;
        }
        const int c = vec_count(kind, L, l);
        const int b = int(i / c), k = int(i - (long long)b * c);
        *item = b;
        *off = b * cstride + 2 * vec_base(kind, kind == 0 ? (l == 0 ? 2 : l) + 2 * k : l, l);
    }
};

// Vectors per CTA for degree l: about `elems` (m, vector) pairs, a multiple of TV.
__host__ __device__ inline int rot_tile(int l, int elems, int TV) {
    const int v = elems / (l + 1) / TV * TV;
    return v < TV ? TV : (v > 128 ? 128 : v);
}
// Row stride of the [m][vector] arrays in shared memory (an even pad against
// bank conflicts of the column-wise stores; 16-byte loads stay aligned).
__host__ __device__ inline int rot_stride(int V) { return V >= 16 ? V + 2 : V; }

// (m, vector) pairs per CTA, `most` where that gives every SM two CTAs (fewer
// for small batches), and vectors per thread TV <= tv: as many as leave a CTA
// one output row per thread, and as fit (`arrays` doubles per pair within 160
// KB; TV = 2 does up to the largest order).
template <class Count>
inline void rot_shape(int L, Count&& count, int arrays, int most, int* elems, int* tv) {
    long long total = 0;
    for (int l = 0; l < L; ++l) total += count(l) * (l + 1);
    *elems = int(std::min<long long>(most, std::max<long long>(256, total / (2 * 152))));
    while (*tv > 2 && (*elems < *tv * 256 || (size_t)arrays * 8 * L * *tv > 160 * 1024)) *tv /= 2;
}

// Launches kernel(TV) over the tiles of every degree, the largest degrees first.
template <class Count, class Go>
inline int launch_tiles(int L, int tv, int arrays, int elems, Count&& count, Go&& go) {
    long long tiles = 0;
    size_t smem = 0;
    for (int l = 0; l < L; ++l) {
        const long long c = count(l);
        if (c <= 0) continue;
        const int V = rot_tile(l, elems, tv);
        tiles = std::max(tiles, (c + V - 1) / V);
        smem = std::max(smem, (size_t)arrays * 8 * (l + 1) * rot_stride(V));
    }
    if (tiles == 0) return ZEST_GPU_OK;
    if (tiles > 0x7fffffff || smem > 220 * 1024) return fail(ZEST_GPU_ERR_UNSUPPORTED, "rotation: too many vectors");
    return go(dim3((unsigned)tiles, (unsigned)L), smem);
}

template <class Kern>
inline int allow_smem(Kern kern) {
    ZG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
    return ZEST_GPU_OK;
}

}  // namespace zgpu
