// dev_common.cuh - device helpers shared by the CUDA translation units.
#ifndef EMOO_DEV_COMMON_CUH
#define EMOO_DEV_COMMON_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "emoo_internal.h"

namespace emoo {

// Division as the reference writes it; when the divisor is a power of two the
// exact reciprocal gives the identical result without the long FP64 divide.
__device__ __forceinline__ double ddiv(double a, double d, double id, int p2) { return p2 ? a * id : a / d; }

__device__ __forceinline__ int64_t gidx(const Geom &g, int i, int j, int k) {
    return (int64_t)i * g.sx + (int64_t)j * g.sy + k;
}

// The 1-based indices (i, j, k) of physical point t (0 <= t < n0 n1 n2, k
// fastest). 32-bit divisions where t fits (every grid these forms allocate):
// a 64-bit divide is a long emulated sequence.
__device__ __forceinline__ void phys_ijk(const int n[3], int64_t t, int &i, int &j, int &k) {
    if (t < ((int64_t)1 << 32)) {
        const uint32_t u = (uint32_t)t, n2 = (uint32_t)n[2], n1 = (uint32_t)n[1];
        const uint32_t r = u / n2;
        k = (int)(u - r * n2) + 1;
        const uint32_t q = r / n1;
        j = (int)(r - q * n1) + 1;
        i = (int)q + 1;
    } else {
        const int64_t r = t / n[2];
        k = (int)(t - r * n[2]) + 1;
        j = (int)(r % n[1]) + 1;
        i = (int)(r / n[1]) + 1;
    }
}

// Grid::getCellID, src/grid/oGrid.cpp:208-227: C truncation plus the ghost
// offset, per axis.
__device__ __forceinline__ void cell_of(const Geom &g, double x, double y, double z, int &ix, int &iy, int &iz) {
    ix = __double2int_rz((x - g.x0[0]) * g.id[0]) + 1;
    iy = __double2int_rz((y - g.x0[1]) * g.id[1]) + 1;
    iz = __double2int_rz((z - g.x0[2]) * g.id[2]) + 1;
}

__device__ __forceinline__ int cell_id(const Geom &g, int ix, int iy, int iz) { return g.cny * ix + g.cnz * iy + iz; }

// Cell indices must address points that exist: ix, ix+1 < n+3. The reference
// asserts 0 <= ix < n+3 (src/grid/oGrid.cpp:212); a position outside that
// range is recorded in the error word and the particle is skipped.
__device__ __forceinline__ bool cell_ok(const Geom &g, int ix, int iy, int iz) {
    return ix >= 0 && iy >= 0 && iz >= 0 && ix + 1 < g.tot[0] && iy + 1 < g.tot[1] && iz + 1 < g.tot[2];
}

__device__ __forceinline__ int species_of(const SpeciesTab &st, int64_t p) {
    int s = 0;
    while (s + 1 < st.nspec && p >= st.off[s + 1]) s++;
    return s;
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The corrected policy's periodic images. Along a periodic dimension of n
// cells (wrap 1) index c of 1..n has images 0 (of n), n + 1 (of 1) and n + 2
// (of 2; of 1 when n is 1); a walled one (wrap 0) has none and keeps its whole
// range. A point's images are the products over the dimensions, itself among
// them; every ghost point along periodic dimensions is the image of exactly
// one such point.
struct Images {
    int64_t off[3][4];  // offsets along each dimension, 0 first
    int n[3];
};

// The point of thread (bx, by, bz) of a launch over `t` = n (periodic) or n + 3
// (walled) points a dimension; false past the range.
__device__ __forceinline__ bool image_point(const int n[3], const int wrap[3], int c[3]) {
    c[0] = (int)blockIdx.z;
    c[1] = (int)(blockIdx.y * blockDim.y + threadIdx.y);
    c[2] = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        c[d] += wrap[d];
        in = in && c[d] < (wrap[d] ? n[d] + 1 : n[d] + 3);
    }
    return in;
}

// Whether the point has images besides itself.
__device__ __forceinline__ bool has_images(const int n[3], const int wrap[3], const int c[3]) {
    bool edge = false;
#pragma unroll
    for (int d = 0; d < 3; d++) edge = edge || (wrap[d] && (c[d] <= 2 || c[d] == n[d]));
    return edge;
}

__device__ __forceinline__ void images_of(const int n[3], const int wrap[3], const int64_t st[3], const int c[3],
                                          Images &im) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
        int m = 0;
        im.off[d][m++] = 0;
        if (wrap[d]) {
            if (c[d] == n[d]) im.off[d][m++] = -n[d] * st[d];
            if (c[d] == 1) im.off[d][m++] = n[d] * st[d];
            if (c[d] == 2 || n[d] == 1) im.off[d][m++] = (n[d] + 2 - c[d]) * st[d];
        }
        im.n[d] = m;
    }
}

// f(offset) for every image but the point itself
template <class F>
__device__ __forceinline__ void for_images(const Images &im, F f) {
    for (int x = 0; x < im.n[0]; x++)
        for (int y = 0; y < im.n[1]; y++)
            for (int z = 0; z < im.n[2]; z++)
                if (x + y + z) f(im.off[0][x] + im.off[1][y] + im.off[2][z]);
}

// Launch shape of image_point (blocks of 32 x 8).
inline dim3 image_grid(const Geom &g, const int wrap[3]) {
    int t[3];
    for (int d = 0; d < 3; d++) t[d] = wrap[d] ? g.n[d] : g.tot[d];
    return dim3((t[2] + 31) / 32, (t[1] + 7) / 8, t[0]);
}

__device__ __forceinline__ void atomic_max_nonneg(double *addr, double v) {
    // non-negative doubles order like their bit patterns
    atomicMax((unsigned long long *)addr, (unsigned long long)__double_as_longlong(v));
}

}  // namespace emoo

#endif
