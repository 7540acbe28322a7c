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

// Launches that are prepared while the kernel before them on the stream runs,
// instead of after its end and flush. Every block of a kernel launched so calls
// after_previous() before it touches memory; it returns once all kernels before
// it have completed and their writes are visible (at once in an ordinary
// launch). Data that those kernels write is not read through the read-only path
// (__ldg, const __restrict__) at an address known beforehand: such loads may be
// moved above the wait. About 2 us a launch where kernels are short: 20 steps
// on 8^3 cells 921 -> 647 us, V-cycles on 128 x 64 x 64 4.9 -> 4.7 ms, the
// gradient of a 32^3 laser run 25.7 -> 24.0 ms.
//
// EARLY: once its own wait is over, the next launch's first blocks may wait on
// the SMs that this kernel's last blocks leave free (allowed before the wait,
// several kernels queue up there: a thousand half-sweeps on 49 x 31 x 27 points
// took 61 ms instead of 43). Not for the particle kernels and the sort: their
// shared memory would leave the waiting kernel its small L1 (a laser between
// walls, 20 steps: 3967 us, 3625 us without).
template <bool EARLY = true>
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P>
struct LaunchAfter {
    void (*kernel)(P...);
    cudaLaunchConfig_t cfg;
    void operator()(P... a) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        (void)cudaLaunchKernelEx(&cfg, kernel, a...);  // callers look at cudaGetLastError, as after <<<>>>
    }
};

template <class... P>
LaunchAfter<P...> launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    LaunchAfter<P...> l{kernel, {}};
    l.cfg.gridDim = grid;
    l.cfg.blockDim = block;
    l.cfg.dynamicSmemBytes = smem;
    l.cfg.stream = stream;
    return l;
}

// The corrected policy's periodic images. Along a periodic dimension of n
// cells (wrap 1) index c of 1..n has images 0 (of n), n + 1 (of 1) and n + 2
// (of 2; of 1 when n is 1); a walled one (wrap 0) has none and keeps its whole
// range. A point's images are the products over the dimensions, itself among
// them; every ghost point along periodic dimensions is the image of exactly
// one such point.
//
// The few points with images, and the ghost points, have threads of their own,
// numbered densely over the slabs they form: in a launch over the whole grid
// every warp holds some (rows are two to six warps long), and pays for them.

// A set of points: dimension by dimension, those whose index is one of
// `listed[d]` there and none of the listed ones in the dimensions before.
struct Slabs {
    int listed[3], rest[3];  // counts per dimension
};

// Point `id` of the slabs as (dimension it is listed in, place in each: of the
// listed in that dimension, of the rest before it, of all after it).
__device__ __forceinline__ bool slab_point(const Slabs &S, uint32_t id, int &d, int at[3]) {
    const uint32_t t1 = S.listed[1] + S.rest[1], t2 = S.listed[2] + S.rest[2];
    uint32_t size = S.listed[0] * t1 * t2;
    uint32_t n1 = t1, n2 = t2;
    d = 0;
    if (id >= size) {
        id -= size;
        d = 1;
        n1 = S.listed[1];
        size = S.rest[0] * n1 * t2;
        if (id >= size) {
            id -= size;
            d = 2;
            n1 = S.rest[1];
            n2 = S.listed[2];
            if (id >= S.rest[0] * n1 * n2) return false;
        }
    }
    const uint32_t q = id / n2;
    at[2] = (int)(id - q * n2);
    at[0] = (int)(q / n1);
    at[1] = (int)(q - at[0] * n1);
    return true;
}

inline int64_t slab_size(const Slabs &S) {
    const int64_t t1 = S.listed[1] + S.rest[1], t2 = S.listed[2] + S.rest[2];
    return S.listed[0] * t1 * t2 + (int64_t)S.rest[0] * (S.listed[1] * t2 + (int64_t)S.rest[1] * S.listed[2]);
}

// The ghost points along the periodic dimensions.
inline Slabs ghost_slabs(const int n[3], const int wrap[3]) {
    Slabs S;
    for (int d = 0; d < 3; d++) {
        S.listed[d] = wrap[d] ? 3 : 0;
        S.rest[d] = wrap[d] ? n[d] : n[d] + 3;
    }
    return S;
}

// Ghost point `id`: its indices c and those of the point it is an image of.
__device__ __forceinline__ bool ghost_point(const Slabs &S, const int n[3], const int wrap[3], uint32_t id, int c[3],
                                            int of[3]) {
    int d;
    if (!slab_point(S, id, d, c)) return false;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (e == d) c[e] = c[e] ? n[e] + c[e] : 0;
        else if (e < d) c[e] += wrap[e];
        of[e] = !wrap[e] || (c[e] >= 1 && c[e] <= n[e]) ? c[e] : c[e] == 0 ? n[e] : c[e] == n[e] + 1 || n[e] == 1 ? 1 : 2;
    }
    return true;
}

// A warp's sums of N values a lane (4 or 8): lane l returns that of value
// total_index<N>(l). Each step over lane bit 16, 8, 4, .. also halves the values
// a lane still holds, which takes 9 FP64 additions for 8 values instead of 40
// (6 instead of 20 for 4); the additions of a sum are paired as in a tree of its
// own, so its bits are that tree's.
template <int N>
__device__ __forceinline__ double warp_totals(double (&v)[N]) {
    const int lane = threadIdx.x & 31;
    int off = 16;
#pragma unroll
    for (int half = N / 2; half >= 1; half >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int q = 0; q < half; q++) {
            const double give = up ? v[q] : v[q + half];
            v[q] = (up ? v[q + half] : v[q]) + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
    for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    return v[0];
}

template <int N>
__device__ __forceinline__ int total_index(int lane) {
    return N == 8 ? ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1)
                  : ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
}

__device__ __forceinline__ void atomic_max_nonneg(double *addr, double v) {
    // non-negative doubles order like their bit patterns
    atomicMax((unsigned long long *)addr, (unsigned long long)__double_as_longlong(v));
}

}  // namespace emoo

#endif
