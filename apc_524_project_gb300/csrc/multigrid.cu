// multigrid.cu - geometric multigrid for the field start (no reference
// counterpart). It solves the discrete equations whose fixed point
// Poisson_Solver::run_poisson_solver_ (src/poisson/poisson.cpp:216-241)
// iterates towards: at every unknown point of the grid the 7-point Laplacian
// of u equals f = mult R. A dimension with periodic field boundaries has the
// unknowns 1..n and wraps; one with external boundaries holds the PoissonBC
// values on planes 1 and n + 1 (src/poisson/poissonBC.cpp:67-80) and has the
// unknowns 2..n.
//
// Precision: FP64 throughput on this GPU is a small fraction of FP32's, so
// the solution u and the residual r = f - Lu are FP64, and each outer step
// solves the correction equation L e = r approximately by one FP32 V-cycle,
// then u += e (iterative refinement: the FP64 residual sets the accuracy, the
// V-cycle only the rate).
//
// Levels are vertex-centred: coarse index C sits on fine index 2C - 1 along a
// coarsened dimension, so periodic grids of even P halve and external grids
// keep their boundary planes on boundary planes (the correction is zero
// there). A dimension coarsens while its P is even and at least 4; the others
// keep their spacing (semi-coarsening). One V-cycle: two red-black
// Gauss-Seidel sweeps, residual, full-weighting restriction, the coarser
// cycle, trilinear prolongation, two sweeps; the coarsest level is swept
// until its few unknowns settle. A level runs in one of three ways by its size:
// those of at most 4096 unknowns have their whole part of the cycle inside one
// thread block, in its shared memory (launched one kernel per stage, they would
// cost a launch latency each for a few microseconds of work, and from global
// memory each stage would wait on L2); those that fit one tile a SM take a leg
// of the cycle a launch; larger ones a kernel a stage. Each level is a dense
// (P+2)^3 block; periodic neighbours are found by index wrap, so no ghost
// planes are kept. Red and black do not colour a periodic dimension of odd P
// (points 1 and P are neighbours of one colour), so a level with one smooths
// by damped Jacobi half-steps between u and a second buffer instead: no two
// threads touch one point, and the result does not depend on their order.
// One outer step (V-cycle, correction, new FP64 residual and its maximum) is
// a CUDA graph, replayed until max |r| <= rtol max |r0|.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "dev_common.cuh"
#include "emoo_internal.h"
#include "f64_ops.cuh"

namespace emoo {
namespace {

struct Lv {
    int P[3];         // points per dimension (see above)
    int per[3];       // 1: periodic
    int lo[3], hi[3]; // unknown index range
    int crs[3];       // 1: the next level halves this dimension
    int64_t sx, sy;   // strides of the (P+2)^3 block
    float c[3];       // 1 / h^2
    float diag;       // 2 (c0 + c1 + c2)
    float idiag;      // 1 / diag
    int rb;           // 1: red-black Gauss-Seidel; 0: damped Jacobi
    float *u, *f;
    float *w;         // second buffer of u
};

// the FP64 solution and right side, on level 0's layout
struct Fine {
    double c[3];
    double diag;
    double *u, *f;
};

struct MgState {
    int n[3];
    int per[3];
    double d[3];
    std::vector<Lv> lv;
    size_t tail_from = 0;  // first level of the shared-memory tail (lv.size(): none)
    uint4 *tail_pts = nullptr;  // its table of points
    Fine fine = {};
    double *part = nullptr;   // per-block sums
    double *hpart = nullptr;  // pinned host copy
    double *dmax = nullptr;   // device max |r|
    double *hmax = nullptr;   // pinned host copy
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int graph_launches = 0;   // kernels per replay
};

constexpr int RB = 256;      // reduction blocks
constexpr int NU = 2;        // smoothing sweeps before and after the coarse correction
constexpr float OMEGA = 6.0f / 7.0f;  // Jacobi damping, the 7-point stencil's smoothing optimum
constexpr int TAIL_MAX = 4096;    // levels of at most this many unknowns run in the one-block tail
constexpr int TAIL_WARP = 32;     // and of this many on one warp of it
constexpr int TAIL_LEVELS = 16;
constexpr int TAIL_THREADS = 1024;

template <class LV>  // Lv, or the tail's levels with 32-bit strides
__device__ __forceinline__ auto lidx(const LV &L, int i, int j, int k) -> decltype(L.sx + L.sy) {
    return i * L.sx + j * L.sy + k;
}
__device__ __forceinline__ int wrap_dn(const Lv &L, int d, int i) { return (L.per[d] && i == 1) ? L.P[d] : i - 1; }
__device__ __forceinline__ int wrap_up(const Lv &L, int d, int i) { return (L.per[d] && i == L.P[d]) ? 1 : i + 1; }

// sum over the six neighbours, each weighted by 1/h^2 of its dimension
template <class R, class C>
__device__ __forceinline__ R nb_sum(const Lv &L, const C *c, const R *u, int i, int j, int k) {
    return c[0] * (u[lidx(L, wrap_dn(L, 0, i), j, k)] + u[lidx(L, wrap_up(L, 0, i), j, k)]) +
           c[1] * (u[lidx(L, i, wrap_dn(L, 1, j), k)] + u[lidx(L, i, wrap_up(L, 1, j), k)]) +
           c[2] * (u[lidx(L, i, j, wrap_dn(L, 2, k))] + u[lidx(L, i, j, wrap_up(L, 2, k))]);
}

// What a level's u takes with a new right side f, by who reads it next: nothing
// (tiles that begin with f, the tail), zero, or the first half-sweep from zero,
// which needs no neighbours (red points, or all of the Jacobi partner w).
enum { START_NONE, START_ZERO, START_SWEPT };

__device__ __forceinline__ void start_level(const Lv &L, int start, int64_t o, int parity, float f) {
    if (start == START_ZERO) L.u[o] = 0.0f;
    if (start != START_SWEPT) return;
    const float v = (0.0f - f) * L.idiag;
    if (L.rb) L.u[o] = parity ? 0.0f : v;
    else L.w[o] = OMEGA * v;
}

// The FP64 residual of the fine problem: level 0's right side takes it (as
// FP32), level 0's correction restarts, and *dmax the maximum |r|,
// taken over the FP32 values (the stop test needs no more): this kernel runs
// on the FP64 pipe, so everything after the residual itself stays off it.
__global__ void k_mg_residual64(Lv L, Fine F, double *dmax, int start) {
    after_previous();
    __shared__ float sh[8];
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    float a = 0.0f;
    if (k <= L.hi[2] && j <= L.hi[1] && i <= L.hi[0]) {
        const int64_t o = lidx(L, i, j, k);
        const float r = f64_to_f32(F.f[o] - (nb_sum(L, F.c, F.u, i, j, k) - F.diag * F.u[o]));
        L.f[o] = r;
        start_level(L, start, o, (i + j + k) & 1, r);
        a = fabsf(r);
    }
    for (int off = 16; off > 0; off >>= 1) a = fmaxf(a, __shfl_down_sync(0xffffffffu, a, off));
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    if ((tid & 31) == 0) sh[tid >> 5] = a;
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < (int)((blockDim.x * blockDim.y) >> 5); w++) a = fmaxf(a, sh[w]);
        atomic_max_nonneg(dmax, f64_of_f32(a));
    }
}

// Full-weighting restriction of r around the fine point at r, its neighbours at
// offsets `dn` and `up` per dimension. All 27 taps, those of a dimension that
// keeps its points (crs 0) with weight zero: straight code whose loads are in
// flight together (loops that skipped taps took 2 us a level).
template <class I>
__device__ __forceinline__ float restrict_sum(const int *crs, const float *r, const I *dn, const I *up) {
    float w[3][3];
    I o[3][3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        w[d][0] = w[d][2] = crs[d] ? 0.25f : 0.0f;
        w[d][1] = crs[d] ? 0.5f : 1.0f;
        o[d][0] = crs[d] ? dn[d] : 0;
        o[d][1] = 0;
        o[d][2] = crs[d] ? up[d] : 0;
    }
    float s = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const float *q = r + o[0][a] + o[1][b];
            float row = w[2][0] * q[o[2][0]];
            row += w[2][1] * q[0];
            row += w[2][2] * q[o[2][2]];
            s += w[0][a] * w[1][b] * row;
        }
    return s;
}

// the same on a whole level, at a coarse point, where the neighbour below may be
// found by wrapping
template <class LV>
__device__ __forceinline__ float restrict_value(const LV &F, const float *r, int I, int J, int K) {
    using S = decltype(F.sx + F.sy);
    const int at[3] = {F.crs[0] ? 2 * I - 1 : I, F.crs[1] ? 2 * J - 1 : J, F.crs[2] ? 2 * K - 1 : K};
    const S up[3] = {F.sx, F.sy, 1};
    S dn[3];
#pragma unroll
    for (int d = 0; d < 3; d++) dn[d] = F.per[d] && at[d] == 1 ? (F.P[d] - 1) * up[d] : -up[d];
    return restrict_sum(F.crs, r + lidx(F, at[0], at[1], at[2]), dn, up);
}

// coarse index pair and weight of the second feeding fine index f of a
// dimension that coarsens (crs) or keeps its points
__device__ __forceinline__ void interp_at(int crs, int f, int &c0, int &c1, float &w1) {
    const int half = crs && !(f & 1);
    c0 = crs ? (f + 1) >> 1 : f;
    c1 = c0 + half;
    w1 = half ? 0.5f : 0.0f;
}

// the same on a whole level, where the second may be found by wrapping
template <class LV>
__device__ __forceinline__ void interp(const LV &F, const LV &Cl, int d, int f, int &c0, int &c1, float &w1) {
    interp_at(F.crs[d], f, c0, c1, w1);
    if (Cl.per[d] && c1 > Cl.P[d]) c1 = 1;
}

// trilinear interpolation of the coarse correction to a fine point
template <class LV>
__device__ __forceinline__ float prolong_value(const LV &Cl, const LV &F, int i, int j, int k) {
    int ci[2], cj[2], ck[2];
    float wi, wj, wk;
    interp(F, Cl, 0, i, ci[0], ci[1], wi);
    interp(F, Cl, 1, j, cj[0], cj[1], wj);
    interp(F, Cl, 2, k, ck[0], ck[1], wk);
    // all eight taps, zero-weighted ones on a repeated (cached) address: the
    // weights change with the parity of k, so skipping taps would split warps
    const float Wi[2] = {1.0f - wi, wi}, Wj[2] = {1.0f - wj, wj}, Wk[2] = {1.0f - wk, wk};
    float s = 0.0f;
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const auto row = ci[a] * Cl.sx + cj[b] * Cl.sy;
            s += Wi[a] * Wj[b] * (Wk[0] * Cl.u[row + ck[0]] + Wk[1] * Cl.u[row + ck[1]]);
        }
    return s;
}

// ---- levels above the tail, a kernel a stage (large levels; see tile_size)

// One colour of a red-black Gauss-Seidel sweep: the points with
// (i + j + k) & 1 == colour take u = (neighbour sum - f) / diag.
__global__ void k_mg_smooth(Lv L, int colour) {
    after_previous();
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (j > L.hi[1] || i > L.hi[0]) return;
    const int k = L.lo[2] + ((colour + i + j + L.lo[2]) & 1) + 2 * (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (k > L.hi[2]) return;
    const int64_t o = lidx(L, i, j, k);
    L.u[o] = (nb_sum(L, L.c, L.u, i, j, k) - L.f[o]) * L.idiag;
}

// One damped Jacobi half-step at the unknowns, src -> dst.
__global__ void k_mg_jacobi(Lv L, const float *src, float *dst) {
    after_previous();
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (k > L.hi[2] || j > L.hi[1] || i > L.hi[0]) return;
    const int64_t o = lidx(L, i, j, k);
    const float x = src[o];
    dst[o] = x + OMEGA * ((nb_sum(L, L.c, src, i, j, k) - L.f[o]) * L.idiag - x);
}

// w = f - Laplacian(u) at the unknowns (FP32 levels)
__global__ void k_mg_residual(Lv L) {
    after_previous();
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (k > L.hi[2] || j > L.hi[1] || i > L.hi[0]) return;
    const int64_t o = lidx(L, i, j, k);
    L.w[o] = L.f[o] - (nb_sum(L, L.c, L.u, i, j, k) - L.diag * L.u[o]);
}

__global__ void k_mg_restrict(Lv F, Lv Cl, int start) {
    after_previous();
    const int K = Cl.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int J = Cl.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int I = Cl.lo[0] + blockIdx.z;
    if (K > Cl.hi[2] || J > Cl.hi[1] || I > Cl.hi[0]) return;
    const int64_t o = lidx(Cl, I, J, K);
    const float f = restrict_value(F, F.w, I, J, K);
    Cl.f[o] = f;
    start_level(Cl, start, o, (I + J + K) & 1, f);
}

__global__ void k_mg_prolong(Lv Cl, Lv F) {
    after_previous();
    const int k = F.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = F.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = F.lo[0] + blockIdx.z;
    if (k > F.hi[2] || j > F.hi[1] || i > F.hi[0]) return;
    F.u[lidx(F, i, j, k)] += prolong_value(Cl, F, i, j, k);
}

// The last half-sweep of level 0 (black points, or the Jacobi step from w), its
// finished correction added to the solution.
__global__ void k_mg_finish(Lv L, Fine F) {
    after_previous();
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (k > L.hi[2] || j > L.hi[1] || i > L.hi[0]) return;
    const int64_t o = lidx(L, i, j, k);
    float e;
    if (L.rb) {
        e = (i + j + k) & 1 ? (nb_sum(L, L.c, L.u, i, j, k) - L.f[o]) * L.idiag : L.u[o];
    } else {
        const float x = L.w[o];
        e = x + OMEGA * ((nb_sum(L, L.c, L.w, i, j, k) - L.f[o]) * L.idiag - x);
    }
    F.u[o] += f64_of_f32(e);
}

// ---- smaller levels above the tail, in tiles
//
// A block holds a tile of T^3 points and their halo in shared memory and takes
// all stages of one leg of the cycle there, so that a leg is one launch and
// reads and writes the level once:
//   DOWN   u = 0, NU sweeps, u out; residual, its restriction the next level's f
//   UP     u plus the next level's interpolated correction, NU sweeps, u out
//   SWEEP  NU sweeps (a coarsest level too large for the tail)
// A half-sweep is valid one point less far into the halo than the one before
// it; halo points are computed again by each block that needs them, from the
// same values by the same arithmetic. No block reads what another writes: UP
// and SWEEP go from one buffer of u to the other, DOWN starts from zero.
//
// A thread owns a column of the tile along dimension 0 (or a segment of one)
// in every stage: its neighbours along the column stay in registers between
// points, which leaves six shared loads a point, and a point costs no index
// arithmetic. The loads of PIPE points are issued before the first of them is
// stored, and the level's arrays come by asynchronous copies, all in flight at
// once: with a wait a point the legs took 2.5 times as long. Plane strides are
// even and row strides odd, so that the two colours of neighbouring lanes,
// which sit one plane apart, fall on different banks.
enum { DOWN, UP, SWEEP };
constexpr int HS = 2 * NU;         // half-sweeps of a leg
constexpr int TILE_MAX = 8;        // largest T; even, so that coarse points sit on tile starts
constexpr int TILE_THREADS = 640;  // two segments of the (TILE_MAX + 2 HS + 1)^2 = 289 columns
constexpr int PIPE = 4;

struct TileLeg {
    int T;
    const float *src;  // u in (UP, SWEEP)
    float *dst;        // u out
    double *sol;       // not null: the FP64 solution takes it instead (level 0's last leg)
    int start;         // DOWN: of the next level
};

__host__ __device__ __forceinline__ int tile_sy(int e2) { return e2 | 1; }
__host__ __device__ __forceinline__ int tile_sx(int e1, int e2) { return (e1 * tile_sy(e2) + 1) & ~1; }

// index i of a periodic dimension of P points into 1..P
__device__ __forceinline__ int wrapped(int i, int P) {
    if (i >= 1 && i <= P) return i;
    const int q = (i - 1) % P;
    return q < 0 ? q + P + 1 : q + 1;
}

__device__ __forceinline__ void copy_async(float *to, const float *from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One stage on a column: v(o) at its points o0, o0 + st, ... (`count` of them)
// from the neighbours in `from` and from f, stored in `to`. `st` is two planes
// for one colour, one for all points.
template <bool BOTH, class V>
__device__ __forceinline__ void column(const Lv &L, const float *from, const float *f, float *to, int o0, int count,
                                       int sx, int sy, V v) {
    if (count <= 0) return;
    const int st = BOTH ? sx : 2 * sx;
    float below = from[o0 - sx], here = BOTH ? from[o0] : 0.0f;
    for (int p = 0; p < count; p += PIPE, o0 += PIPE * st) {
        float up[PIPE], y0[PIPE], y1[PIPE], z0[PIPE], z1[PIPE], ff[PIPE];
#pragma unroll
        for (int q = 0; q < PIPE; q++) {
            const int o = p + q < count ? o0 + q * st : o0;
            up[q] = from[o + sx];
            y0[q] = from[o - sy];
            y1[q] = from[o + sy];
            z0[q] = from[o - 1];
            z1[q] = from[o + 1];
            ff[q] = f[o];
        }
#pragma unroll
        for (int q = 0; q < PIPE; q++) {
            if (p + q >= count) break;
            const float nb = L.c[0] * (below + up[q]) + L.c[1] * (y0[q] + y1[q]) + L.c[2] * (z0[q] + z1[q]);
            to[o0 + q * st] = v(nb, ff[q], here);
            below = BOTH ? here : up[q];
            here = up[q];
        }
    }
}

template <bool RBGS, int MODE>
__global__ void __launch_bounds__(TILE_THREADS, 1) k_mg_tile(const __grid_constant__ Lv L, const __grid_constant__ Lv C,
                                                             const __grid_constant__ TileLeg G) {
    after_previous();
    extern __shared__ float sm[];
    const int bt[3] = {(int)blockIdx.z, (int)blockIdx.y, (int)blockIdx.x};
    int b0[3], bs[3], first[3], last[3];  // tile with halo: origin and size; its own points
#pragma unroll
    for (int d = 0; d < 3; d++) {
        first[d] = 1 + bt[d] * G.T;
        last[d] = min(first[d] + G.T - 1, L.P[d]);
        // DOWN: the residual's point below a coarsened tile, its stencil, and
        // the half-sweeps after the first, which needs no neighbours
        const int low = MODE == DOWN ? HS + L.crs[d] : HS;
        b0[d] = first[d] - low;
        bs[d] = last[d] - first[d] + 1 + low + HS;
    }
    const int sy = tile_sy(bs[2]), sx = tile_sx(bs[1], bs[2]), n = bs[0] * sx;
    float *u = sm, *f = sm + n, *t = sm + 2 * n;  // t: Jacobi only
    // this thread's column (offset c in each plane) and segment of it
    const int cols = bs[1] * sy, segs = (int)blockDim.x / cols;
    const int seg = threadIdx.x / cols, c = threadIdx.x - seg * cols;
    const int J = b0[1] + c / sy, K = b0[2] + c % sy;
    const bool mine = seg < segs && c % sy < bs[2];
    // its points i of rows lo..hi
    auto rows = [&](int lo, int hi, int &i0, int &i1) {
        const int len = (hi - lo + segs) / segs;
        i0 = lo + seg * len;
        i1 = min(i0 + len - 1, hi);
    };
    // is the column within `low`, `high` of the tile's own and of the unknowns?
    // Then its rows of these
    auto part = [&](const int *low, int high, int &i0, int &i1) {
        int lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = first[d] - low[d];
            hi[d] = last[d] + high;
            if (!L.per[d]) {
                lo[d] = max(lo[d], L.lo[d]);
                hi[d] = min(hi[d], L.hi[d]);
            }
        }
        rows(lo[0], hi[0], i0, i1);
        return mine && J >= lo[1] && J <= hi[1] && K >= lo[2] && K <= hi[2];
    };
    auto place = [&](int i) { return (i - b0[0]) * sx + c; };
    int i0, i1;
    if (mine) {  // the level's arrays, zero outside its unknowns
        const bool in = (L.per[1] || (J >= L.lo[1] && J <= L.hi[1])) && (L.per[2] || (K >= L.lo[2] && K <= L.hi[2]));
        const int64_t col =
            (L.per[1] ? wrapped(J, L.P[1]) : J) * L.sy + (L.per[2] ? wrapped(K, L.P[2]) : K);
        rows(b0[0], b0[0] + bs[0] - 1, i0, i1);
        for (int i = i0; i <= i1; i++) {
            const int o = place(i);
            if (in && (L.per[0] || (i >= L.lo[0] && i <= L.hi[0]))) {
                const int64_t g = (L.per[0] ? wrapped(i, L.P[0]) : i) * L.sx + col;
                copy_async(f + o, L.f + g);
                // red points take their first value from black ones
                if (MODE != DOWN && (!RBGS || ((i + J + K) & 1))) copy_async(u + o, G.src + g);
            } else {
                f[o] = 0.0f;
                if (MODE != DOWN) u[o] = 0.0f;
            }
            if (MODE == DOWN || !RBGS) (MODE == DOWN ? u : t)[o] = 0.0f;
        }
    }
    float *co = sm + (RBGS ? 2 : 3) * n;  // UP: the coarse correction around the tile
    int e0[3], es[3];
    if (MODE == UP) {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            e0[d] = L.crs[d] ? (b0[d] + 1) >> 1 : b0[d];
            es[d] = (L.crs[d] ? ((b0[d] + bs[d] - 1) >> 1) + 1 : b0[d] + bs[d] - 1) - e0[d] + 1;
        }
        for (int q = threadIdx.x; q < es[0] * es[1] * es[2]; q += blockDim.x) {
            const int a = q / es[2];
            int x[3] = {e0[0] + a / es[1], e0[1] + a % es[1], e0[2] + q - a * es[2]};
            bool in = true;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (C.per[d]) x[d] = wrapped(x[d], C.P[d]);
                else in = in && x[d] >= C.lo[d] && x[d] <= C.hi[d];
            }
            if (in) copy_async(co + q, C.u + lidx(C, x[0], x[1], x[2]));
            else co[q] = 0.0f;
        }
    }
    copies_done();
    if (MODE == DOWN && mine) {  // the first half-sweep, from zero, on the whole tile
        for (int i = i0; i <= i1; i++) {
            const int o = place(i);
            const float v = (0.0f - f[o]) * L.idiag;
            if (!RBGS) t[o] = OMEGA * v;
            else if (((i + J + K) & 1) == 0) u[o] = v;
        }
    }
    if (MODE == UP) {  // the coarse correction, at the unknowns
        __syncthreads();
        const int low[3] = {HS, HS, HS};
        if (part(low, HS, i0, i1)) {
            int cj[2], ck[2];
            float wj, wk;
            interp_at(L.crs[1], J, cj[0], cj[1], wj);
            interp_at(L.crs[2], K, ck[0], ck[1], wk);
            const float Wj[2] = {1.0f - wj, wj}, Wk[2] = {1.0f - wk, wk};
            const int p = (cj[0] - e0[1]) * es[2] + ck[0] - e0[2], dj = (cj[1] - cj[0]) * es[2], dk = ck[1] - ck[0];
            const int st = RBGS ? 2 : 1, ep = es[1] * es[2];
            if (RBGS) i0 += (1 + i0 + J + K) & 1;
#pragma unroll 2
            for (int i = i0; i <= i1; i += st) {
                int c0, c1;
                float wi;
                interp_at(L.crs[0], i, c0, c1, wi);
                const float Wi[2] = {1.0f - wi, wi};
                float v = 0.0f;
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    const float *r = co + p + ((a ? c1 : c0) - e0[0]) * ep;
                    v += Wi[a] * Wj[0] * (Wk[0] * r[0] + Wk[1] * r[dk]);
                    v += Wi[a] * Wj[1] * (Wk[0] * r[dj] + Wk[1] * r[dj + dk]);
                }
                u[place(i)] += v;
            }
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int h = MODE == DOWN ? 1 : 0; h < HS; h++) {
        const int e = HS - 1 - h + (MODE == DOWN);  // outside the tile, still valid
        const int x = MODE == DOWN;
        const int low[3] = {e + x * L.crs[0], e + x * L.crs[1], e + x * L.crs[2]};
        if (part(low, e, i0, i1)) {
            if (RBGS) {
                i0 += (h + i0 + J + K) & 1;
                column<false>(L, u, f, u, place(i0), (i1 - i0 + 2) >> 1, sx, sy,
                              [&](float nb, float ff, float) { return (nb - ff) * L.idiag; });
            } else {
                column<true>(L, h & 1 ? t : u, f, h & 1 ? u : t, place(i0), i1 - i0 + 1, sx, sy,
                             [&](float nb, float ff, float x) { return x + OMEGA * ((nb - ff) * L.idiag - x); });
            }
        }
        __syncthreads();
    }
    // u out, a point a thread, the solution's loads PIPE at a time
    const int lg = 31 - __clz(G.T), points = G.T << (2 * lg);
    for (int q0 = threadIdx.x; q0 < points; q0 += PIPE * blockDim.x) {
        int64_t g[PIPE];
        float v[PIPE];
        double x[PIPE];
#pragma unroll
        for (int q = 0; q < PIPE; q++) {
            const int p = q0 + q * (int)blockDim.x;
            const int i = first[0] + (p >> (2 * lg)), j = first[1] + ((p >> lg) & (G.T - 1)), k = first[2] + (p & (G.T - 1));
            const bool in = p < points && i >= L.lo[0] && i <= L.hi[0] && j >= L.lo[1] && j <= L.hi[1] && k >= L.lo[2] &&
                            k <= L.hi[2];
            g[q] = in ? lidx(L, i, j, k) : -1;
            v[q] = in ? u[(i - b0[0]) * sx + (j - b0[1]) * sy + k - b0[2]] : 0.0f;
            if (MODE != DOWN) x[q] = in && G.sol ? G.sol[g[q]] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < PIPE; q++) {
            if (g[q] < 0) continue;
            if (MODE != DOWN && G.sol) G.sol[g[q]] = x[q] + f64_of_f32(v[q]);
            else G.dst[g[q]] = v[q];
        }
    }
    if (MODE != DOWN) return;
    // the residual takes f's place: a point's f is read by that point alone
    if (part(L.crs, 0, i0, i1))
        column<true>(L, u, f, f, place(i0), i1 - i0 + 1, sx, sy,
                     [&](float nb, float ff, float x) { return ff - (nb - L.diag * x); });
    __syncthreads();
    int lo[3], m[3];  // the coarse points at the tile's own
#pragma unroll
    for (int d = 0; d < 3; d++) {
        lo[d] = max(L.crs[d] ? (first[d] + 1) / 2 : first[d], C.lo[d]);
        m[d] = min(L.crs[d] ? (last[d] + 1) / 2 : last[d], C.hi[d]) - lo[d] + 1;
    }
    if (m[0] <= 0 || m[1] <= 0 || m[2] <= 0) return;
    const int up[3] = {sx, sy, 1}, dn[3] = {-sx, -sy, -1};
    for (int q = threadIdx.x; q < m[0] * m[1] * m[2]; q += blockDim.x) {
        const int a = q / m[2];
        const int k = lo[2] + q - a * m[2], i = lo[0] + a / m[1], j = lo[1] + a % m[1];
        const float *r = f + ((L.crs[0] ? 2 * i - 1 : i) - b0[0]) * sx + ((L.crs[1] ? 2 * j - 1 : j) - b0[1]) * sy +
                         (L.crs[2] ? 2 * k - 1 : k) - b0[2];
        const int64_t o = lidx(C, i, j, k);
        const float v = restrict_sum(L.crs, r, dn, up);
        C.f[o] = v;
        start_level(C, G.start, o, (i + j + k) & 1, v);
    }
}

// ---- the one-block tail: levels lv[0..nl-1] of at most TAIL_MAX unknowns,
// lv[0]'s right side already restricted and its u zero
//
// All of them stay in the block's shared memory. A table of the levels' points
// (in L1 after the first stage) gives each its position and the sides it wraps
// at, red points before black, so that a half-sweep has every thread on a
// point of its colour and no index divisions. Levels of at most TAIL_WARP
// unknowns, with their dozens of stages, are cycled by one warp, whose
// barriers cost a tenth of the block's. What is left is the chain of stages,
// each a few shared loads deep: a cycle from 16x8x8 down takes 18 us (33 us
// with 1024 threads on every stage, index divisions and skipped taps).

struct TLv {
    int P[3], per[3], crs[3];
    int sx, sy;
    float c[3], diag, idiag;
    int rb;
    float *u, *f, *r, *t;
};

struct TailLevel {
    TLv L;                // without its arrays
    int ou, of, orr, ot;  // their places in shared memory; ot < 0: none
    int lo[3], m[3];      // unknown ranges: first index and count
    int n, n0;            // unknowns; those of colour 0, listed first
    int pts;              // first table entry
};

struct Tail {
    int nl;
    int sweeps;  // on the coarsest
    int smem;    // floats of shared memory the levels take
    Lv top;      // the first level's global arrays: f in, u out
    double *sol; // the FP64 solution when that is level 0: it takes the correction; else null
    const uint4 *pts;  // x: o | wrap flags << 16 (bit 2 d: low side of dimension d, 2 d + 1: high side); y, z, w: i, j, k
    TailLevel lv[TAIL_LEVELS];
};

// level l of the tail with its arrays in shared memory
__device__ __forceinline__ TLv tail_level(const Tail &T, int l, float *sm) {
    TLv L = T.lv[l].L;
    L.u = sm + T.lv[l].ou;
    L.f = sm + T.lv[l].of;
    L.r = sm + T.lv[l].orr;
    L.t = T.lv[l].ot >= 0 ? sm + T.lv[l].ot : nullptr;
    return L;
}

// A table point: its position and its six neighbours'.
struct TailPt {
    int o, nb[6];
};

__device__ __forceinline__ TailPt tail_pt(const TLv &L, uint32_t e) {
    const int st[3] = {L.sx, L.sy, 1};
    TailPt p;
    p.o = (int)(e & 0xffffu);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        p.nb[2 * d] = p.o - st[d] + ((e >> (16 + 2 * d)) & 1u ? L.P[d] * st[d] : 0);
        p.nb[2 * d + 1] = p.o + st[d] - ((e >> (17 + 2 * d)) & 1u ? L.P[d] * st[d] : 0);
    }
    return p;
}

// as nb_sum
__device__ __forceinline__ float tail_nb_sum(const TLv &L, const float *u, const TailPt &p) {
    return L.c[0] * (u[p.nb[0]] + u[p.nb[1]]) + L.c[1] * (u[p.nb[2]] + u[p.nb[3]]) +
           L.c[2] * (u[p.nb[4]] + u[p.nb[5]]);
}

__device__ __forceinline__ void tail_relax(const TLv &L, const TailPt &p, int half) {
    if (L.rb) {
        L.u[p.o] = (tail_nb_sum(L, L.u, p) - L.f[p.o]) * L.idiag;
    } else {
        const float *src = half ? L.t : L.u;
        float *dst = half ? L.u : L.t;
        const float x = src[p.o];
        dst[p.o] = x + OMEGA * ((tail_nb_sum(L, src, p) - L.f[p.o]) * L.idiag - x);
    }
}

// The threads a stage runs on: the block, or one warp of it.
template <bool WARP>
struct Team {
    __device__ __forceinline__ static int rank() { return WARP ? (int)(threadIdx.x & 31) : (int)threadIdx.x; }
    __device__ __forceinline__ static int size() { return WARP ? 32 : (int)blockDim.x; }
    __device__ __forceinline__ static void sync() {
        if (WARP) __syncwarp();
        else __syncthreads();
    }
};

// Every loop below has a trip count fixed by the level; every thread of the
// team reaches every barrier.
template <bool WARP>
__device__ void tail_smooth(const Tail &T, int l, float *sm, int sweeps) {
    using G = Team<WARP>;
    const TLv L = tail_level(T, l, sm);
    const uint4 *pts = T.pts + T.lv[l].pts;
    const int n = T.lv[l].n, n0 = L.rb ? T.lv[l].n0 : n;
    if (max(n0, n - n0) <= G::size()) {  // one point of a colour a thread: found once
        TailPt p[2] = {};
        const int t = G::rank();
        const bool in[2] = {t < n0, L.rb ? n0 + t < n : t < n};
        if (in[0]) p[0] = tail_pt(L, __ldg(&pts[t].x));
        if (in[1]) p[1] = L.rb ? tail_pt(L, __ldg(&pts[n0 + t].x)) : p[0];
        for (int s = 0; s < sweeps; s++) {
            if (in[0]) tail_relax(L, p[0], 0);
            G::sync();
            if (in[1]) tail_relax(L, p[1], 1);
            G::sync();
        }
        return;
    }
    for (int s = 0; s < sweeps; s++)
        for (int half = 0; half < 2; half++) {
            const int from = L.rb && half ? n0 : 0, to = L.rb && !half ? n0 : n;
            for (int t = from + G::rank(); t < to; t += G::size()) tail_relax(L, tail_pt(L, __ldg(&pts[t].x)), half);
            G::sync();
        }
}

// pre-smoothing, residual and restriction of level l
template <bool WARP>
__device__ void tail_down(const Tail &T, int l, float *sm) {
    using G = Team<WARP>;
    tail_smooth<WARP>(T, l, sm, NU);
    const TLv L = tail_level(T, l, sm), C = tail_level(T, l + 1, sm);
    const uint4 *pts = T.pts + T.lv[l].pts;
    for (int t = G::rank(); t < T.lv[l].n; t += G::size()) {
        const TailPt q = tail_pt(L, __ldg(&pts[t].x));
        L.r[q.o] = L.f[q.o] - (tail_nb_sum(L, L.u, q) - L.diag * L.u[q.o]);
    }
    G::sync();
    for (int t = G::rank(); t < T.lv[l + 1].n; t += G::size()) {
        const uint4 q = __ldg(T.pts + T.lv[l + 1].pts + t);
        C.f[q.x & 0xffffu] = restrict_value(L, L.r, q.y, q.z, q.w);
        C.u[q.x & 0xffffu] = 0.0f;
    }
    G::sync();
}

// prolongation into level l and post-smoothing
template <bool WARP>
__device__ void tail_up(const Tail &T, int l, float *sm) {
    using G = Team<WARP>;
    const TLv L = tail_level(T, l, sm), C = tail_level(T, l + 1, sm);
    for (int t = G::rank(); t < T.lv[l].n; t += G::size()) {
        const uint4 q = __ldg(T.pts + T.lv[l].pts + t);
        L.u[q.x & 0xffffu] += prolong_value(C, L, q.y, q.z, q.w);
    }
    G::sync();
    tail_smooth<WARP>(T, l, sm, NU);
}

__global__ void __launch_bounds__(TAIL_THREADS) k_mg_tail(const __grid_constant__ Tail T) {
    after_previous();
    extern __shared__ float sm[];
    for (int t = threadIdx.x; t < T.smem; t += blockDim.x) sm[t] = 0.0f;
    __syncthreads();
    const TailLevel &V = T.lv[0];
    for (int t = threadIdx.x; t < V.n; t += blockDim.x) {
        const int o = __ldg(&T.pts[V.pts + t].x) & 0xffffu;
        sm[V.of + o] = T.top.f[o];
    }
    __syncthreads();
    int l = 0;
    while (l + 1 < T.nl && T.lv[l].n > TAIL_WARP) tail_down<false>(T, l++, sm);
    const int top = l;  // the first level of the warp's part
    if (T.lv[top].n > TAIL_WARP) {
        tail_smooth<false>(T, top, sm, T.sweeps);  // a large coarsest level
    } else if (threadIdx.x < 32) {
        while (l + 1 < T.nl) tail_down<true>(T, l++, sm);
        tail_smooth<true>(T, l, sm, T.sweeps);
        while (l-- > top) tail_up<true>(T, l, sm);
    }
    __syncthreads();
    for (l = top - 1; l >= 0; l--) tail_up<false>(T, l, sm);
    for (int t = threadIdx.x; t < V.n; t += blockDim.x) {
        const int o = __ldg(&T.pts[V.pts + t].x) & 0xffffu;
        const float e = sm[V.ou + o];
        if (T.sol) T.sol[o] += f64_of_f32(e);
        else T.top.u[o] = e;
    }
}

// the FP64 problem from the grid slots: u takes the slot's values on the
// unknowns and on external boundary planes (the PoissonBC values), f = mult R
__global__ void k_mg_load(Geom g, Lv L, Fine F, const double *slot, const double *R, double mult) {
    after_previous();
    const int k = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = 1 + blockIdx.z;
    const int ek = L.per[2] ? L.P[2] : L.P[2] + 1, ej = L.per[1] ? L.P[1] : L.P[1] + 1;
    if (k > ek || j > ej) return;
    const int64_t o = lidx(L, i, j, k), s = gidx(g, i, j, k);
    F.u[o] = slot[s];
    F.f[o] = mult * R[s];
}

// the unknowns of the solution (less `shift`) into the zeroed slot
__global__ void k_mg_store(Geom g, Lv L, const double *u, double *slot, double shift) {
    after_previous();
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (k > L.hi[2] || j > L.hi[1] || i > L.hi[0]) return;
    slot[gidx(g, i, j, k)] = u[lidx(L, i, j, k)] - shift;
}

// per-block sums of a over the unknowns (fixed order within a block)
__global__ void k_mg_sum(Lv L, const double *a, double *part) {
    after_previous();
    __shared__ double sh[32];
    const int64_t m0 = L.hi[0] - L.lo[0] + 1, m1 = L.hi[1] - L.lo[1] + 1, m2 = L.hi[2] - L.lo[2] + 1;
    const int64_t n = m0 * m1 * m2;
    double v = 0.0;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        const int k = L.lo[2] + (int)(t % m2);
        const int64_t q = t / m2;
        const int j = L.lo[1] + (int)(q % m1);
        const int i = L.lo[0] + (int)(q / m1);
        v += a[lidx(L, i, j, k)];
    }
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = sh[0];
        for (int q = 1; q < (int)(blockDim.x >> 5); q++) s += sh[q];
        part[blockIdx.x] = s;
    }
}

__global__ void k_mg_shift(Lv L, double *a, double m) {
    after_previous();
    const int k = L.lo[2] + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = L.lo[1] + blockIdx.y * blockDim.y + threadIdx.y;
    const int i = L.lo[0] + blockIdx.z;
    if (k > L.hi[2] || j > L.hi[1] || i > L.hi[0]) return;
    a[lidx(L, i, j, k)] -= m;
}

dim3 pts_grid(const Lv &L, dim3 blk) {
    return dim3((L.hi[2] - L.lo[2] + 1 + blk.x - 1) / blk.x, (L.hi[1] - L.lo[1] + 1 + blk.y - 1) / blk.y,
                L.hi[0] - L.lo[0] + 1);
}

int64_t unknowns(const Lv &L) {
    return (int64_t)(L.hi[0] - L.lo[0] + 1) * (L.hi[1] - L.lo[1] + 1) * (L.hi[2] - L.lo[2] + 1);
}

void mg_release(MgState *s) {
    for (Lv &L : s->lv) {
        cudaFree(L.u);
        cudaFree(L.f);
        cudaFree(L.w);
    }
    s->lv.clear();
    cudaFree(s->fine.u);
    cudaFree(s->fine.f);
    s->fine = Fine{};
    if (s->exec) cudaGraphExecDestroy(s->exec);
    if (s->graph) cudaGraphDestroy(s->graph);
    s->exec = nullptr;
    s->graph = nullptr;
    cudaFree(s->tail_pts);
    s->tail_pts = nullptr;
    cudaFree(s->part);
    cudaFree(s->dmax);
    cudaFreeHost(s->hpart);
    cudaFreeHost(s->hmax);
    s->part = s->dmax = s->hpart = s->hmax = nullptr;
}

int alloc_zero(void **p, size_t bytes, cudaStream_t st) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(*p, 0, bytes, st);
    return e == cudaSuccess ? EMOO_OK : cuda_status(e);
}

// The tile of a level, 0 where a kernel a stage is better. A leg takes 7 to 8 us
// with tiles of 4 points a side and 8 to 10 with 8, on 152 SMs for one wave of
// blocks; the five or six kernels it replaces take 2.2 us each while the level
// is small, 3 at half a million points. So: the smallest tile that gives one
// wave. With 16 points a side a leg takes 15 to 19 us, and a second wave costs
// as much again: both lose to the kernels. So does SWEEP, four stages, on a
// Jacobi level in tiles of 8 (9 us).
int tile_size(const Lv &L, bool coarsest) {
    for (int T = 4; T <= TILE_MAX; T *= 2) {
        int64_t tiles = 1;
        for (int d = 0; d < 3; d++) tiles *= (L.P[d] + T - 1) / T;
        if (tiles <= 152) return T == 8 && coarsest && !L.rb ? 0 : T;
    }
    return 0;
}

size_t tile_smem(const Lv &L, int T, int mode) {
    int e[3], c[3];
    for (int d = 0; d < 3; d++) {
        e[d] = std::min(T, L.P[d]) + 2 * HS + (mode == DOWN ? L.crs[d] : 0);
        c[d] = L.crs[d] ? e[d] / 2 + 1 : e[d];
    }
    return sizeof(float) *
           ((L.rb ? 2 : 3) * e[0] * tile_sx(e[1], e[2]) + (mode == UP ? c[0] * c[1] * c[2] : 0));
}

constexpr int TILE_SMEM_MAX = 70 * 1024;  // of the largest, a Jacobi level's UP: 16^3 points in three arrays, 9 x 16 x 16 coarse
static_assert((TILE_MAX + 2 * HS + 1) * (TILE_MAX + 2 * HS + 1) <= TILE_THREADS, "a column each");

using TileKernel = void (*)(const Lv, const Lv, const TileLeg);

TileKernel tile_kernel(const Lv &L, int mode) {
    if (L.rb) return mode == DOWN ? k_mg_tile<true, DOWN> : mode == UP ? k_mg_tile<true, UP> : k_mg_tile<true, SWEEP>;
    return mode == DOWN ? k_mg_tile<false, DOWN> : mode == UP ? k_mg_tile<false, UP> : k_mg_tile<false, SWEEP>;
}

void tile_leg(emoo_handle *h, int mode, const Lv &L, const Lv &C, TileLeg G, int &launches) {
    G.T = tile_size(L, mode == SWEEP);
    const dim3 grd((L.P[2] + G.T - 1) / G.T, (L.P[1] + G.T - 1) / G.T, (L.P[0] + G.T - 1) / G.T);
    launches++;
    launch_after(tile_kernel(L, mode), grd, G.T == 8 ? TILE_THREADS : TILE_THREADS / 2, tile_smem(L, G.T, mode), h->stream)(L, C, G);
}

int coarse_sweeps(const Lv &L) {
    int m = 1;
    for (int d = 0; d < 3; d++) m = std::max(m, L.hi[d] - L.lo[d] + 1);
    return std::min(500, 2 * m * m + 8);
}

constexpr int TAIL_SMEM_MAX = 200 * 1024;

// The tail from level l: its shared-memory layout, or nl = 0 when it does not
// fit; with `pts` also its table of points, colour 0 before colour 1.
Tail make_tail(const MgState *s, size_t l, std::vector<uint4> *pts = nullptr) {
    Tail T = {};
    if (s->lv.size() - l > (size_t)TAIL_LEVELS) return T;
    int off = 0, entries = 0;
    for (size_t q = l; q < s->lv.size(); q++) {
        const Lv &L = s->lv[q];
        const int64_t n = (int64_t)(L.P[0] + 2) * L.sx;
        if (n > 65535) return T;  // positions are 16 bits in the table
        TailLevel &V = T.lv[q - l];
        for (int d = 0; d < 3; d++) {
            V.L.P[d] = L.P[d];
            V.L.per[d] = L.per[d];
            V.L.crs[d] = L.crs[d];
            V.L.c[d] = L.c[d];
            V.lo[d] = L.lo[d];
            V.m[d] = L.hi[d] - L.lo[d] + 1;
        }
        V.L.sx = (int)L.sx;
        V.L.sy = (int)L.sy;
        V.L.diag = L.diag;
        V.L.idiag = L.idiag;
        V.L.rb = L.rb;
        V.ou = off;
        V.of = off + (int)n;
        V.orr = off + 2 * (int)n;
        V.ot = L.rb ? -1 : off + 3 * (int)n;
        off += (L.rb ? 3 : 4) * (int)n;
        V.n = V.m[0] * V.m[1] * V.m[2];
        V.pts = entries;
        entries += V.n;
        for (int colour = 0; colour < 2; colour++) {
            int count = 0;
            for (int i = L.lo[0]; i <= L.hi[0]; i++)
                for (int j = L.lo[1]; j <= L.hi[1]; j++)
                    for (int k = L.lo[2]; k <= L.hi[2]; k++) {
                        if (((i + j + k) & 1) != colour) continue;
                        count++;
                        if (!pts) continue;
                        const int c[3] = {i, j, k};
                        uint32_t e = (uint32_t)(i * (int)L.sx + j * (int)L.sy + k);
                        for (int d = 0; d < 3; d++) {
                            if (L.per[d] && c[d] == 1) e |= 1u << (16 + 2 * d);
                            if (L.per[d] && c[d] == L.P[d]) e |= 1u << (17 + 2 * d);
                        }
                        pts->push_back(make_uint4(e, i, j, k));
                    }
            if (colour == 0) V.n0 = count;
        }
    }
    if ((size_t)off * sizeof(float) > (size_t)TAIL_SMEM_MAX) return T;
    T.nl = (int)(s->lv.size() - l);
    T.smem = off;
    T.sweeps = coarse_sweeps(s->lv.back());
    T.top = s->lv[l];
    T.pts = s->tail_pts;
    T.sol = l == 0 ? s->fine.u : nullptr;
    return T;
}

// `sweeps` sweeps of a level a kernel a half-sweep, without the first `skip`
// half-sweeps (done where the right side was formed) and, with `sol`, the last
// adding the correction to it.
void smooth(emoo_handle *h, const Lv &L, int sweeps, int skip, const Fine *sol, int &launches) {
    dim3 blk(32, 8);
    const int m2 = L.hi[2] - L.lo[2] + 1;
    const dim3 half(((m2 + 1) / 2 + blk.x - 1) / blk.x, (L.hi[1] - L.lo[1] + 1 + blk.y - 1) / blk.y, L.hi[0] - L.lo[0] + 1);
    for (int s = skip; s < 2 * sweeps; s++) {
        launches++;
        if (sol && s + 1 == 2 * sweeps) launch_after(k_mg_finish, pts_grid(L, blk), blk, 0, h->stream)(L, *sol);
        else if (L.rb) launch_after(k_mg_smooth, half, blk, 0, h->stream)(L, s & 1);
        else launch_after(k_mg_jacobi, pts_grid(L, blk), blk, 0, h->stream)(L, s & 1 ? L.w : L.u, s & 1 ? L.u : L.w);
    }
}

// How level l starts from a new right side.
int level_start(const MgState *s, size_t l) {
    if (l == s->tail_from) return START_NONE;
    const bool coarsest = l + 1 == s->lv.size();
    if (tile_size(s->lv[l], coarsest)) return coarsest ? START_ZERO : START_NONE;
    return START_SWEPT;
}

// One V-cycle from level l; returns where the level's correction is (level 0's
// goes into the solution).
const float *vcycle(emoo_handle *h, MgState *s, size_t l, int &launches) {
    const Lv &L = s->lv[l];
    double *sol = l == 0 ? s->fine.u : nullptr;
    if (l == s->tail_from) {
        const Tail T = make_tail(s, l);
        launches++;
        launch_after(k_mg_tail, 1, TAIL_THREADS, T.smem * sizeof(float), h->stream)(T);
        return L.u;
    }
    dim3 blk(32, 8);
    const bool coarsest = l + 1 == s->lv.size(), tiles = tile_size(L, coarsest) > 0;
    if (tiles && coarsest) {  // too large for the tail
        float *a = L.u, *b = L.w;
        for (int q = coarse_sweeps(L) / NU; q > 0; q--) {  // an even number of sweeps
            tile_leg(h, SWEEP, L, L, {0, a, b, q == 1 ? sol : nullptr, 0}, launches);
            std::swap(a, b);
        }
        return a;
    }
    if (tiles) {
        Lv C = s->lv[l + 1];
        tile_leg(h, DOWN, L, C, {0, nullptr, L.u, nullptr, level_start(s, l + 1)}, launches);
        C.u = const_cast<float *>(vcycle(h, s, l + 1, launches));
        tile_leg(h, UP, L, C, {0, L.u, L.w, sol, 0}, launches);
        return L.w;
    }
    const Fine *fine = l == 0 ? &s->fine : nullptr;
    if (coarsest) {
        smooth(h, L, coarse_sweeps(L), 1, fine, launches);
        return L.u;
    }
    Lv C = s->lv[l + 1];
    smooth(h, L, NU, 1, nullptr, launches);
    launches += 2;
    launch_after(k_mg_residual, pts_grid(L, blk), blk, 0, h->stream)(L);
    launch_after(k_mg_restrict, pts_grid(C, blk), blk, 0, h->stream)(L, C, level_start(s, l + 1));
    C.u = const_cast<float *>(vcycle(h, s, l + 1, launches));
    launches++;
    launch_after(k_mg_prolong, pts_grid(L, blk), blk, 0, h->stream)(C, L);
    smooth(h, L, NU, 0, fine, launches);
    return L.u;
}

// the FP64 residual, its maximum into the pinned host word
void residual64(emoo_handle *h, MgState *s, int &launches) {
    dim3 blk(32, 8);
    const Lv &L0 = s->lv[0];
    cudaMemsetAsync(s->dmax, 0, sizeof(double), h->stream);
    launches++;
    launch_after(k_mg_residual64, pts_grid(L0, blk), blk, 0, h->stream)(L0, s->fine, s->dmax, level_start(s, 0));
    cudaMemcpyAsync(s->hmax, s->dmax, sizeof(double), cudaMemcpyDeviceToHost, h->stream);
}

// one outer step: V-cycle, u += its correction, new residual
void outer_step(emoo_handle *h, MgState *s, int &launches) {
    vcycle(h, s, 0, launches);
    residual64(h, s, launches);
}

int mg_setup(emoo_handle *h, MgState *s) {
    const Geom &g = h->g;
    bool same = !s->lv.empty();
    for (int d = 0; d < 3 && same; d++)
        same = s->n[d] == g.n[d] && s->per[d] == (h->bc.fbc[2 * d] == FBC_PERIODIC) && s->d[d] == g.d[d];
    if (same) return EMOO_OK;
    mg_release(s);
    for (int d = 0; d < 3; d++) {
        s->n[d] = g.n[d];
        s->per[d] = h->bc.fbc[2 * d] == FBC_PERIODIC;
        s->d[d] = g.d[d];
    }
    int P[3] = {g.n[0], g.n[1], g.n[2]};
    double hh[3] = {g.d[0], g.d[1], g.d[2]};
    for (;;) {
        Lv L = {};
        for (int d = 0; d < 3; d++) {
            L.P[d] = P[d];
            L.per[d] = s->per[d];
            L.lo[d] = L.per[d] ? 1 : 2;
            L.hi[d] = P[d];
            L.c[d] = (float)(1.0 / (hh[d] * hh[d]));
            L.crs[d] = (P[d] % 2 == 0) && P[d] >= 4;
        }
        if (L.hi[0] < L.lo[0] || L.hi[1] < L.lo[1] || L.hi[2] < L.lo[2] || L.hi[0] - L.lo[0] + 1 > 65535) {
            mg_release(s);  // no unknowns (checked by the caller first), or too many planes for one grid launch
            return EMOO_ERR_UNSUPPORTED;
        }
        const double diag = 2.0 * (1.0 / (hh[0] * hh[0]) + 1.0 / (hh[1] * hh[1]) + 1.0 / (hh[2] * hh[2]));
        L.diag = (float)diag;
        L.idiag = (float)(1.0 / diag);
        L.rb = 1;
        for (int d = 0; d < 3; d++)
            if (L.per[d] && (P[d] & 1)) L.rb = 0;
        L.sy = P[2] + 2;
        L.sx = (int64_t)(P[1] + 2) * (P[2] + 2);
        const size_t bytes = (size_t)(P[0] + 2) * L.sx * sizeof(float);
        int rc = alloc_zero((void **)&L.u, bytes, h->stream);
        if (rc == EMOO_OK) rc = alloc_zero((void **)&L.f, bytes, h->stream);
        if (rc == EMOO_OK) rc = alloc_zero((void **)&L.w, bytes, h->stream);
        const bool more = L.crs[0] || L.crs[1] || L.crs[2];
        s->lv.push_back(L);
        if (rc != EMOO_OK) {
            mg_release(s);
            return rc;
        }
        if (!more) break;
        for (int d = 0; d < 3; d++)
            if (L.crs[d]) {
                P[d] /= 2;
                hh[d] *= 2.0;
            }
    }
    for (const Lv &L : s->lv)
        for (int mode : {DOWN, UP, SWEEP}) {
            const cudaError_t e = cudaFuncSetAttribute(tile_kernel(L, mode), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       TILE_SMEM_MAX);
            if (e != cudaSuccess) {
                mg_release(s);
                return cuda_status(e);
            }
        }
    // the shared-memory tail: the first level of at most TAIL_MAX unknowns
    // from which the rest fits
    s->tail_from = s->lv.size();
    for (size_t q = 0; q < s->lv.size(); q++)
        if (unknowns(s->lv[q]) <= TAIL_MAX && make_tail(s, q).nl > 0) {
            s->tail_from = q;
            std::vector<uint4> pts;
            make_tail(s, q, &pts);
            // the limit is the function's, for every handle: always the largest tail's
            cudaError_t e =
                cudaFuncSetAttribute(k_mg_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_SMEM_MAX);
            if (e == cudaSuccess) e = cudaMalloc(&s->tail_pts, pts.size() * sizeof(uint4));
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(s->tail_pts, pts.data(), pts.size() * sizeof(uint4), cudaMemcpyHostToDevice,
                                    h->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);  // pts goes out of scope
            if (e != cudaSuccess) {
                mg_release(s);
                return cuda_status(e);
            }
            break;
        }
    const Lv &L0 = s->lv[0];
    const size_t b64 = (size_t)(L0.P[0] + 2) * L0.sx * sizeof(double);
    for (int d = 0; d < 3; d++) s->fine.c[d] = 1.0 / (g.d[d] * g.d[d]);
    s->fine.diag = 2.0 * (s->fine.c[0] + s->fine.c[1] + s->fine.c[2]);
    int rc = alloc_zero((void **)&s->fine.u, b64, h->stream);
    if (rc == EMOO_OK) rc = alloc_zero((void **)&s->fine.f, b64, h->stream);
    if (rc == EMOO_OK) rc = alloc_zero((void **)&s->part, RB * sizeof(double), h->stream);
    if (rc == EMOO_OK) rc = alloc_zero((void **)&s->dmax, sizeof(double), h->stream);
    if (rc == EMOO_OK && cudaMallocHost(&s->hpart, RB * sizeof(double)) != cudaSuccess) rc = EMOO_ERR_OOM;
    if (rc == EMOO_OK && cudaMallocHost(&s->hmax, sizeof(double)) != cudaSuccess) rc = EMOO_ERR_OOM;
    if (rc == EMOO_OK) {  // one outer step as a graph
        int launches = 0;
        cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            outer_step(h, s, launches);
            e = cudaStreamEndCapture(h->stream, &s->graph);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&s->exec, s->graph, 0);
        if (e != cudaSuccess) rc = cuda_status(e);
        s->graph_launches = launches;
    }
    if (rc != EMOO_OK) mg_release(s);
    return rc;
}

int sum_unknowns(emoo_handle *h, MgState *s, const double *a, double *out) {
    h->launches++;
    launch_after(k_mg_sum, RB, 256, 0, h->stream)(s->lv[0], a, s->part);
    EMOO_CUDA(cudaGetLastError());
    EMOO_CUDA(cudaMemcpyAsync(s->hpart, s->part, RB * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    EMOO_CUDA(cudaStreamSynchronize(h->stream));
    double v = 0.0;
    for (int b = 0; b < RB; b++) v += s->hpart[b];
    *out = v;
    return EMOO_OK;
}

}  // namespace

void multigrid_free(emoo_handle *h) {
    if (!h->mg) return;
    MgState *s = (MgState *)h->mg;
    mg_release(s);
    delete s;
    h->mg = nullptr;
}

// The solve of one field: u in slot id1 (ghost planes by the reference's
// boundary fill, a copy in id2), f = mult R from slot rid. *cycles receives
// the outer steps (V-cycles) run, *converged whether max |r| <= rtol max |r0|
// was met within the cap.
int multigrid_f64(emoo_handle *h, int id1, int id2, int rid, double mult, int *cycles, int *converged) {
    bool none = false;  // an external dimension of one cell has no unknowns: the boundary planes are the solution
    for (int d = 0; d < 3; d++) none = none || (h->bc.fbc[2 * d] != FBC_PERIODIC && h->g.n[d] < 2);
    if (none) {
        EMOO_CUDA(cudaMemsetAsync(h->slot[id1], 0, (size_t)h->g.npts * sizeof(double), h->stream));
        EMOO_TRY(poisson_field_bc(h, id1));
        EMOO_CUDA(cudaMemcpyAsync(h->slot[id2], h->slot[id1], (size_t)h->g.npts * sizeof(double),
                                  cudaMemcpyDeviceToDevice, h->stream));
        if (cycles) *cycles = 0;
        if (converged) *converged = 1;
        return EMOO_OK;
    }
    if (!h->mg) h->mg = new MgState();
    MgState *s = (MgState *)h->mg;
    EMOO_TRY(mg_setup(h, s));
    const Geom &g = h->g;
    const Lv &L0 = s->lv[0];
    dim3 blk(32, 8);
    // the slot zeroed, then its boundary planes from the reference's fill
    EMOO_CUDA(cudaMemsetAsync(h->slot[id1], 0, (size_t)g.npts * sizeof(double), h->stream));
    EMOO_TRY(poisson_field_bc(h, id1));
    {
        const int ek = L0.per[2] ? L0.P[2] : L0.P[2] + 1, ej = L0.per[1] ? L0.P[1] : L0.P[1] + 1;
        const int ei = L0.per[0] ? L0.P[0] : L0.P[0] + 1;
        dim3 grd((ek + blk.x - 1) / blk.x, (ej + blk.y - 1) / blk.y, ei);
        h->launches++;
        launch_after(k_mg_load, grd, blk, 0, h->stream)(g, L0, s->fine, h->slot[id1], h->slot[rid], mult);
    }
    const bool allper = L0.per[0] && L0.per[1] && L0.per[2];
    const double nunk = (double)unknowns(L0);
    if (allper) {  // the singular periodic system is consistent only for a mean-free right side
        double sum;
        EMOO_TRY(sum_unknowns(h, s, s->fine.f, &sum));
        h->launches++;
        launch_after(k_mg_shift, pts_grid(L0, blk), blk, 0, h->stream)(L0, s->fine.f, sum / nunk);
    }
    int launches = 0;
    residual64(h, s, launches);
    h->launches += launches;
    EMOO_CUDA(cudaGetLastError());
    EMOO_CUDA(cudaStreamSynchronize(h->stream));
    const double r0 = *s->hmax;
    const double tol = h->poisson_rtol * r0;
    int it = 0;
    const int cap = 200;
    bool ok = r0 == 0.0;
    while (!ok && it < cap) {
        EMOO_CUDA(cudaGraphLaunch(s->exec, h->stream));
        h->launches += s->graph_launches;
        EMOO_CUDA(cudaStreamSynchronize(h->stream));
        it++;
        ok = *s->hmax <= tol;
    }
    double shift = 0.0;
    if (allper) {
        double sum;
        EMOO_TRY(sum_unknowns(h, s, s->fine.u, &sum));
        shift = sum / nunk;
    }
    h->launches++;
    launch_after(k_mg_store, pts_grid(L0, blk), blk, 0, h->stream)(g, L0, s->fine.u, h->slot[id1], shift);
    EMOO_CUDA(cudaGetLastError());
    EMOO_TRY(poisson_field_bc(h, id1));
    EMOO_CUDA(cudaMemcpyAsync(h->slot[id2], h->slot[id1], (size_t)g.npts * sizeof(double), cudaMemcpyDeviceToDevice,
                              h->stream));
    if (cycles) *cycles = it;
    if (converged) *converged = ok ? 1 : 0;
    return EMOO_OK;
}

}  // namespace emoo
