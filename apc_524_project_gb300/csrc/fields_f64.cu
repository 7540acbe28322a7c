// fields_f64.cu - FP64 grid kernels: Yee E/B update, ghost fill, periodic
// J/rho fold, LightBC / Dirichlet plane sets, Jacobi Poisson sweeps, phiToE,
// AToB, field-energy and Gauss-law reductions.
//
// Compiled with --fmad=false: every expression keeps the reference's order of
// operations with separately rounded multiplies and adds, so on identical
// inputs the results are bit-identical to the reference serial build.
// All kernels are HBM-bound stencils over the (n+3)^3 reference layout with
// k (the contiguous axis) mapped to threadIdx.x for coalescing.
#include <cuda_runtime.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "dev_common.cuh"
#include "emoo_internal.h"

namespace emoo {

namespace {

constexpr double FOURPI = 4.0 * PI_D;

struct F3 {
    double *p[3];
};
struct CF3 {
    const double *p[3];
};

dim3 phys_grid(const Geom &g, dim3 blk) {
    return dim3((g.n[2] + blk.x - 1) / blk.x, (g.n[1] + blk.y - 1) / blk.y, g.n[0]);
}

// Grid::evolveFields, E half (src/grid/oGrid.cpp:23-40): E -= dt (curl-ish of
// B_tm1 + 4 pi J) over physical points, B_tm1 being the freshly swapped role.
// FOLD: first the reference policy's periodic folds of J (k_fold, dimension by
// dimension): plane 1 adds plane n + 1's two transverse components over the
// physical transverse range. Those sources are no fold's target, so each point
// forms its own sums in the folds' order.
struct FoldDims {
    int per[3];
};

template <bool FOLD>
__global__ void k_yee_e(Geom g, double dt, F3 E, CF3 T, F3 J, FoldDims f) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    const double *Tx = T.p[0], *Ty = T.p[1], *Tz = T.p[2];
    double dx = g.d[0], dy = g.d[1], dz = g.d[2];
    double jx = J.p[0][o], jy = J.p[1][o], jz = J.p[2][o];
    bool folded = false;
    if (FOLD) {
        const int64_t s0 = o + (int64_t)g.n[0] * g.sx, s1 = o + (int64_t)g.n[1] * g.sy, s2 = o + g.n[2];
        const bool f0 = f.per[0] && i == 1, f1 = f.per[1] && j == 1, f2 = f.per[2] && k == 1;
        if (f0) jy += J.p[1][s0], jz += J.p[2][s0];
        if (f1) jx += J.p[0][s1], jz += J.p[2][s1];
        if (f2) jx += J.p[0][s2], jy += J.p[1][s2];
        folded = f0 || f1 || f2;
    }
    double ex = E.p[0][o] - dt * (ddiv(Ty[o] - Ty[o - 1], dz, g.id[2], g.p2[2]) -
                                  ddiv(Tz[o] - Tz[o - g.sy], dy, g.id[1], g.p2[1]) + FOURPI * jx);
    double ey = E.p[1][o] - dt * (ddiv(Tz[o] - Tz[o - g.sx], dx, g.id[0], g.p2[0]) -
                                  ddiv(Tx[o] - Tx[o - 1], dz, g.id[2], g.p2[2]) + FOURPI * jy);
    double ez = E.p[2][o] - dt * (ddiv(Tx[o] - Tx[o - g.sy], dy, g.id[1], g.p2[1]) -
                                  ddiv(Ty[o] - Ty[o - g.sx], dx, g.id[0], g.p2[0]) + FOURPI * jz);
    E.p[0][o] = ex;
    E.p[1][o] = ey;
    E.p[2][o] = ez;
    if (FOLD && folded) {
        J.p[0][o] = jx;
        J.p[1][o] = jy;
        J.p[2][o] = jz;
    }
}

// Grid::evolveFields, B half (src/grid/oGrid.cpp:43-57): B = B_tm1 + dt curl E.
// Reads the E ghost planes as they are (refreshed only after the update).
__global__ void k_yee_b(Geom g, double dt, F3 B, CF3 T, CF3 E) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    const double *Ex = E.p[0], *Ey = E.p[1], *Ez = E.p[2];
    double dx = g.d[0], dy = g.d[1], dz = g.d[2];
    const double bx = T.p[0][o] + dt * (ddiv(Ey[o + 1] - Ey[o], dz, g.id[2], g.p2[2]) -
                                  ddiv(Ez[o + g.sy] - Ez[o], dy, g.id[1], g.p2[1]));
    const double by = T.p[1][o] + dt * (ddiv(Ez[o + g.sx] - Ez[o], dx, g.id[0], g.p2[0]) -
                                  ddiv(Ex[o + 1] - Ex[o], dz, g.id[2], g.p2[2]));
    const double bz = T.p[2][o] + dt * (ddiv(Ex[o + g.sy] - Ex[o], dy, g.id[1], g.p2[1]) -
                                  ddiv(Ey[o + g.sx] - Ey[o], dx, g.id[0], g.p2[0]));
    B.p[0][o] = bx;  // stores last: the loads may not pass them
    B.p[1][o] = by;
    B.p[2][o] = bz;
}

// Grid::evolveFieldsES, src/grid/oGrid.cpp:67-81
__global__ void k_yee_es(Geom g, double dt, F3 E, CF3 J) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    double mdt = -dt;
    E.p[0][o] = mdt * (FOURPI * J.p[0][o]);
    E.p[1][o] = mdt * (FOURPI * J.p[1][o]);
    E.p[2][o] = mdt * (FOURPI * J.p[2][o]);
}

struct FieldList {
    double *p[6];
    int n;
};

// Periodic ghost fill (BC_F_Periodic::completeBC for sendID -1 or one field,
// src/boundaries/b_fields/bc_f_periodic.cpp:47-52 via
// src/grid/spookyGrid.cpp:17-184): ghost plane 0 <- plane n, ghost plane
// n+1 <- plane 1, over the physical transverse range only. All copies read
// physical points and write ghost points, so any set of dims runs at once.
// blockIdx.z = (field * 3 + dim) * 2 + side.
__global__ void k_ghost(Geom g, FieldList fl, int dims_mask, const int *skip) {
    after_previous();
    if (skip && *skip) return;
    int z = blockIdx.z;
    int r = z & 1;
    int d = (z >> 1) % 3;
    int f = (z >> 1) / 3;
    if (!((dims_mask >> d) & 1) || f >= fl.n) return;
    int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    int q = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int p = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (q > g.n[o2] || p > g.n[o1]) return;
    int nd = g.n[d];
    int src = r == 0 ? nd : 1, dst = r == 0 ? 0 : nd + 1;
    int is[3], it[3];
    is[d] = src;
    it[d] = dst;
    is[o1] = it[o1] = p;
    is[o2] = it[o2] = q;
    double *F = fl.p[f];
    F[gidx(g, it[0], it[1], it[2])] = F[gidx(g, is[0], is[1], is[2])];
}

// Periodic fold of one dimension (BC_F_Periodic::completeBC(-2) of the left
// side, src/boundaries/b_fields/bc_f_periodic.cpp:40-46): the two transverse
// J components and rho of ghost plane n+1 are added into plane 1.
__global__ void k_fold(Geom g, int d, double *f0, double *f1, double *f2) {
    after_previous();
    int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    int q = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int p = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (q > g.n[o2] || p > g.n[o1]) return;
    int is[3], it[3];
    is[d] = g.n[d] + 1;
    it[d] = 1;
    is[o1] = it[o1] = p;
    is[o2] = it[o2] = q;
    int64_t s = gidx(g, is[0], is[1], is[2]), t = gidx(g, it[0], it[1], it[2]);
    double *F = blockIdx.z == 0 ? f0 : (blockIdx.z == 1 ? f1 : f2);
    F[t] += F[s];
}

struct PlaneList {
    PlaneSet s[12];
    int n;
};

// Grid::setFieldInPlane over the whole (n+3)^2 plane, src/grid/oGrid.cpp:446-476.
__global__ void k_plane_set(Geom g, PlaneList pl, const int *skip) {
    after_previous();
    if (skip && *skip) return;
    int e = blockIdx.z;
    if (e >= pl.n) return;
    const PlaneSet &ps = pl.s[e];
    int d = ps.dim;
    int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    int p = blockIdx.y * blockDim.y + threadIdx.y;
    if (q >= g.tot[o2] || p >= g.tot[o1]) return;
    int ii[3];
    ii[d] = ps.idx;
    ii[o1] = p;
    ii[o2] = q;
    double v = ps.v;
    if (ps.t1) v = __dadd_rn(v, __dmul_rn(__dmul_rn(ps.vs, ps.t1[p]), ps.t2[q]));  // v + (vs t1) t2
    ps.f[gidx(g, ii[0], ii[1], ii[2])] = v;
}

__global__ void k_fill(double *p, int64_t n, double v) {
    after_previous();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

// ---- Jacobi ----

struct JacobiState {
    int done;
    int iter;       // iterations completed
    int converged;
    int skip;       // boundary fills no-ops (one sweep after done, with the test in the sweep)
    double maxdiff; // current iteration's max |u2 - u1|
    unsigned int blocks_done;
    int error;      // a bounded wait ran out
};

// One Jacobi sweep, src/poisson/poisson.cpp:216-241.
__global__ void k_jacobi(Geom g, const double *src, double *dst, const double *R, double ax, double ay, double az,
                         double af, double mult, const JacobiState *st) {
    if (st->done) return;
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    dst[o] = ax * (src[o - g.sx] + src[o + g.sx]) + ay * (src[o - g.sy] + src[o + g.sy]) +
             az * (src[o - 1] + src[o + 1]) - af * R[o] * mult;
}

// max |u2 - u1| over physical points, then convergence bookkeeping by the
// last block (src/poisson/poisson.cpp:250-283).
__global__ void k_jacobi_check(Geom g, const double *u1, const double *u2, double tol, JacobiState *st) {
    if (st->done) return;
    __shared__ double smax[32];
    __shared__ bool last;
    double m = 0.0;
    int64_t nphys = (int64_t)g.n[0] * g.n[1] * g.n[2];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nphys; t += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        phys_ijk(g.n, t, i, j, k);
        int64_t o = gidx(g, i, j, k);
        double a = fabs(u2[o] - u1[o]);
        m = a > m ? a : m;
    }
    for (int off = 16; off > 0; off >>= 1) {
        double o = __shfl_down_sync(0xffffffffu, m, off);
        m = o > m ? o : m;
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) smax[w] = m;
    __syncthreads();
    if (w == 0) {
        m = lane < (int)(blockDim.x >> 5) ? smax[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1) {
            double o = __shfl_down_sync(0xffffffffu, m, off);
            m = o > m ? o : m;
        }
        if (lane == 0) {
            atomic_max_nonneg(&st->maxdiff, m);
            __threadfence();
            unsigned int prev = atomicAdd(&st->blocks_done, 1u);
            last = (prev == gridDim.x - 1);
        }
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        double md = *((volatile double *)&st->maxdiff);
        int it = st->iter;  // iternum of this iteration
        if (md < tol) {
            st->done = 1;
            st->converged = 1;
        } else if (it >= ITER_MAX) {
            st->done = 1;
            st->converged = 0;
        }
        st->iter = it + 1;
        st->maxdiff = 0.0;
        st->blocks_done = 0u;
    }
}

// ---- Jacobi on tiles held in shared memory ---------------------------------
//
// The whole iteration of a small grid (every side periodic) in one cooperative
// launch: the grid is cut into one tile a block, at most one block an SM, and
// a tile's two buffers (ping-pong, one ghost layer) and right side stay in
// shared memory. After each sweep a block hands its face values to its six
// neighbours and takes theirs; no block waits for any other. A value travels
// as two 64-bit words of (sequence number, 32 bits), each the element of a
// vector access and so written and read whole (a vector access is no more than
// its elements' accesses): the reader polls the value itself and no fence or
// flag is needed. This is the exchange that collective libraries use for small
// messages. Two slots a face suffice, because a block writes
// sequence q + 2 only after it has read its neighbours' q + 1, which they made
// from its q. A sweep of 32^3 takes 1.8 us, of which the FP64 pipe needs 0.6
// (10 instructions a point, 8 warps an SM) and the exchange's latency the
// rest; as two kernels a sweep it took 7.7 us. Used where a tile fits a
// block's shared memory, up to about 100^3.
//
// The stop test must stop the iteration at the same sweep as the reference.
// Blocks run JT_BATCH sweeps between grid barriers, each noting for every
// sweep whether one of its points moved by tol or more; the barrier ORs the
// notes, and if some sweep has none, every block goes back to the state at the
// start of the batch (kept in the first potential's array) and repeats it up
// to that sweep. Every wait is bounded; one that runs out sets st->error.
constexpr int JT_BATCH = 64;
constexpr int JT_THREADS = 1024;
constexpr int JT_SPIN = 1 << 22;

struct JacobiTiles {
    int b[3];           // tiles per dimension
    int t[3];           // points of the largest tile per dimension
    int face;           // points of the largest face
    ulonglong2 *faces;  // [block][side][slot][face]
    unsigned long long *moved;  // [batch] OR over the blocks
    unsigned int *arrived;      // grid barrier
};

__device__ __forceinline__ void jt_send(ulonglong2 *to, double v, unsigned int seq) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), tag = (unsigned long long)seq << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(to), "l"(tag | (b & 0xffffffffull)), "l"(tag | b >> 32)
                 : "memory");
}

// the value that carries number seq; false when the wait ran out
__device__ __forceinline__ bool jt_take(const ulonglong2 *from, unsigned int seq, double &v) {
    unsigned long long x, y;
    int spin = 0;
    do {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(from) : "memory");
    } while (((unsigned int)(x >> 32) != seq || (unsigned int)(y >> 32) != seq) && ++spin < JT_SPIN);
    v = __hiloint2double((int)(unsigned int)y, (int)(unsigned int)x);
    return spin < JT_SPIN;
}

// blocks that passed barrier number `round` (1, 2, ..); false when it ran out
__device__ __forceinline__ bool jt_barrier(unsigned int *arrived, unsigned int round) {
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        const unsigned int target = round * gridDim.x;
        __threadfence();
        atomicAdd(arrived, 1u);
        int spin = 0;
        while (*((volatile unsigned int *)arrived) < target && ++spin < JT_SPIN) __nanosleep(64);
        ok = spin < JT_SPIN;
        __threadfence();
    }
    return __syncthreads_and(threadIdx.x == 0 ? ok : 1);
}

__global__ void __launch_bounds__(JT_THREADS) k_jacobi_tiles(Geom g, double *u1, double *u2, const double *R, double ax,
                                                             double ay, double az, double af, double mult, double tol,
                                                             JacobiTiles jt, JacobiState *st) {
    extern __shared__ double jt_sm[];
    int bc[3], lo[3], sz[3], nb[6];
    {
        int r = blockIdx.x;
        bc[2] = r % jt.b[2];
        r /= jt.b[2];
        bc[1] = r % jt.b[1];
        bc[0] = r / jt.b[1];
        for (int d = 0; d < 3; d++) {
            const int q = g.n[d] / jt.b[d], m = g.n[d] % jt.b[d];  // the first m tiles have one point more
            lo[d] = bc[d] * q + min(bc[d], m) + 1;
            sz[d] = q + (bc[d] < m ? 1 : 0);
            for (int side = 0; side < 2; side++) {
                int c[3] = {bc[0], bc[1], bc[2]};
                c[d] = side ? (bc[d] + 1 == jt.b[d] ? 0 : bc[d] + 1) : (bc[d] == 0 ? jt.b[d] - 1 : bc[d] - 1);
                nb[2 * d + side] = (c[0] * jt.b[1] + c[1]) * jt.b[2] + c[2];
            }
        }
    }
    const int py = sz[2] + 2, px = (sz[1] + 2) * py;  // strides of the tile with its ghost layer
    const int vol = sz[0] * sz[1] * sz[2], whole = (sz[0] + 2) * px;
    double *cur = jt_sm, *next = cur + whole, *rhs = next + whole;
    const int area[3] = {sz[1] * sz[2], sz[0] * sz[2], sz[0] * sz[1]};
    const int halo = 2 * (area[0] + area[1] + area[2]);
    auto point = [&](int p, int &i, int &j, int &k) {  // of the tile, from 0
        k = p % sz[2];
        const int r = p / sz[2];
        j = r % sz[1];
        i = r / sz[1];
    };
    // halo value q of side `side` of dimension d: its ghost point in the tile
    auto halo_at = [&](int p, int &d, int &side, int &q) -> int {
        d = 0;
        q = p;
        while (q >= 2 * area[d]) q -= 2 * area[d++];
        side = q >= area[d];
        q -= side * area[d];
        const int o1 = d == 0 ? 1 : 0, o2 = d == 2 ? 1 : 2;
        int c[3];
        c[d] = side ? sz[d] + 1 : 0;
        c[o1] = q / sz[o2] + 1;
        c[o2] = q % sz[o2] + 1;
        return c[0] * px + c[1] * py + c[2];
    };
    // this thread's first point and first halo value, kept: most tiles have no
    // more than one a thread, and the divisions would cost each sweep 0.1 us
    int mi = 0, mj = 0, mk = 0, hd = 0, hside = 0, hq = 0, hat = 0;
    if (threadIdx.x < vol) point(threadIdx.x, mi, mj, mk);
    if (threadIdx.x < halo) hat = halo_at(threadIdx.x, hd, hside, hq);
    auto load = [&](double *dst, const double *u) {  // tile and ghost layer of a global potential
        for (int p = threadIdx.x; p < whole; p += blockDim.x) {
            int c[3] = {p / px, (p % px) / py, p % py};
            for (int d = 0; d < 3; d++) {
                c[d] += lo[d] - 1;
                c[d] = c[d] < 1 ? g.n[d] : (c[d] > g.n[d] ? 1 : c[d]);
            }
            dst[p] = __ldcg(u + gidx(g, c[0], c[1], c[2]));
        }
    };
    auto store = [&](const double *src, double *u) {
        for (int p = threadIdx.x; p < vol; p += blockDim.x) {
            int i, j, k;
            point(p, i, j, k);
            u[gidx(g, lo[0] + i, lo[1] + j, lo[2] + k)] = src[(i + 1) * px + (j + 1) * py + k + 1];
        }
    };
    auto slot = [&](int block, int side, unsigned int seq) {
        return jt.faces + ((size_t)(block * 6 + side) * 2 + (seq & 1u)) * jt.face;
    };
    for (int p = threadIdx.x; p < vol; p += blockDim.x) {
        int i, j, k;
        point(p, i, j, k);
        rhs[p] = af * R[gidx(g, lo[0] + i, lo[1] + j, lo[2] + k)] * mult;
    }
    load(cur, u1);
    __syncthreads();
    const long long ltol = __double_as_longlong(tol), linf = 0x7ff0000000000000LL;
    unsigned int seq = 0, round = 0;
    bool fresh = true, ok = true;  // fresh: cur's ghost layer is filled
    // one sweep; whether a point of the block moved by tol or more
    auto sweep = [&]() -> bool {
        if (!fresh) {
            bool got = true;
            for (int p = threadIdx.x; p < halo; p += blockDim.x) {
                int d = hd, side = hside, q = hq, at = hat;
                if (p != threadIdx.x) at = halo_at(p, d, side, q);
                // my ghost plane on this side is the neighbour's face on the other
                const ulonglong2 *src = slot(nb[2 * d + side], 2 * d + 1 - side, seq) + q;
                got = jt_take(src, seq, cur[at]) && got;
            }
            ok = __syncthreads_and(got);
            if (!ok) return true;
        }
        seq++;
        bool far = false;
        for (int p = threadIdx.x; p < vol; p += blockDim.x) {
            int c[3] = {mi, mj, mk};
            if (p != threadIdx.x) point(p, c[0], c[1], c[2]);
            const int o = (c[0] + 1) * px + (c[1] + 1) * py + c[2] + 1;
            const double v = ax * (cur[o - px] + cur[o + px]) + ay * (cur[o - py] + cur[o + py]) +
                             az * (cur[o - 1] + cur[o + 1]) - rhs[p];
            next[o] = v;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const int o1 = d == 0 ? 1 : 0, o2 = d == 2 ? 1 : 2;
#pragma unroll
                for (int side = 0; side < 2; side++) {
                    if (c[d] != (side ? sz[d] - 1 : 0)) continue;
                    jt_send(slot(blockIdx.x, 2 * d + side, seq) + c[o1] * sz[o2] + c[o2], v, seq);
                }
            }
            // |v - u| >= tol on the words (false for NaN, as the comparison is)
            const long long a = __double_as_longlong(fabs(v - cur[o]));
            far = far || (a >= ltol && a <= linf);
        }
        far = __syncthreads_or(far);
        double *t = cur;
        cur = next;
        next = t;
        fresh = false;
        return far;
    };
    int done = 0;  // sweeps completed before this batch; sweep s is iteration number s
    bool converged = false;
    for (int batch = 0; ok; batch++) {
        const int n = min(JT_BATCH, ITER_MAX + 1 - done);
        if (batch) store(cur, u1);
        unsigned long long moved = 0;
        for (int s = 0; s < n && ok; s++)
            if (sweep()) moved |= 1ull << s;
        if (!ok) break;
        if (threadIdx.x == 0 && moved) atomicOr(jt.moved + batch, moved);
        ok = jt_barrier(jt.arrived, ++round);
        if (!ok) break;
        const unsigned long long still = ~__ldcg(jt.moved + batch);
        const int first = still ? __ffsll((long long)still) - 1 : JT_BATCH;  // first sweep in which nothing moved
        if (first < n) {
            converged = true;
            if (first < n - 1) {  // back to the batch's start, and up to that sweep
                load(cur, u1);
                fresh = true;
                ok = jt_barrier(jt.arrived, ++round);
                for (int s = 0; s <= first && ok; s++) sweep();
            }
            done += first + 1;
            break;
        }
        done += n;
        if (done > ITER_MAX) break;
    }
    // the last sweep's result and the one before it, in the arrays the
    // alternating sweeps leave them in
    if (ok) {
        store(cur, (done - 1) % 2 == 0 ? u2 : u1);
        store(next, (done - 1) % 2 == 0 ? u1 : u2);
    }
    if (threadIdx.x == 0) {
        if (!ok) st->error = 1;
        if (blockIdx.x == 0) {
            st->done = 1;
            st->iter = done;
            st->converged = converged;
        }
    }
}

// One Jacobi sweep with the stop test of k_jacobi_check folded in, for grids
// periodic on every side: there the boundary fill writes only ghost planes,
// so max |u2 - u1| over the physical points is max |dst - src| of this sweep,
// the same value in any order. The sweep's arithmetic is k_jacobi's. Once the
// test has fired, the next sweep sets `skip`, so the fill after the last
// sweep still runs and the later ones do not.
__global__ void k_jacobi_fused(Geom g, const double *src, double *dst, const double *R, double ax, double ay,
                               double az, double af, double mult, double tol, JacobiState *st) {
    if (st->done) {
        if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.x == 0 && threadIdx.y == 0) st->skip = 1;
        return;
    }
    __shared__ double smax[32];
    __shared__ bool last;
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z + 1;
    double m = 0.0;
    if (k <= g.n[2] && j <= g.n[1]) {
        const int64_t o = gidx(g, i, j, k);
        const double v = ax * (src[o - g.sx] + src[o + g.sx]) + ay * (src[o - g.sy] + src[o + g.sy]) +
                         az * (src[o - 1] + src[o + 1]) - af * R[o] * mult;
        dst[o] = v;
        m = fabs(v - src[o]);
    }
    for (int off = 16; off > 0; off >>= 1) {
        const double q = __shfl_down_sync(0xffffffffu, m, off);
        m = q > m ? q : m;
    }
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int nw = (int)((blockDim.x * blockDim.y) >> 5);
    if (lane == 0) smax[w] = m;
    __syncthreads();
    if (w == 0) {
        m = lane < nw ? smax[lane] : 0.0;
        for (int off = 16; off > 0; off >>= 1) {
            const double q = __shfl_down_sync(0xffffffffu, m, off);
            m = q > m ? q : m;
        }
        if (lane == 0) {
            atomic_max_nonneg(&st->maxdiff, m);
            __threadfence();
            const unsigned int nb = gridDim.x * gridDim.y * gridDim.z;
            const unsigned int prev = atomicAdd(&st->blocks_done, 1u);
            last = (prev == nb - 1);
        }
    }
    __syncthreads();
    if (last && tid == 0) {
        __threadfence();
        const double md = *((volatile double *)&st->maxdiff);
        const int it = st->iter;
        if (md < tol) {
            st->done = 1;
            st->converged = 1;
        } else if (it >= ITER_MAX) {
            st->done = 1;
            st->converged = 0;
        }
        st->iter = it + 1;
        st->maxdiff = 0.0;
        st->blocks_done = 0u;
    }
}

// phiToE, src/poisson/convertFields.cpp:20-68 (reads phi1 storage).
__global__ void k_phi_to_e(Geom g, const double *phi, F3 E) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    E.p[0][o] = ddiv(-(phi[o + g.sx] - phi[o]), g.d[0], g.id[0], g.p2[0]);
    E.p[1][o] = ddiv(-(phi[o + g.sy] - phi[o]), g.d[1], g.id[1], g.p2[1]);
    E.p[2][o] = ddiv(-(phi[o + 1] - phi[o]), g.d[2], g.id[2], g.p2[2]);
}

// AToB, src/poisson/convertFields.cpp:83-154, including its use of the same
// A component in both differences.
__global__ void k_a_to_b(Geom g, const double *Ax, const double *Ay, const double *Az, F3 B) {
    after_previous();
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    int64_t o = gidx(g, i, j, k);
    // Bx: Ak = Az (hk = dz), Aj = Ay (hj = dy); next_k = Ak[j+1], next_j = Ak[k+1]
    B.p[0][o] = ddiv(Az[o + g.sy] - Az[o], g.d[1], g.id[1], g.p2[1]) + ddiv(Az[o + 1] - Ay[o], g.d[2], g.id[2], g.p2[2]);
    // By: Ak = Ax (hk = dx), Aj = Az (hj = dz); next_k = Ak[k+1], next_j = Ak[i+1]
    B.p[1][o] = ddiv(Ax[o + 1] - Ax[o], g.d[2], g.id[2], g.p2[2]) + ddiv(Ax[o + g.sx] - Az[o], g.d[0], g.id[0], g.p2[0]);
    // Bz: Ak = Ay (hk = dy), Aj = Ax (hj = dx); next_k = Ak[i+1], next_j = Ak[j+1]
    B.p[2][o] = ddiv(Ay[o + g.sx] - Ay[o], g.d[0], g.id[0], g.p2[0]) + ddiv(Ay[o + g.sy] - Ax[o], g.d[1], g.id[1], g.p2[1]);
}

// Per-block partial sums of the six field energies of the history row
// (src/IO/output.cpp:98-114; SQR(x) expands to x*x unparenthesised).
__global__ void k_field_energy(Geom g, CF3 E, CF3 B, double *part) {
    after_previous();
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // 6 used
    int64_t nphys = (int64_t)g.n[0] * g.n[1] * g.n[2];
    double hv = 0.5 * g.vol;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nphys; t += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        phys_ijk(g.n, t, i, j, k);
        int64_t o = gidx(g, i, j, k);
        int64_t nb[3] = {o + g.sx, o + g.sy, o + 1};
        for (int q = 0; q < 3; q++) {
            double s = E.p[q][o] + E.p[q][nb[q]];
            acc[q] += hv * (0.5 * s * 0.5 * s);
            double sb = B.p[q][o] + B.p[q][nb[q]];
            acc[3 + q] += hv * (0.5 * sb * 0.5 * sb);
        }
    }
    __shared__ double sh[32][6];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double total = warp_totals<8>(acc);
    const int at = total_index<8>(lane);
    if ((lane & 3) == 0 && at < 6) sh[w][at] = total;
    __syncthreads();
    if (threadIdx.x < 6) {
        double v = 0.0;
        for (int ww = 0; ww < (int)(blockDim.x >> 5); ww++) v += sh[ww][threadIdx.x];
        part[blockIdx.x * 6 + threadIdx.x] = v;
    }
}

// Gauss-law residual partials: {max |div E - 4 pi rho|, sum r^2}.
__global__ void k_gauss(Geom g, CF3 E, const double *rho, double *part) {
    double mx = 0.0, s2 = 0.0;
    int64_t nphys = (int64_t)g.n[0] * g.n[1] * g.n[2];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nphys; t += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        phys_ijk(g.n, t, i, j, k);
        int64_t o = gidx(g, i, j, k);
        double dv = ddiv(E.p[0][o] - E.p[0][o - g.sx], g.d[0], g.id[0], g.p2[0]) +
                    ddiv(E.p[1][o] - E.p[1][o - g.sy], g.d[1], g.id[1], g.p2[1]) +
                    ddiv(E.p[2][o] - E.p[2][o - 1], g.d[2], g.id[2], g.p2[2]);
        double res = dv - FOURPI * rho[o];
        double a = fabs(res);
        mx = a > mx ? a : mx;
        s2 += res * res;
    }
    __shared__ double sh[32][2];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int off = 16; off > 0; off >>= 1) {
        double o = __shfl_down_sync(0xffffffffu, mx, off);
        mx = o > mx ? o : mx;
        s2 += __shfl_down_sync(0xffffffffu, s2, off);
    }
    if (lane == 0) {
        sh[w][0] = mx;
        sh[w][1] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int ww = 0; ww < (int)(blockDim.x >> 5); ww++) {
            a = sh[ww][0] > a ? sh[ww][0] : a;
            b += sh[ww][1];
        }
        part[blockIdx.x * 2] = a;
        part[blockIdx.x * 2 + 1] = b;
    }
}

int ensure_red(emoo_handle *h, size_t n) {
    if (h->red_cap >= n) return EMOO_OK;
    if (h->red) cudaFree(h->red);
    h->red = nullptr;
    EMOO_CUDA(cudaMalloc(&h->red, n * sizeof(double)));
    h->red_cap = n;
    return EMOO_OK;
}

int reduce_blocks(const Geom &g) {
    int64_t nphys = (int64_t)g.n[0] * g.n[1] * g.n[2];
    int64_t b = (nphys + 255) / 256;
    return (int)std::min<int64_t>(b, 152 * 8);
}

}  // namespace

double *role_b(emoo_handle *h, int c) { return h->bswap ? h->slot[EMOO_BX_TM1 + c] : h->slot[EMOO_BX + c]; }
double *role_t(emoo_handle *h, int c) { return h->bswap ? h->slot[EMOO_BX + c] : h->slot[EMOO_BX_TM1 + c]; }

int yee_f64(emoo_handle *h, double dt, bool fold_j) {
    // std::swap of the member pointers only (src/grid/oGrid.cpp:18-20)
    h->bswap ^= 1;
    const Geom &g = h->g;
    dim3 blk(32, 8);
    dim3 grd = phys_grid(g, blk);
    F3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
    CF3 T = {{role_t(h, 0), role_t(h, 1), role_t(h, 2)}};
    F3 J = {{h->slot[EMOO_JX], h->slot[EMOO_JY], h->slot[EMOO_JZ]}};
    h->launches++;
    FoldDims f;
    for (int d = 0; d < 3; d++) f.per[d] = h->bc.fbc[2 * d] == FBC_PERIODIC;
    if (fold_j) launch_after(k_yee_e<true>, grd, blk, 0, h->stream)(g, dt, E, T, J, f);
    else launch_after(k_yee_e<false>, grd, blk, 0, h->stream)(g, dt, E, T, J, f);
    // The B half reads E one plane past the high faces. The reference refreshes
    // those ghosts only after both halves, so at the periodic wrap B sees the
    // previous step's E: the leapfrog loses its time centring there and vacuum
    // fields grow without bound at dt 0.5. The corrected policy refreshes them.
    if (h->policy == EMOO_POLICY_CORRECTED) EMOO_TRY(ghost_e_full_f64(h));
    F3 B = {{role_b(h, 0), role_b(h, 1), role_b(h, 2)}};
    CF3 Ec = {{E.p[0], E.p[1], E.p[2]}};
    h->launches++;
    launch_after(k_yee_b, grd, blk, 0, h->stream)(g, dt, B, T, Ec);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int yee_half_f64(emoo_handle *h, double dt, int half) {
    const Geom &g = h->g;
    dim3 blk(32, 8);
    dim3 grd = phys_grid(g, blk);
    CF3 T = {{role_t(h, 0), role_t(h, 1), role_t(h, 2)}};
    h->launches++;
    if (half == 0) {
        F3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
        F3 J = {{h->slot[EMOO_JX], h->slot[EMOO_JY], h->slot[EMOO_JZ]}};
        launch_after(k_yee_e<false>, grd, blk, 0, h->stream)(g, dt, E, T, J, FoldDims{});
    } else {
        F3 B = {{role_b(h, 0), role_b(h, 1), role_b(h, 2)}};
        CF3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
        launch_after(k_yee_b, grd, blk, 0, h->stream)(g, dt, B, T, E);
    }
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int yee_es_f64(emoo_handle *h, double dt) {
    const Geom &g = h->g;
    dim3 blk(32, 8);
    F3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
    CF3 J = {{h->slot[EMOO_JX], h->slot[EMOO_JY], h->slot[EMOO_JZ]}};
    h->launches++;
    launch_after(k_yee_es, phys_grid(g, blk), blk, 0, h->stream)(g, dt, E, J);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

static int ghost_launch(emoo_handle *h, const int *ids, int nids, int dims_mask, const int *skip) {
    const Geom &g = h->g;
    FieldList fl;
    fl.n = nids;
    for (int i = 0; i < nids; i++) fl.p[i] = h->slot[ids[i]];
    int ta = std::max(g.n[1], g.n[0]);
    int tb = std::max(g.n[2], g.n[1]);
    dim3 blk(32, 8);
    dim3 grd((tb + 31) / 32, (ta + 7) / 8, nids * 6);
    h->launches++;
    launch_after(k_ghost, grd, blk, 0, h->stream)(g, fl, dims_mask, skip);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int ghost_fill_f64(emoo_handle *h, const int *ids, int nids, int dims_mask) {
    return ghost_launch(h, ids, nids, dims_mask, nullptr);
}

// what: FOLD_J (the two transverse J components), FOLD_RHO, or both
int fold_f64(emoo_handle *h, int d, int what) {
    const Geom &g = h->g;
    int f0 = (d == 0) ? EMOO_JY : EMOO_JX;
    int f1 = (d == 2) ? EMOO_JY : EMOO_JZ;
    int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    dim3 blk(32, 8);
    double *a = h->slot[f0], *b = h->slot[f1], *r = h->slot[EMOO_RHO];
    int nz = 3;
    if (what == FOLD_J) nz = 2;
    if (what == FOLD_RHO) {
        nz = 1;
        a = r;
    }
    dim3 grd((g.n[o2] + 31) / 32, (g.n[o1] + 7) / 8, nz);
    h->launches++;
    launch_after(k_fold, grd, blk, 0, h->stream)(g, d, a, b, r);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

// ---- corrected policy: periodic copies and folds over the whole range ----

struct Slots9 {
    double *p[9];
};

// Fold along dim d, for every transverse point of the whole (n+3)^2 plane:
// f[n] += f[0], f[1] += f[n+1], f[2] += f[n+2] (the ghost planes' deposits to
// their periodic images). One field per blockIdx.z.
__global__ void k_periodic_full(Geom g, Slots9 fl, int d) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (q >= g.tot[o2] || r >= g.tot[o1]) return;
    double *F = fl.p[blockIdx.z];
    const int n = g.n[d];
    int c[3];
    c[o1] = r;
    c[o2] = q;
    auto at = [&](int i) -> double & {
        c[d] = i;
        return F[gidx(g, c[0], c[1], c[2])];
    };
    at(n) += at(0);
    at(1) += at(n + 1);
    at(2) += at(n + 2);
}

struct Wrap {
    int w[3];
};

// Ghost copies of nf fields over the whole range in one launch: each ghost
// point takes the value of the point it is an image of (never a ghost), all
// fields' loads in flight together. 49 x 37 x 29 cells, nine fields: 4.0 us
// (9.6 us from the sources, a thread a point of the grid).
__global__ void k_copy_images(Geom g, Slots9 fl, int nf, Wrap w, Slabs S) {
    after_previous();
    int c[3], of[3];
    if (!ghost_point(S, g.n, w.w, blockIdx.x * blockDim.x + threadIdx.x, c, of)) return;
    const int64_t o = gidx(g, c[0], c[1], c[2]), from = gidx(g, of[0], of[1], of[2]);
    double v[9];
#pragma unroll
    for (int q = 0; q < 9; q++)
        if (q < nf) v[q] = fl.p[q][from];
#pragma unroll
    for (int q = 0; q < 9; q++)
        if (q < nf) fl.p[q][o] = v[q];
}

// Mirror fold at a reflecting wall (corrected policy, no reference
// counterpart): a particle reflected at the wall moved along the mirror image
// of the part of its straight path beyond it, so the current that part
// deposited in the ghost layer goes to the mirrored points inside - the
// component normal to the wall negated, the transverse ones as they are - and
// the ghost values are cleared. Left wall (vertex plane 1): normal edge 0 ->
// 1, transverse plane 0 -> 2; right wall (plane n+1): normal edge n+1 -> n,
// transverse plane n+2 -> n. Whole transverse range; blockIdx.z = component.
__global__ void k_mirror_fold(Geom g, Slots9 fl, int d, int right) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (q >= g.tot[o2] || r >= g.tot[o1]) return;
    const int a = blockIdx.z;
    double *F = fl.p[a];
    const int n = g.n[d];
    const bool normal = a == d;
    const int src = normal ? (right ? n + 1 : 0) : (right ? n + 2 : 0);
    const int dst = normal ? (right ? n : 1) : (right ? n : 2);
    int c[3];
    c[o1] = r;
    c[o2] = q;
    c[d] = src;
    const int64_t ks = gidx(g, c[0], c[1], c[2]);
    c[d] = dst;
    const int64_t kd = gidx(g, c[0], c[1], c[2]);
    if (normal) F[kd] -= F[ks];
    else F[kd] += F[ks];
    F[ks] = 0.0;
}

// The corrected policy's folds (J and / or rho), dimension by dimension so edge
// and corner lines follow: periodic dimensions as images over the whole range;
// walled dimensions (corrected policy with reflecting or absorbing particle
// sides) fold J by mirror at reflecting sides only (at absorbing ones the
// current of the path beyond the wall stays in the ghost layer).
static int periodic_fold(emoo_handle *h, const int *ids, int nids) {
    const Geom &g = h->g;
    Slots9 fl;
    for (int k = 0; k < nids; k++) fl.p[k] = h->slot[ids[k]];
    dim3 blk(32, 8);
    for (int d = 0; d < 3; d++) {
        const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
        if (h->bc.fbc[2 * d] != FBC_PERIODIC) {
            const bool j3 = nids >= 3 && ids[0] == EMOO_JX && ids[1] == EMOO_JY && ids[2] == EMOO_JZ;
            for (int r = 0; r < 2 && j3; r++) {
                if (h->bc.pbc[2 * d + r] != PBC_REFLECTING) continue;
                dim3 grd((g.tot[o2] + 31) / 32, (g.tot[o1] + 7) / 8, 3);
                h->launches++;
                launch_after(k_mirror_fold, grd, blk, 0, h->stream)(g, fl, d, r);
            }
            continue;
        }
        dim3 grd((g.tot[o2] + 31) / 32, (g.tot[o1] + 7) / 8, nids);
        h->launches++;
        launch_after(k_periodic_full, grd, blk, 0, h->stream)(g, fl, d);
    }
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

// what: FOLD_J (the three J components), FOLD_RHO, or both
int fold_full_f64(emoo_handle *h, int what) {
    int ids[4], n = 0;
    if (what & FOLD_J)
        for (int c = 0; c < 3; c++) ids[n++] = EMOO_JX + c;
    if (what & FOLD_RHO) ids[n++] = EMOO_RHO;
    return periodic_fold(h, ids, n);
}

// LightBC planes of every external side (E and B roles through the slots), one
// launch a dimension (its sides are both external).
static int light_all_f64(emoo_handle *h) {
    PlaneSet ps[12];
    int n = 0;
    for (int s = 0; s < 6; s++) {
        if (h->bc.fbc[s] != FBC_EXTERNAL) continue;
        n += light_planes_slots(h, s, ps + n);
        if (n > 6 || h->g.n[s / 2] < 2) {  // of one cell, both sides set the same plane: in order
            EMOO_TRY(plane_set_f64(h, ps, n));
            n = 0;
        }
    }
    return n ? plane_set_f64(h, ps, n) : EMOO_OK;
}

// E's boundary values between the Yee halves (corrected policy): periodic
// images and LightBC planes, so the B half reads E at the new time everywhere.
int ghost_e_full_f64(emoo_handle *h) {
    static const int ids[3] = {EMOO_EX, EMOO_EY, EMOO_EZ};
    EMOO_TRY(periodic_copies_f64(h, ids, 3));
    return light_all_f64(h);
}

// The corrected policy's ghost copies; walled dimensions copy nothing (their
// field sides are LightBC planes).
int periodic_copies_f64(emoo_handle *h, const int *ids, int nids) {
    Slots9 fl;
    Wrap w;
    for (int k = 0; k < nids; k++) fl.p[k] = h->slot[ids[k]];
    for (int d = 0; d < 3; d++) w.w[d] = h->bc.fbc[2 * d] == FBC_PERIODIC;
    const Slabs S = ghost_slabs(h->g.n, w.w);
    const int64_t ghosts = slab_size(S);
    if (!ghosts) return EMOO_OK;
    h->launches++;
    launch_after(k_copy_images, (unsigned)((ghosts + 127) / 128), 128, 0, h->stream)(h->g, fl, nids, w, S);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int ghost_full_f64(emoo_handle *h) {
    static const int ids[9] = {EMOO_EX, EMOO_EY, EMOO_EZ, EMOO_BX, EMOO_BY, EMOO_BZ, EMOO_BX_TM1, EMOO_BY_TM1,
                               EMOO_BZ_TM1};
    EMOO_TRY(periodic_copies_f64(h, ids, 9));
    return light_all_f64(h);
}

static int plane_launch(emoo_handle *h, const PlaneSet *ps, int n, const int *skip) {
    const Geom &g = h->g;
    for (int b = 0; b < n; b += 12) {
        PlaneList pl;
        pl.n = std::min(12, n - b);
        for (int i = 0; i < pl.n; i++) pl.s[i] = ps[b + i];
        int m = std::max(std::max(g.tot[0], g.tot[1]), g.tot[2]);
        dim3 blk(32, 8);
        dim3 grd((m + 31) / 32, (m + 7) / 8, pl.n);
        h->launches++;
        launch_after(k_plane_set, grd, blk, 0, h->stream)(g, pl, skip);
    }
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int plane_set_f64(emoo_handle *h, const PlaneSet *ps, int n) { return plane_launch(h, ps, n, nullptr); }

// rho += background at the physical points with x index >= i0 (immobile
// neutralising ions; no reference counterpart).
__global__ void k_add_phys(Geom g, double *f, double v, int i0) {
    int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    int i = blockIdx.z + i0;
    if (k > g.n[2] || j > g.n[1]) return;
    f[(int64_t)i * g.sx + (int64_t)j * g.sy + k] += v;
}

int rho_background_f64(emoo_handle *h, int with_rho) {
    if (!with_rho || h->opts.rho_background == 0.0 || h->rho_bg_first > h->g.n[0]) return EMOO_OK;
    const Geom &g = h->g;
    dim3 blk(32, 8);
    dim3 grd((g.n[2] + 31) / 32, (g.n[1] + 7) / 8, g.n[0] - h->rho_bg_first + 1);
    h->launches++;
    k_add_phys<<<grd, blk, 0, h->stream>>>(g, h->slot[EMOO_RHO], h->opts.rho_background, h->rho_bg_first);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int fill_f64(emoo_handle *h, double *p, int64_t n, double v, cudaStream_t s) {
    (void)h;
    int64_t b = std::min<int64_t>((n + 255) / 256, 152 * 16);
    if (b < 1) b = 1;
    h->launches++;
    launch_after(k_fill, (int)b, 256, 0, s)(p, n, v);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

// executeBC(fieldID) for one Poisson field: periodic dims by ghost copy,
// external sides by PoissonBC Dirichlet planes (left: plane 1, right: n+1),
// in the reference's dimension order; `skip` makes the launches no-ops once
// the Jacobi loop has finished.
static int single_field_bc(emoo_handle *h, int id, const int *skip) {
    int mask_run = 0;
    for (int d = 0; d < 3; d++) {
        bool per = h->bc.fbc[2 * d] == FBC_PERIODIC;
        if (per) {
            mask_run |= 1 << d;
            continue;
        }
        if (mask_run) {
            EMOO_TRY(ghost_launch(h, &id, 1, mask_run, skip));
            mask_run = 0;
        }
        if (!h->poisson || id <= 0) continue;
        PlaneSet ps[2] = {};
        int np = 0;
        for (int r = 0; r < 2; r++) {
            int s = 2 * d + r;
            if (h->bc.fbc[s] != FBC_EXTERNAL) continue;
            int fid = (id == EMOO_PHI1 || id == EMOO_PHI2) ? 0 : (id == EMOO_AX1 || id == EMOO_AX2) ? 1
                      : (id == EMOO_AY1 || id == EMOO_AY2) ? 2 : (id == EMOO_AZ1 || id == EMOO_AZ2) ? 3 : -1;
            if (fid < 0) continue;
            double v = fid == 0 ? h->info.bound_phi[s] : fid == 1 ? h->info.bound_Ax[s]
                                : fid == 2 ? h->info.bound_Ay[s] : h->info.bound_Az[s];
            ps[np].f = h->slot[id];
            ps[np].dim = d;
            ps[np].idx = r == 0 ? 1 : h->g.n[d] + 1;
            ps[np].v = v;
            np++;
        }
        for (int i = 0; i < np; i++) EMOO_TRY(plane_launch(h, &ps[i], 1, skip));
    }
    if (mask_run) EMOO_TRY(ghost_launch(h, &id, 1, mask_run, skip));
    return EMOO_OK;
}

// The Poisson fields' boundary fill (executeBC(fieldID)) as the Jacobi loop
// applies it, for the multigrid's start and result.
int poisson_field_bc(emoo_handle *h, int id) { return single_field_bc(h, id, nullptr); }

// The tiles of k_jacobi_tiles for this grid and their scratch (kept with the
// handle); b[0] = 0 where the kernel does not apply: a side that is not
// periodic, or a tile that does not fit a block's shared memory. The cut is
// the one whose largest tile takes the fewest cycles: 160 of the FP64 pipe for
// each 32 points, and about 4 for a face value sent and received. Six grids from
// 8^3 to 64^3, twenty cuts each: its choice was within 4 % of the fastest (32^3:
// 1.86 us a sweep, fastest 1.83, slowest 3.70; 24 x 40 x 16: 2.02, 1.94, 2.55).
static int jacobi_tiling(emoo_handle *h, JacobiTiles *jt, size_t *smem) {
    const Geom &g = h->g;
    *jt = JacobiTiles{};
    for (int s = 0; s < 6; s++)
        if (h->bc.fbc[s] != FBC_PERIODIC) return EMOO_OK;
    int sms = 0, smem_max = 0, coop = 0;
    EMOO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->dev));
    EMOO_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->dev));
    EMOO_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->dev));
    if (!coop) return EMOO_OK;
    int64_t best = INT64_MAX;
    for (int bx = 1; bx <= std::min(sms, g.n[0]); bx++)
        for (int by = 1; by <= std::min(sms / bx, g.n[1]); by++) {
            const int bz = std::min(sms / (bx * by), g.n[2]);
            const int64_t t[3] = {(g.n[0] + bx - 1) / bx, (g.n[1] + by - 1) / by, (g.n[2] + bz - 1) / bz};
            const int64_t vol = t[0] * t[1] * t[2], halo = 2 * (t[0] * t[1] + t[0] * t[2] + t[1] * t[2]);
            const int64_t bytes = (2 * (t[0] + 2) * (t[1] + 2) * (t[2] + 2) + vol) * (int64_t)sizeof(double);
            const int64_t cost = (vol + 31) / 32 * 160 + halo * 4;
            if (bytes > smem_max || cost >= best) continue;
            best = cost;
            *smem = (size_t)bytes;
            const int b[3] = {bx, by, bz};
            for (int d = 0; d < 3; d++) {
                jt->b[d] = b[d];
                jt->t[d] = (int)t[d];
            }
            jt->face = (int)std::max(t[0] * t[1], std::max(t[0] * t[2], t[1] * t[2]));
        }
    if (!jt->b[0]) return EMOO_OK;
    // the limit is the function's, for every handle: always the device's largest
    EMOO_CUDA(cudaFuncSetAttribute(k_jacobi_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    const int blocks = jt->b[0] * jt->b[1] * jt->b[2], batches = ITER_MAX / JT_BATCH + 2;
    const size_t faces = (size_t)blocks * 12 * jt->face * sizeof(ulonglong2);
    const size_t bytes = faces + batches * sizeof(unsigned long long) + sizeof(unsigned long long);
    if (!h->jacobi_tiles) EMOO_CUDA(cudaMalloc(&h->jacobi_tiles, bytes));  // one grid, one size a handle
    char *p = (char *)h->jacobi_tiles;
    jt->faces = (ulonglong2 *)p;
    jt->moved = (unsigned long long *)(p + faces);
    jt->arrived = (unsigned int *)(jt->moved + batches);
    EMOO_CUDA(cudaMemsetAsync(p, 0, bytes, h->stream));
    return EMOO_OK;
}

// Poisson_Solver::run_poisson_solver_, src/poisson/poisson.cpp:172-287, with
// the iteration control on the device: iterations are queued in batches and
// become no-ops once the stop test of the reference has fired.
int jacobi_f64(emoo_handle *h, int id1, int id2, int rid, double tol, double mult, int *iters, int *converged) {
    const Geom &g = h->g;
    double dx = g.d[0], dy = g.d[1], dz = g.d[2];
    double celldist2 = pow(dx, 2.0) * pow(dy, 2.0) + pow(dy, 2.0) * pow(dz, 2.0) + pow(dx, 2.0) * pow(dz, 2.0);
    double ax = pow(dy, 2.0) * pow(dz, 2.0) / (2.0 * celldist2);
    double ay = pow(dx, 2.0) * pow(dz, 2.0) / (2.0 * celldist2);
    double az = pow(dx, 2.0) * pow(dy, 2.0) / (2.0 * celldist2);
    double af = pow(dx, 2.0) * pow(dy, 2.0) * pow(dz, 2.0) / (2.0 * celldist2);
    if (!h->jacobi_state) EMOO_CUDA(cudaMalloc(&h->jacobi_state, sizeof(JacobiState)));
    JacobiState *st = (JacobiState *)h->jacobi_state;
    EMOO_CUDA(cudaMemsetAsync(st, 0, sizeof(JacobiState), h->stream));
    EMOO_TRY(single_field_bc(h, id1, nullptr));
    double *u1 = h->slot[id1], *u2 = h->slot[id2];
    const double *R = h->slot[rid];
    JacobiState hs;
    JacobiTiles jt;
    size_t smem = 0;
    EMOO_TRY(jacobi_tiling(h, &jt, &smem));
    if (jt.b[0]) {
        int threads = std::min(JT_THREADS, (jt.t[0] * jt.t[1] * jt.t[2] + 31) / 32 * 32);
        void *args[] = {(void *)&g,  &u1, &u2, (void *)&R, &ax, &ay, &az, &af, &mult, &tol, &jt, &st};
        h->launches++;
        EMOO_CUDA(cudaLaunchCooperativeKernel((const void *)k_jacobi_tiles, dim3(jt.b[0] * jt.b[1] * jt.b[2]),
                                              dim3(threads), args, smem, h->stream));
        EMOO_TRY(single_field_bc(h, id1, nullptr));
        EMOO_TRY(single_field_bc(h, id2, nullptr));
        EMOO_CUDA(cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, h->stream));
        EMOO_CUDA(cudaStreamSynchronize(h->stream));
        if (hs.error) {
            fprintf(stderr, "emoo: a wait of the Jacobi kernel ran out\n");
            return EMOO_ERR_CUDA;
        }
        if (iters) *iters = hs.iter - 1;
        if (converged) *converged = hs.converged;
        return EMOO_OK;
    }
    dim3 blk(32, 8);
    dim3 grd = phys_grid(g, blk);
    int rb = reduce_blocks(g);
    // Sweeps are queued in batches of 32 (an even count, so every batch starts
    // on the same ping-pong parity), captured once as a CUDA graph and
    // replayed: at small grids each sweep's three kernels would otherwise cost
    // a launch latency each. Once the stop test has fired they are no-ops.
    const int batch = 32;
    int batch_launches = 0;
    // With every side periodic (and a grid past the tiles' shared memory) the
    // stop test can run inside the sweep: one kernel fewer per sweep. On large
    // grids the sweep's per-block FP64 max trees (FP64 pipe) cost more than
    // the separate check's grid-stride reduction, so it stays separate there.
    bool all_periodic = (int64_t)g.n[0] * g.n[1] * g.n[2] <= (int64_t)1 << 21;
    for (int sd = 0; sd < 6; sd++) all_periodic = all_periodic && h->bc.fbc[sd] == FBC_PERIODIC;
    auto queue_batch = [&]() -> int {
        for (int b = 0; b < batch; b++) {
            const bool even = (b % 2) == 0;
            batch_launches++;
            if (all_periodic)  // (and small)
                k_jacobi_fused<<<grd, blk, 0, h->stream>>>(g, even ? u1 : u2, even ? u2 : u1, R, ax, ay, az, af, mult,
                                                           tol, st);
            else
                k_jacobi<<<grd, blk, 0, h->stream>>>(g, even ? u1 : u2, even ? u2 : u1, R, ax, ay, az, af, mult, st);
            const int64_t before = h->launches;
            EMOO_TRY(single_field_bc(h, even ? id2 : id1, all_periodic ? &st->skip : &st->done));
            batch_launches += (int)(h->launches - before);
            h->launches = before;
            if (!all_periodic) {
                batch_launches++;
                k_jacobi_check<<<rb, 256, 0, h->stream>>>(g, u1, u2, tol, st);
            }
        }
        return EMOO_OK;
    };
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    EMOO_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int qrc = queue_batch();
    const cudaError_t ce = cudaStreamEndCapture(h->stream, &graph);
    if (qrc != EMOO_OK || ce != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return qrc != EMOO_OK ? qrc : cuda_status(ce);
    }
    cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return cuda_status(ie);
    int launched = 0;
    int rc = EMOO_OK;
    for (;;) {
        cudaError_t e = cudaGraphLaunch(exec, h->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) {
            rc = cuda_status(e);
            break;
        }
        h->launches += batch_launches;
        launched += batch;
        if (hs.done || launched > ITER_MAX) break;
    }
    cudaGraphExecDestroy(exec);
    if (rc != EMOO_OK) return rc;
    if (iters) *iters = hs.iter - 1;
    if (converged) *converged = hs.converged;
    return EMOO_OK;
}

int phi_to_e_f64(emoo_handle *h) {
    const Geom &g = h->g;
    dim3 blk(32, 8);
    F3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
    h->launches++;
    launch_after(k_phi_to_e, phys_grid(g, blk), blk, 0, h->stream)(g, h->slot[EMOO_PHI1], E);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int a_to_b_f64(emoo_handle *h) {
    const Geom &g = h->g;
    dim3 blk(32, 8);
    // AToB writes through the field pointer table: the fixed B slots.
    F3 B = {{h->slot[EMOO_BX], h->slot[EMOO_BY], h->slot[EMOO_BZ]}};
    h->launches++;
    launch_after(k_a_to_b, phys_grid(g, blk), blk, 0, h->stream)(g, h->slot[EMOO_AX1], h->slot[EMOO_AY1], h->slot[EMOO_AZ1], B);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int field_energy_f64(emoo_handle *h, double out6[6]) {
    const Geom &g = h->g;
    int rb = reduce_blocks(g);
    EMOO_TRY(ensure_red(h, (size_t)rb * 6));
    CF3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
    // the history reads the field pointer table: fixed B slots
    CF3 B = {{h->slot[EMOO_BX], h->slot[EMOO_BY], h->slot[EMOO_BZ]}};
    h->launches++;
    launch_after(k_field_energy, rb, 256, 0, h->stream)(g, E, B, h->red);
    EMOO_CUDA(cudaGetLastError());
    std::vector<double> part((size_t)rb * 6);
    EMOO_CUDA(cudaMemcpyAsync(part.data(), h->red, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    EMOO_CUDA(cudaStreamSynchronize(h->stream));
    for (int q = 0; q < 6; q++) out6[q] = 0.0;
    for (int b = 0; b < rb; b++)
        for (int q = 0; q < 6; q++) out6[q] += part[(size_t)b * 6 + q];
    return EMOO_OK;
}

int gauss_residual_f64(emoo_handle *h, double out2[2]) {
    const Geom &g = h->g;
    int rb = reduce_blocks(g);
    EMOO_TRY(ensure_red(h, (size_t)rb * 2));
    CF3 E = {{h->slot[EMOO_EX], h->slot[EMOO_EY], h->slot[EMOO_EZ]}};
    h->launches++;
    k_gauss<<<rb, 256, 0, h->stream>>>(g, E, h->slot[EMOO_RHO], h->red);
    EMOO_CUDA(cudaGetLastError());
    std::vector<double> part((size_t)rb * 2);
    EMOO_CUDA(cudaMemcpyAsync(part.data(), h->red, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    EMOO_CUDA(cudaStreamSynchronize(h->stream));
    double mx = 0.0, s2 = 0.0;
    for (int b = 0; b < rb; b++) {
        mx = std::max(mx, part[(size_t)b * 2]);
        s2 += part[(size_t)b * 2 + 1];
    }
    out2[0] = mx;
    out2[1] = sqrt(s2);
    return EMOO_OK;
}

}  // namespace emoo
