// adjoint_fields.cuh - transposed field kernels of the differentiated step,
// templated on the adjoint's scalar (double for the FP64 form, float for the
// mixed form). The forward maps are the same linear stencils in both forms
// (the Yee update of src/grid/oGrid.cpp:15-60, the periodic ghost copy of
// src/boundaries/b_fields/bc_f_periodic.cpp:47-52 over the physical
// transverse range, the J fold of src/grid/spookyGrid.cpp:21-26, LightBC's
// plane sets), so one transpose serves both.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "dev_common.cuh"
#include "emoo_internal.h"

namespace emoo {
namespace adf {

constexpr double FOURPI = 4.0 * PI_D;

template <class R>
struct FOutT {
    R *E[3], *B[3], *T[3];  // E, B role, B_tm1 role
};
template <class R>
struct JPtrsT {
    R *J[3];
};
template <class R>
struct Slots6T {
    R *p[6];
};
template <class R>
struct Slots9T {
    R *p[9];
};

__device__ __forceinline__ bool phys(const Geom &g, int i, int j, int k) {
    return i >= 1 && i <= g.n[0] && j >= 1 && j <= g.n[1] && k >= 1 && k <= g.n[2];
}

// The stencil coefficients dt / d (and -4 pi dt), computed once on the host:
// per-thread FP64 divisions would run on this GPU's narrow FP64 pipe.
template <class R>
struct YeeCoef {
    R cx, cy, cz, cj;
};

template <class R>
YeeCoef<R> yee_coef(const Geom &g, double dt) {
    return YeeCoef<R>{(R)(dt / g.d[0]), (R)(dt / g.d[1]), (R)(dt / g.d[2]), (R)(-FOURPI * dt)};
}

// Adjoint of the B update (B = T + dt curl E over the physical points),
// gather form over every grid point: LT += LB (physical), LE += dt C_E^T LB.
template <class R>
__global__ void k_yee_b_adj(Geom g, YeeCoef<R> yc, FOutT<R> A) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= g.tot[2] || j >= g.tot[1] || i >= g.tot[0]) return;
    const int64_t p = gidx(g, i, j, k), sx = g.sx, sy = g.sy;
    const R cx = yc.cx, cy = yc.cy, cz = yc.cz;
    const bool here = phys(g, i, j, k);
    if (here)
        for (int c = 0; c < 3; c++) A.T[c][p] += A.B[c][p];
    const R *Bx = A.B[0], *By = A.B[1], *Bz = A.B[2];
    // Ey: Bx(o) += cz (Ey[o+1] - Ey[o]); Bz(o) -= cx (Ey[o+sx] - Ey[o])
    R ley = 0, lez = 0, lex = 0;
    if (phys(g, i, j, k - 1)) ley += cz * Bx[p - 1];
    if (here) ley += -cz * Bx[p] + cx * Bz[p];
    if (phys(g, i - 1, j, k)) ley += -cx * Bz[p - sx];
    // Ez: Bx(o) -= cy (Ez[o+sy] - Ez[o]); By(o) += cx (Ez[o+sx] - Ez[o])
    if (phys(g, i, j - 1, k)) lez += -cy * Bx[p - sy];
    if (here) lez += cy * Bx[p] - cx * By[p];
    if (phys(g, i - 1, j, k)) lez += cx * By[p - sx];
    // Ex: By(o) -= cz (Ex[o+1] - Ex[o]); Bz(o) += cy (Ex[o+sy] - Ex[o])
    if (phys(g, i, j, k - 1)) lex += -cz * By[p - 1];
    if (here) lex += cz * By[p] - cy * Bz[p];
    if (phys(g, i, j - 1, k)) lex += cy * Bz[p - sy];
    A.E[0][p] += lex;
    A.E[1][p] += ley;
    A.E[2][p] += lez;
}

// Adjoint of the E update (E -= dt (curl T + 4 pi J) over the physical
// points): LJ = -4 pi dt LE (physical, 0 elsewhere), LT += transposed curl;
// the B role was overwritten by the step, so its physical points' adjoint is
// cleared.
template <class R>
__global__ void k_yee_e_adj(Geom g, YeeCoef<R> yc, FOutT<R> A, JPtrsT<R> LJ) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= g.tot[2] || j >= g.tot[1] || i >= g.tot[0]) return;
    const int64_t p = gidx(g, i, j, k), sx = g.sx, sy = g.sy;
    const R cx = yc.cx, cy = yc.cy, cz = yc.cz, cj = yc.cj;
    const bool here = phys(g, i, j, k);
    const R *Ex = A.E[0], *Ey = A.E[1], *Ez = A.E[2];
    for (int c = 0; c < 3; c++) LJ.J[c][p] = here ? cj * A.E[c][p] : (R)0;
    R lty = 0, ltz = 0, ltx = 0;
    // Ty: ex(o) -= cz (Ty[o] - Ty[o-1]); ez(o) += cx (Ty[o] - Ty[o-sx])
    if (here) lty += -cz * Ex[p] + cx * Ez[p];
    if (phys(g, i, j, k + 1)) lty += cz * Ex[p + 1];
    if (phys(g, i + 1, j, k)) lty += -cx * Ez[p + sx];
    // Tz: ex(o) += cy (Tz[o] - Tz[o-sy]); ey(o) -= cx (Tz[o] - Tz[o-sx])
    if (here) ltz += cy * Ex[p] - cx * Ey[p];
    if (phys(g, i, j + 1, k)) ltz += -cy * Ex[p + sy];
    if (phys(g, i + 1, j, k)) ltz += cx * Ey[p + sx];
    // Tx: ey(o) += cz (Tx[o] - Tx[o-1]); ez(o) -= cy (Tx[o] - Tx[o-sy])
    if (here) ltx += cz * Ey[p] - cy * Ez[p];
    if (phys(g, i, j, k + 1)) ltx += -cz * Ey[p + 1];
    if (phys(g, i, j + 1, k)) ltx += cy * Ez[p + sy];
    A.T[0][p] += ltx;
    A.T[1][p] += lty;
    A.T[2][p] += ltz;
    if (here)
        for (int c = 0; c < 3; c++) A.B[c][p] = (R)0;
}

// Adjoint of the fold (F[plane 1] += F[plane n+1], transverse physical
// range, the two transverse J components): LF[n+1] += LF[1].
template <class R>
__global__ void k_fold_adj(Geom g, int d, R *f0, R *f1) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int r = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (q > g.n[o2] || r > g.n[o1]) return;
    int is[3], it[3];
    is[d] = g.n[d] + 1;
    it[d] = 1;
    is[o1] = it[o1] = r;
    is[o2] = it[o2] = q;
    const int64_t s = gidx(g, is[0], is[1], is[2]), t = gidx(g, it[0], it[1], it[2]);
    R *F = blockIdx.z == 0 ? f0 : f1;
    F[s] += F[t];
}

// Adjoint of one side of the ghost copy (ghost plane <- physical plane,
// transverse physical range): LF[src] += LF[dst], LF[dst] = 0.
template <class R>
__global__ void k_ghost_adj(Geom g, Slots6T<R> fl, int d, int side) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int r = blockIdx.y * blockDim.y + threadIdx.y + 1;
    if (q > g.n[o2] || r > g.n[o1]) return;
    const int nd = g.n[d];
    const int src = side == 0 ? nd : 1, dst = side == 0 ? 0 : nd + 1;
    int is[3], it[3];
    is[d] = src;
    it[d] = dst;
    is[o1] = it[o1] = r;
    is[o2] = it[o2] = q;
    R *F = fl.p[blockIdx.z];
    const int64_t ps = gidx(g, is[0], is[1], is[2]), pd = gidx(g, it[0], it[1], it[2]);
    F[ps] += F[pd];
    F[pd] = (R)0;
}

// ---- corrected policy ------------------------------------------------------
//
// Adjoint of the whole-range periodic fold along d (f[n] += f[0], f[1] +=
// f[n+1], f[2] += f[n+2]), per transverse point of the (n+3)^2 plane, the
// forward steps reversed (so any n is exact). One field per blockIdx.z.
template <class R>
__global__ void k_periodic_full_adj(Geom g, Slots9T<R> fl, int d) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (q >= g.tot[o2] || r >= g.tot[o1]) return;
    R *F = fl.p[blockIdx.z];
    const int n = g.n[d];
    int c[3];
    c[o1] = r;
    c[o2] = q;
    auto at = [&](int i) -> R & {
        c[d] = i;
        return F[gidx(g, c[0], c[1], c[2])];
    };
    at(n + 2) += at(2);
    at(n + 1) += at(1);
    at(0) += at(n);
}

struct WrapDims {
    int w[3];
};

// Adjoint of the whole-range ghost copies of the fields: each point with images
// takes in their adjoints and clears them; blockIdx.y = field. 32^3 cells, nine
// fields: 4.0 us (26 us with a thread a point of the grid for all fields).
template <class R>
__global__ void k_copy_images_adj(Geom g, Slots9T<R> fl, WrapDims w, Slabs S) {
    after_previous();
    int d, c[3];
    if (!slab_point(S, blockIdx.x * blockDim.x + threadIdx.x, d, c)) return;
    unsigned m[3];  // images along each dimension: bit 0 the point itself, 1, 2, 3 index 0, n + 1, n + 2
    bool one = true;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        const int n = g.n[e];
        m[e] = 1u;
        if (!w.w[e]) continue;
        // listed: 1, 2, n; the rest of a periodic dimension: 3 .. n - 1
        if (e < d) c[e] += 3;
        else if (e == d) c[e] = c[e] < 2 ? c[e] + 1 : n;
        else c[e] += 1;
        m[e] |= (c[e] == n ? 2u : 0u) | (c[e] == 1 ? 4u : 0u) | (c[e] == 2 || n == 1 ? 8u : 0u);
        one = one && n >= 3;
    }
    auto index = [&](int e, int b) { return b == 0 ? c[e] : b == 1 ? 0 : g.n[e] + b - 1; };
    R *F = fl.p[blockIdx.y];
    R v = (R)0;
    if (one) {  // at most one image along each dimension: all loads at once
        int at[3][2];
        bool has[3][2];
#pragma unroll
        for (int e = 0; e < 3; e++) {
            at[e][0] = c[e];
            at[e][1] = m[e] > 1u ? index(e, 31 - __clz(m[e])) : c[e];
            has[e][0] = true;
            has[e][1] = m[e] > 1u;
        }
        R x[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int i = q >> 2, j = (q >> 1) & 1, k = q & 1;
            if (has[0][i] && has[1][j] && has[2][k]) x[q] = F[gidx(g, at[0][i], at[1][j], at[2][k])];
        }
        v = x[0];
#pragma unroll
        for (int q = 1; q < 8; q++) {
            const int i = q >> 2, j = (q >> 1) & 1, k = q & 1;
            if (has[0][i] && has[1][j] && has[2][k]) {
                v += x[q];
                F[gidx(g, at[0][i], at[1][j], at[2][k])] = (R)0;
            }
        }
    } else {
        for (unsigned x = m[0]; x; x &= x - 1)
            for (unsigned y = m[1]; y; y &= y - 1)
                for (unsigned z = m[2]; z; z &= z - 1) {
                    R *p = F + gidx(g, index(0, __ffs(x) - 1), index(1, __ffs(y) - 1), index(2, __ffs(z) - 1));
                    v += *p;
                    *p = (R)0;
                }
    }
    F[gidx(g, c[0], c[1], c[2])] = v;
}

// Adjoint of the mirror fold at a reflecting wall (dst += s src, src = 0, s =
// -1 for the component normal to the wall): L[src] = s L[dst]. Same launch
// shape as the forward; blockIdx.z = component.
template <class R>
__global__ void k_mirror_fold_adj(Geom g, Slots9T<R> fl, int d, int right) {
    after_previous();
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (q >= g.tot[o2] || r >= g.tot[o1]) return;
    const int a = blockIdx.z;
    R *F = fl.p[a];
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
    F[ks] = normal ? -F[kd] : F[kd];
}

// Clears three arrays at the physical points (the adjoint of values a step
// overwrites there).
template <class R>
__global__ void k_clear_phys(Geom g, Slots9T<R> fl) {
    after_previous();
    const int k = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int i = blockIdx.z + 1;
    if (k > g.n[2] || j > g.n[1]) return;
    const int64_t p = gidx(g, i, j, k);
    for (int c = 0; c < 3; c++) fl.p[c][p] = (R)0;
}

// Adjoint of a plane set v + vs t1[p] t2[q]: the plane's values depend only
// on the wave parameters, so the step needs sum(LF) and sum(LF t1 t2) over
// the plane; the host turns them into the parameter gradient. Block b of the
// PLANE_BLOCKS launched writes its partial pair to sums2[2 b], sums2[2 b + 1]
// (FP64, fixed order within the block; the host adds the blocks in order).
// The plane's adjoint is cleared.
constexpr int PLANE_BLOCKS = 64;

// A launch takes the planes of up to 12 sets (blockIdx.y), none of which
// share a point; entry e's partials follow entry e - 1's.
template <class R>
struct PlaneAdjList {
    R *f[12];
    int idx[12];
    const double *t1[12], *t2[12];
    int dim, n;
};

template <class R>
__global__ void k_plane_adj(Geom g, PlaneAdjList<R> pl, double *sums) {
    after_previous();
    __shared__ double s_u[32], s_s[32];
    const int entry = blockIdx.y, d = pl.dim, idx = pl.idx[entry];
    R *F = pl.f[entry];
    const double *t1 = pl.t1[entry], *t2 = pl.t2[entry];
    double *sums2 = sums + 2 * (size_t)PLANE_BLOCKS * entry;
    const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
    double su = 0.0, ss = 0.0;
    const int64_t m = (int64_t)g.tot[o1] * g.tot[o2];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
        int c[3];
        c[d] = idx;
        c[o1] = (int)(t / g.tot[o2]);
        c[o2] = (int)(t % g.tot[o2]);
        const int64_t p = gidx(g, c[0], c[1], c[2]);
        const double l = (double)F[p];
        su += l;
        if (t1) ss += l * t1[c[o1]] * t2[c[o2]];
        F[p] = (R)0;
    }
    for (int off = 16; off > 0; off >>= 1) {
        su += __shfl_down_sync(0xffffffffu, su, off);
        ss += __shfl_down_sync(0xffffffffu, ss, off);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_u[w] = su;
        s_s[w] = ss;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
            a += s_u[i];
            b += s_s[i];
        }
        sums2[2 * blockIdx.x] = a;
        sums2[2 * blockIdx.x + 1] = b;
    }
}

// The plane sets met by the adjoint steps, in reverse order, with the device
// sums (sum LF, sum LF t1 t2) each one left in `sums`; the wave parameter
// gradient is formed from them on the host at the end.
struct PlaneLedger {
    std::vector<AdBcOp> ops;
    double *sums = nullptr;
    size_t cap = 0;
};

// Adjoints of the plane sets among ops [first, last), last first, each
// recorded in the ledger; one launch for those of a dimension, whose planes
// are disjoint (unless it has one cell: both sides set the same plane).
template <class R>
int planes_adj(emoo_handle *h, const std::vector<AdBcOp> &ops, size_t first, size_t last, R *const *lslot,
               PlaneLedger &pl) {
    PlaneAdjList<R> list = {};
    size_t start = pl.ops.size();
    auto flush = [&]() -> int {
        if (!list.n) return EMOO_OK;
        h->launches++;
        launch_after(k_plane_adj<R>, dim3(PLANE_BLOCKS, list.n), 256, 0, h->stream)(h->g, list,
                                                                          pl.sums + 2 * (size_t)PLANE_BLOCKS * start);
        EMOO_CUDA(cudaGetLastError());
        list.n = 0;
        start = pl.ops.size();
        return EMOO_OK;
    };
    for (size_t i = last; i-- > first;) {
        const AdBcOp &op = ops[i];
        if (op.kind != 1) continue;
        if (pl.ops.size() >= pl.cap) return EMOO_ERR_STATE;
        bool apart = list.n < 12 && (!list.n || op.dim == list.dim);
        for (int e = 0; e < list.n; e++) apart = apart && !(list.f[e] == lslot[op.slot] && list.idx[e] == op.idx);
        if (!apart) EMOO_TRY(flush());
        list.dim = op.dim;
        list.f[list.n] = lslot[op.slot];
        list.idx[list.n] = op.idx;
        list.t1[list.n] = op.t1;
        list.t2[list.n] = op.t2;
        list.n++;
        pl.ops.push_back(op);
    }
    return flush();
}

// Adjoint of the corrected policy's whole-range folds (J with its mirror folds
// at reflecting walls), dimensions and sides reversed.
template <class R>
int periodic_fold_adj(emoo_handle *h, R *const *lslot, const int *ids, int nids) {
    const Geom &g = h->g;
    Slots9T<R> fl{};
    for (int k = 0; k < nids; k++) fl.p[k] = lslot[ids[k]];
    dim3 blk(32, 8);
    for (int d = 2; d >= 0; d--) {
        const int o1 = (d == 0) ? 1 : 0, o2 = (d == 2) ? 1 : 2;
        if (h->bc.fbc[2 * d] != FBC_PERIODIC) {
            for (int r = 1; r >= 0; r--) {
                if (h->bc.pbc[2 * d + r] != PBC_REFLECTING) continue;
                dim3 grd((g.tot[o2] + 31) / 32, (g.tot[o1] + 7) / 8, 3);
                h->launches++;
                launch_after(k_mirror_fold_adj<R>, grd, blk, 0, h->stream)(g, fl, d, r);
            }
            continue;
        }
        dim3 grd((g.tot[o2] + 31) / 32, (g.tot[o1] + 7) / 8, nids);
        h->launches++;
        launch_after(k_periodic_full_adj<R>, grd, blk, 0, h->stream)(g, fl, d);
    }
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

// Adjoint of the corrected policy's ghost copies.
template <class R>
int copy_images_adj(emoo_handle *h, R *const *lslot, const int *ids, int nids) {
    Slots9T<R> fl{};
    WrapDims w;
    for (int k = 0; k < nids; k++) fl.p[k] = lslot[ids[k]];
    for (int d = 0; d < 3; d++) w.w[d] = h->bc.fbc[2 * d] == FBC_PERIODIC;
    Slabs S;  // the points with images
    for (int d = 0; d < 3; d++) {
        S.listed[d] = w.w[d] ? std::min(3, h->g.n[d]) : 0;
        S.rest[d] = (w.w[d] ? h->g.n[d] : h->g.tot[d]) - S.listed[d];
    }
    const int64_t points = slab_size(S);
    if (!points) return EMOO_OK;
    h->launches++;
    launch_after(k_copy_images_adj<R>, dim3((unsigned)((points + 127) / 128), nids), 128, 0, h->stream)(h->g, fl, w, S);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

}  // namespace adf
}  // namespace emoo
