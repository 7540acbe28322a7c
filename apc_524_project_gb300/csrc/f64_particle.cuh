// f64_particle.cuh - one particle's FP64 step, shared by the time loop
// (particles_f64.cu) and its differentiation (adjoint_f64.cu): cell and vertex,
// field gather, Boris and Vay pushes. The arithmetic is on Rn, whose operations
// are separately rounded however the translation unit is compiled, in the
// reference's order, so both give the same words.
#ifndef EMOO_F64_PARTICLE_CUH
#define EMOO_F64_PARTICLE_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "dev_common.cuh"
#include "emoo_internal.h"
#include "f64_ops.cuh"

namespace emoo {

struct Rn {
    double v;
    __device__ __forceinline__ Rn() {}
    __device__ __forceinline__ Rn(double x) : v(x) {}
};
__device__ __forceinline__ Rn operator+(Rn a, Rn b) { return __dadd_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator-(Rn a, Rn b) { return __dsub_rn(a.v, b.v); }
__device__ __forceinline__ Rn operator*(Rn a, Rn b) { return __dmul_rn(a.v, b.v); }
// a * b + c rounded once, where a * b is exact (a power of two times b): the
// value of the separate operations
__device__ __forceinline__ Rn exact_fma(double a, Rn b, Rn c) { return __fma_rn(a, b.v, c.v); }
// a sum as it comes out when it starts with 0: a zero is +0
__device__ __forceinline__ Rn sum_from_zero(Rn a) {
    return __hiloint2double(f64_zero(a.v) ? 0 : __double2hiint(a.v), __double2loint(a.v));
}
// x / d (ddiv): the exact reciprocal where d is a power of two
__device__ __forceinline__ Rn div_by(Rn a, double d, double id, int p2) { return p2 ? __dmul_rn(a.v, id) : __ddiv_rn(a.v, d); }

struct GatherPtrs {
    const double *E[3];
    const double *B[3];  // current B role
    const double *T[3];  // B_tm1 role
};

// What a kernel's instance may take for granted: unit cells at the origin,
// and with them a time step that is a power of two.
enum { ANY = 0, UNIT_CELLS = 1, UNIT_DT2 = 2 };

// Removed particles carry a NaN position.
__device__ __forceinline__ bool alive(double x) { return f64_not_nan(x); }

// A position's cell index (dev_common's cell_of, getCellID's truncation) on
// each axis, and the position relative to the cell's vertex x0 + d (i -
// vshift). UNIT: unit cells at the origin.
template <bool UNIT>
__device__ __forceinline__ void locate(const Geom &g, const double p[3], int c[3]) {
#pragma unroll
    for (int a = 0; a < 3; a++) c[a] = f64_trunc(UNIT ? p[a] : ((Rn(p[a]) - g.x0[a]) * g.id[a]).v) + 1;
}

template <bool UNIT>
__device__ __forceinline__ void from_vertex(const Geom &g, const int c[3], const double p[3], double ds[3]) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const Rn i = f64_of_int(c[a] - g.vshift);
        ds[a] = (Rn(p[a]) - (UNIT ? i : Rn(g.x0[a]) + Rn(g.d[a]) * i)).v;
    }
}

// Grid::getFieldInterpolatorVec (src/grid/oGrid.cpp:153-197) and
// Interpolator::interpolate_fields (src/particles/interpolate.cpp:11-47) for a
// particle in the cell at grid point o, ds from its vertex. e: the electric
// field; b2: twice the magnetic field (the halves of the averages of B and
// B_tm1 are exact, so the pushers take them where they cost nothing). E12,
// S6: the values read, 4 a component and B + B_tm1 at the two faces.
template <bool UNIT>
__device__ __forceinline__ void gather_cell(const Geom &g, const GatherPtrs &P, int64_t o, const double ds[3],
                                            double e[3], double b2[3], double E12[12], double S6[6]) {
    const int64_t st[3] = {g.sx, g.sy, 1};
    Rn r[3], w[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        r[i] = ds[i];
        w[i] = Rn(UNIT ? 1.0 : g.d[i]) - r[i];
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        const double *E = P.E[i] + o, *B = P.B[i] + o, *T = P.T[i] + o;
        double *v = E12 + 4 * i, *S = S6 + 2 * i;
        v[0] = E[0], v[1] = E[st[j]], v[2] = E[st[j] + st[k]], v[3] = E[st[k]];
        S[0] = (Rn(T[0]) + B[0]).v;
        S[1] = (Rn(T[st[i]]) + B[st[i]]).v;
        const Rn s = sum_from_zero(w[j] * w[k] * v[0] + r[j] * w[k] * v[1] + r[j] * r[k] * v[2] + w[j] * r[k] * v[3]);
        const Rn b = sum_from_zero(w[i] * S[0] + r[i] * S[1]);
        e[i] = UNIT ? s.v : div_by(s, g.area[i], g.iarea[i], g.area_p2[i]).v;
        b2[i] = UNIT ? b.v : div_by(b, g.d[i], g.id[i], g.p2[i]).v;
    }
}

// x + dt v; with dt a power of two the product is exact and one fused
// instruction gives the same sum.
template <int MODE>
__device__ __forceinline__ double advance(double x, double dt, Rn v) {
    return MODE == UNIT_DT2 ? exact_fma(dt, v, x).v : (Rn(x) + Rn(dt) * v).v;
}

// Boris::Step, src/pusher/boris.cpp:33-85 (q_p precomputed per species, hq
// half of it), on e and b2 = 2 B: hq b2 = q_p B, and 2 / (1 + q_p q_p B^2)
// from the same scaled words.
template <int MODE>
__device__ __forceinline__ void boris_push(double q_p, double hq, const double e[3], const double b2[3], double dt,
                                           double p[3], double v[3]) {
    const Rn qp = q_p, h = hq, bx = b2[0], by = b2[1], bz = b2[2];
    const Rn tx = h * bx, ty = h * by, tz = h * bz;
    const Rn bsqr4 = bx * bx + by * by + bz * bz;
    const Rn tsqr = __ddiv_rn(2.0, (Rn(1.0) + h * h * bsqr4).v);
    const Rn sx = tsqr * tx, sy = tsqr * ty, sz = tsqr * tz;
    const Rn qex = qp * e[0], qey = qp * e[1], qez = qp * e[2];
    const Rn v_mx = Rn(v[0]) + qex, v_my = Rn(v[1]) + qey, v_mz = Rn(v[2]) + qez;
    const Rn v_ix = v_mx + v_my * tz - v_mz * ty;
    const Rn v_iy = v_my + v_mz * tx - v_mx * tz;
    const Rn v_iz = v_mz + v_mx * ty - v_my * tx;
    const Rn v_px = v_mx + v_iy * sz - v_iz * sy;
    const Rn v_py = v_my + v_iz * sx - v_ix * sz;
    const Rn v_pz = v_mz + v_ix * sy - v_iy * sx;
    v[0] = (v_px + qex).v;
    v[1] = (v_py + qey).v;
    v[2] = (v_pz + qez).v;
#pragma unroll
    for (int a = 0; a < 3; a++) p[a] = advance<MODE>(p[a], dt, v[a]);
}

// The intermediates of one Vay push, for its reverse (ad::VayTape).
struct VayStep {
    double up[3], tau[3], tsq, sigma, ustar, gi1, igi, tt[3], s, udott, w[3];
};

// The part of the Vay push with quotients by gamma, from u', tau and u*.
struct VayTurn {
    double t[3], s, udott, w[3], sw[3], v[3];
};

template <class Quot>
__device__ __forceinline__ void vay_turn(const double up[3], const double tau[3], double ustar, Quot by_gamma,
                                         VayTurn &n) {
    const Rn upx = up[0], upy = up[1], upz = up[2];
    const Rn tx = by_gamma(tau[0]), ty = by_gamma(tau[1]), tz = by_gamma(tau[2]);
    const Rn s = __drcp_rn((Rn(1.0) + tx * tx + ty * ty + tz * tz).v);
    const Rn udott = by_gamma(ustar);
    const Rn wx = upx + udott * tx + (upy * tz - upz * ty);
    const Rn wy = upy + udott * ty + (upz * tx - upx * tz);
    const Rn wz = upz + udott * tz + (upx * ty - upy * tx);
    n.t[0] = tx.v, n.t[1] = ty.v, n.t[2] = tz.v;
    n.s = s.v, n.udott = udott.v;
    n.w[0] = wx.v, n.w[1] = wy.v, n.w[2] = wz.v;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        n.sw[a] = (s * n.w[a]).v;
        n.v[a] = by_gamma(n.sw[a]);
    }
}

// the same with divisions, for what f64_quot does not take
static __device__ __noinline__ void vay_turn_divided(const double (&up)[3], const double (&tau)[3], double ustar,
                                                     double gamma, VayTurn &n) {
    vay_turn(up, tau, ustar, [&](double a) { return __ddiv_rn(a, gamma); }, n);
}

// Relativistic_Boris::Step (Vay), src/pusher/relativisticBoris.cpp:53-140, on
// e and b2 = 2 B: hq b2 = q_p B; e + v x B as one fused instruction with the
// exact half of v x b2; sigma^2 + 4 (..) likewise. (Exact where no product of a
// field is denormal: below, the last bit of a denormal may differ.)
template <int MODE>
__device__ __forceinline__ void vay_push(double q_p, double hq, const double e[3], const double b2[3], double dt,
                                         double p[3], double v[3], double &gamma, VayStep &T) {
    const Rn qp = q_p, h = hq, bx = b2[0], by = b2[1], bz = b2[2], vx = v[0], vy = v[1], vz = v[2], ga = gamma;
    const Rn vXbx = vy * bz - vz * by, vXby = vz * bx - vx * bz, vXbz = vx * by - vy * bx;
    const Rn uhx = ga * vx + qp * exact_fma(0.5, vXbx, e[0]);
    const Rn uhy = ga * vy + qp * exact_fma(0.5, vXby, e[1]);
    const Rn uhz = ga * vz + qp * exact_fma(0.5, vXbz, e[2]);
    const Rn upx = uhx + qp * e[0], upy = uhy + qp * e[1], upz = uhz + qp * e[2];
    const Rn gammap_sq = Rn(1.0) + upx * upx + upy * upy + upz * upz;
    const Rn taux = h * bx, tauy = h * by, tauz = h * bz;
    const Rn tau_sq = taux * taux + tauy * tauy + tauz * tauz;
    const Rn sigma = gammap_sq - tau_sq;
    const Rn ustar = upx * taux + upy * tauy + upz * tauz;
    const Rn gi1 = sqrt(exact_fma(4.0, tau_sq + ustar * ustar, sigma * sigma).v);
    const double gi = sqrt(f64_half((sigma + gi1).v));
    const F64Quot dg = f64_divisor(gi);
    const double up[3] = {upx.v, upy.v, upz.v}, tau[3] = {taux.v, tauy.v, tauz.v};
    VayTurn n;
    vay_turn(up, tau, ustar.v, [&](double a) { return f64_quot(a, dg); }, n);
    // tested last, all at once: 0.8 % of a gradient (1.6 % with a branch before
    // each group of quotients)
    bool fit = dg.ordinary && f64_fit(ustar.v);
#pragma unroll
    for (int a = 0; a < 3; a++) fit = fit && f64_fit(tau[a]) && f64_fit(n.sw[a]);
    if (!fit) vay_turn_divided(up, tau, ustar.v, gi, n);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        v[a] = n.v[a];
        p[a] = advance<MODE>(p[a], dt, v[a]);
    }
    gamma = gi;
#pragma unroll
    for (int a = 0; a < 3; a++) T.up[a] = up[a], T.tau[a] = tau[a], T.tt[a] = n.t[a], T.w[a] = n.w[a];
    T.tsq = tau_sq.v, T.sigma = sigma.v, T.ustar = ustar.v, T.gi1 = gi1.v, T.igi = dg.y;
    T.s = n.s, T.udott = n.udott;
}

// Whether the straight move p0 -> p1 of a particle in cell c leaves the cell
// (or starts outside the box), by the ends' truncated positions.
template <bool UNIT>
__device__ __forceinline__ bool leaves_cell(const Geom &g, const int c[3], const double p0[3], const double p1[3],
                                            double u0[3], double u1[3]) {
    bool out = false;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        u0[a] = UNIT ? p0[a] : ((Rn(p0[a]) - g.x0[a]) * g.id[a]).v;
        u1[a] = UNIT ? p1[a] : ((Rn(p1[a]) - g.x0[a]) * g.id[a]).v;
        out = out || f64_sign(u0[a]) || f64_sign(u1[a]) || f64_trunc(u1[a]) + 1 != c[a];
    }
    return out;
}

// Whether apply_bc may find a side crossed, from integer comparisons: true
// for every crossing, and for a -0 against a wall at 0 or a NaN, where
// apply_bc then finds none.
__device__ __forceinline__ bool maybe_crossed(const BCTab &bc, const double p[3]) {
    bool hit = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const long long k = f64_key(p[d]);
        hit = hit || k < f64_key(bc.xmin[d]) || k > f64_key(bc.xmax[d]);
    }
    return hit;
}

}  // namespace emoo

#endif
