// particles_f64.cu - FP64 particle kernels: field gather, Boris / relativistic
// Boris push, particle boundaries, current and charge deposition, and the
// fused gather + push + boundary + deposit kernel of the time loop.
//
// Compiled with --fmad=false and written in the reference's order of
// operations, so each particle's interpolated field, pushed state and
// deposited contributions are bit-identical to the reference serial build on
// the same inputs. Only the order in which contributions of different
// particles are summed differs: consecutive particles of a warp that share a
// cell are summed in a fixed order, then added with FP64 atomics.
//
// These kernels are bound by the FP64 pipe (two lanes per clock per SM), so
// the arithmetic is arranged for few FP64 instructions without changing a
// result: cell indices, tests and halvings run as integer instructions
// (f64_ops.cuh), an exact product by a power of two joins the addition that
// follows it in one fused instruction, the seven quotients by gamma share one
// reciprocal, and grids of unit cells at the origin (UNIT) skip the divisions
// and products by 1.
#include <cuda_runtime.h>
#include <stddef.h>

#include <algorithm>
#include <vector>

#include "dev_common.cuh"
#include "emoo_internal.h"
#include "f64_particle.cuh"

namespace emoo {

double *role_b(emoo_handle *h, int c);
double *role_t(emoo_handle *h, int c);

namespace {

struct DepositPtrs {
    double *J[3];
    double *rho;
};

struct PState {
    double *x, *y, *z, *vx, *vy, *vz, *g;
};

// The six particle boundaries applied to one particle in the reference's
// side order (src/particles/particle_handler.cpp:287-295). A periodic side's
// ghost copy (src/boundaries/b_particles/bc_p_periodic.cpp:52-87) becomes an
// in-place wrap that later sides see, as they see the copy; reflecting folds
// position and velocity (src/boundaries/b_particles/bc_p_reflecting.cpp:43-52);
// absorbing removes the particle. Returns the crossed-side bit mask; bit 6
// set means removed.
__device__ __forceinline__ int apply_bc(const BCTab &bc, double p[3], double v[3]) {
    int mask = 0;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        const int d = s >> 1;
        const bool right = s & 1;
        double xmin = bc.xmin[d], xmax = bc.xmax[d];
        bool hit = right ? (p[d] > xmax) : (p[d] < xmin);
        if (!hit) continue;
        mask |= 1 << s;
        int kind = bc.pbc[s];
        if (kind == PBC_PERIODIC) {
            if (right) p[d] -= (xmax - xmin);
            else p[d] += (xmax - xmin);
        } else if (kind == PBC_REFLECTING) {
            p[d] = right ? 2.0 * xmax - p[d] : 2.0 * xmin - p[d];
            v[d] = -v[d];
        } else {
            mask |= 1 << 6;
            break;
        }
    }
    return mask;
}

// Depositor::deposit_particle_J (src/particles/deposit.cpp:12-39) for one
// particle at offsets r from its cell's vertex: the 12 edge contributions in
// the reference's order of operations.
template <bool UNIT>
__device__ __forceinline__ void deposit_terms_j(const Geom &g, double uq, const double r[3], const double v[3],
                                                double c[12]) {
    double w[3];
#pragma unroll
    for (int i = 0; i < 3; i++) w[i] = (UNIT ? 1.0 : g.d[i]) - r[i];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int j = (i + 1) % 3, k = (i + 2) % 3;
        double ratio = uq * v[i];
        if (!UNIT) ratio = ddiv(ddiv(ratio, g.vol, g.ivol, g.vol_p2), g.area[i], g.iarea[i], g.area_p2[i]);
        const double rw = ratio * w[j], rr = ratio * r[j];
        c[4 * i] = rw * w[k];
        c[4 * i + 1] = rr * w[k];
        c[4 * i + 2] = rr * r[k];
        c[4 * i + 3] = rw * r[k];
    }
}

// Depositor::deposit_particle_Rho (src/particles/deposit.cpp:42-62): the 8
// vertex contributions.
__device__ __forceinline__ void deposit_terms_rho(const Geom &g, double cr, const double r[3], double c[8]) {
    double l[3];
#pragma unroll
    for (int i = 0; i < 3; i++) l[i] = g.d[i] - r[i];
    c[0] = cr * l[0] * l[1] * l[2];
    c[1] = cr * r[0] * l[1] * l[2];
    c[2] = cr * r[0] * r[1] * l[2];
    c[3] = cr * l[0] * r[1] * l[2];
    c[4] = cr * l[0] * r[1] * r[2];
    c[5] = cr * r[0] * r[1] * r[2];
    c[6] = cr * r[0] * l[1] * r[2];
    c[7] = cr * l[0] * l[1] * r[2];
}

// Grid point of contribution q of cell o (Grid::addJ with its Jx index as in
// src/grid/oGrid.cpp:98-111, Grid::addRho src/grid/oGrid.cpp:129-136).
__device__ __forceinline__ int64_t deposit_point(const Geom &g, int64_t o, int q) {
    const int64_t sx = g.sx, sy = g.sy;
    switch (q) {
        case 0: return o;
        case 1: return o + sy;
        case 2: return o + sy + 1;
        case 3: return g.vshift ? o + 1 : o + sy;  // reference: Jx[ix][iy+1][iz] (src/grid/oGrid.cpp:101)
        case 4: return o;
        case 5: return o + 1;
        case 6: return o + sx + 1;
        case 7: return o + sx;
        case 8: return o;
        case 9: return o + sx;
        case 10: return o + sx + sy;
        case 11: return o + sy;
        case 12: return o;
        case 13: return o + sx;
        case 14: return o + sx + sy;
        case 15: return o + sy;
        case 16: return o + sy + 1;
        case 17: return o + sx + sy + 1;
        case 18: return o + sx + 1;
        default: return o + 1;
    }
}

// Warp-cooperative commit of NQ contributions a particle (the 12 of J, or
// the 8 of rho, contribution Q0 + q of deposit_point): each lane writes its
// particle's as a column of the warp's shared tile; lane (q, half) then walks
// row q over its half of the particles, in pairs, and adds each run of equal
// cells to the grid with one atomic; the parts of a run that spans both halves
// are joined first. A warp of particles all in cells of their own commits from
// registers. Summing by rows takes some 17 FP64 additions a warp (a shuffle tree
// per contribution took 60 for J). Pairs and joined halves because of the
// rounding: the root mean square error of a grid value is then the trees' (J:
// 1.08 of it with 16 particles a cell, 0.96 with 61; rho 1.03, 0.97). Summed one
// after the other, with an atomic for each half, J's was 1.20 and 1.16 of it; the
// step then took 0.6 % less.
constexpr int PART_BLOCK = 256;
constexpr int FUSED_BLOCK = 128;  // k_fused, k_fused_vb (see launch_fused)
constexpr int ROW = 34;  // doubles: rows on 16-byte boundaries, 16-byte reads of 8 rows without bank conflicts

struct alignas(16) CommitTile {
    double w[12 * ROW];
    int key[32];
};
// a row's parts are read as double2, in every tile of an array of them
static_assert(alignof(CommitTile) % sizeof(double2) == 0 && offsetof(CommitTile, w) % sizeof(double2) == 0 &&
                  sizeof(CommitTile) % sizeof(double2) == 0 && ROW * sizeof(double) % sizeof(double2) == 0,
              "16-byte reads of a tile's rows");

template <int NQ, int Q0>
__device__ __forceinline__ void commit_deposit(const Geom &g, const DepositPtrs &D, CommitTile &tile, bool active,
                                               int64_t cell_o, const double c[NQ]) {
    static_assert(NQ == 12 || NQ == 8, "J or rho");
    const int lane = threadIdx.x & 31;
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (act == 0u) return;
    const int key = active ? (int)cell_o : -1 - lane;  // (21 FP64 arrays of 2^31 points fit no device)
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != key);
    auto target = [&](int q) {
        double *base = Q0 == 12 ? D.rho : (q < 4 ? D.J[0] : q < 8 ? D.J[1] : D.J[2]);
        return base + deposit_point(g, 0, Q0 + q);
    };
    if (heads == 0xffffffffu) {
        if (active) {
#pragma unroll
            for (int q = 0; q < NQ; q++) atomicAdd(target(q) + cell_o, c[q]);
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < NQ; q++) tile.w[q * ROW + lane] = active ? c[q] : 0.0;
    tile.key[lane] = key;
    __syncwarp();
    const int q = lane & 15, half = lane >> 4;
    double *dst = target(q < NQ ? q : 0);
    const int *keys = tile.key + 16 * half;
    const unsigned ends = (((heads >> 1) | 0x80000000u) & act) >> (16 * half);  // of active runs
    // a run that spans particles 15 and 16: its first part is what half 0 has
    // left, its last the first total of half 1
    const bool spans = !((heads >> 16) & 1u);
    const unsigned joined = spans && half ? ends & (0u - ends) : 0u;
    double acc = 0.0, last = 0.0;
    if (q < NQ) {
        const double2 *row = reinterpret_cast<const double2 *>(tile.w + q * ROW + 16 * half);
        auto commit = [&](int i, double total) {
            if ((joined >> i) & 1u) last = total;
            else atomicAdd(dst + keys[i], total);
        };
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const double2 v = row[i / 2];
            if ((ends >> i) & 1u) {
                commit(i, acc + v.x);
                acc = v.y;
            } else {
                acc += v.x + v.y;
            }
            if ((ends >> (i + 1)) & 1u) {
                commit(i + 1, acc);
                acc = 0.0;
            }
        }
    }
    if (spans) {
        const double first = __shfl_sync(0xffffffffu, acc, q);
        if (half && q < NQ) atomicAdd(dst + keys[__ffs((int)joined) - 1], first + last);
    }
    __syncwarp();
}

__device__ __forceinline__ void count_crossings(DevCounters *ctr, int mask) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        unsigned b = __ballot_sync(0xffffffffu, (mask >> s) & 1);
        if (lane == 0 && b) atomicAdd(&ctr->cross[s], (unsigned long long)__popc(b));
    }
}

// emoo_interpolate: per-particle field cache (Particle::field).
__global__ void k_interpolate(Geom g, GatherPtrs P, PState S, int64_t np, int64_t cap, double *fc, DevCounters *ctr) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    const double pos[3] = {S.x[p], S.y[p], S.z[p]};
    if (!alive(pos[0])) return;
    int c[3];
    locate<false>(g, pos, c);
    if (!cell_ok(g, c[0], c[1], c[2])) {
        atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
        return;
    }
    double ds[3], e[3], b2[3], E12[12], S6[6];
    from_vertex<false>(g, c, pos, ds);
    gather_cell<false>(g, P, gidx(g, c[0], c[1], c[2]), ds, e, b2, E12, S6);
#pragma unroll
    for (int q = 0; q < 3; q++) {
        fc[q * cap + p] = e[q];
        fc[(3 + q) * cap + p] = 0.5 * b2[q];
    }
}

// emoo_push: Particle_Handler::Push with the cached fields.
__global__ void k_push_cached(SpeciesTab st, PState S, int64_t np, int64_t cap, const double *fc, double dt, int rel) {
    constexpr int MODE = ANY;
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    double pos[3] = {S.x[p], S.y[p], S.z[p]};
    if (!alive(pos[0])) return;
    int s = species_of(st, p);
    double e[3], b2[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        e[q] = fc[q * cap + p];
        b2[q] = 2.0 * fc[(3 + q) * cap + p];
    }
    double v[3] = {S.vx[p], S.vy[p], S.vz[p]};
    if (rel) {
        double ga = S.g[p];
        VayStep vt;
        vay_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v, ga, vt);
        S.g[p] = ga;
    } else {
        boris_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v);
    }
    S.x[p] = pos[0]; S.y[p] = pos[1]; S.z[p] = pos[2];
    S.vx[p] = v[0]; S.vy[p] = v[1]; S.vz[p] = v[2];
}

__global__ void k_particle_bc(BCTab bc, PState S, int64_t np, DevCounters *ctr) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int mask = 0;
    if (p < np) {
        double pos[3] = {S.x[p], S.y[p], S.z[p]};
        if (alive(pos[0])) {
            double v[3] = {S.vx[p], S.vy[p], S.vz[p]};
            mask = apply_bc(bc, pos, v);
            if (mask & 64) pos[0] = __longlong_as_double(0x7ff8000000000000LL);
            if (mask) {
                S.x[p] = pos[0]; S.y[p] = pos[1]; S.z[p] = pos[2];
                S.vx[p] = v[0]; S.vy[p] = v[1]; S.vz[p] = v[2];
            }
        }
    }
    count_crossings(ctr, mask);
}

// what: 0 J, 1 J and rho, 2 rho only
__global__ void __launch_bounds__(PART_BLOCK) k_deposit(Geom g, SpeciesTab st, PState S, int64_t np, DepositPtrs D,
                                                        int what, DevCounters *ctr) {
    after_previous<false>();
    __shared__ CommitTile tiles[PART_BLOCK / 32];
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    bool active = false;
    int64_t o = 0;
    int s = 0;
    double r[3] = {0.0, 0.0, 0.0};
    if (p < np) {
        const double pos[3] = {S.x[p], S.y[p], S.z[p]};
        s = species_of(st, p);
        if (alive(pos[0]) && st.deposit[s]) {
            int c[3];
            locate<false>(g, pos, c);
            if (cell_ok(g, c[0], c[1], c[2])) {
                active = true;
                o = gidx(g, c[0], c[1], c[2]);
                from_vertex<false>(g, c, pos, r);
            } else {
                atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
            }
        }
    }
    CommitTile &tile = tiles[threadIdx.x >> 5];
    if (what != 2) {
        double c[12];
        const double v[3] = {active ? S.vx[p] : 0.0, active ? S.vy[p] : 0.0, active ? S.vz[p] : 0.0};
        deposit_terms_j<false>(g, st.uq[s], r, v, c);
        commit_deposit<12, 0>(g, D, tile, active, o, c);
    }
    if (what != 0) {
        double c[8];
        deposit_terms_rho(g, st.cr[s], r, c);
        commit_deposit<8, 12>(g, D, tile, active, o, c);
    }
}

// Villasenor-Buneman current (J. Villasenor and O. Buneman, Comput. Phys.
// Commun. 69 (1992) 306) of a particle moving in a straight line from p0 to
// p1 (unwrapped, at most one cell face per axis), for the corrected policy:
// the path is split at the faces it crosses; a piece with offsets a -> b in a
// cell (cell units, m = (a + b) / 2, D = b - a) adds to the cell's four x
// edges coef dx Dx ((1-my)(1-mz) + Dy Dz / 12), (my (1-mz) - ..),
// ((1-my) mz - ..), (my mz + ..), and likewise for y and z; with the linear
// charge assignment, rho(t + dt) - rho(t) + dt div J = 0 at every point.
// coef = UNIT_RHOJ q / V / dt. Pieces outside the box land in the ghost
// planes, which the periodic fold adds back.
__device__ void vb_deposit(const Geom &g, const DepositPtrs &D, const double p0[3], const double p1[3], double coef) {
    double u0[3], u1[3], ts[5];
    int nt = 0;
    ts[nt++] = 0.0;
    for (int a = 0; a < 3; a++) {
        u0[a] = (p0[a] - g.x0[a]) * g.id[a];
        u1[a] = (p1[a] - g.x0[a]) * g.id[a];
        const double f0 = floor(u0[a]), f1 = floor(u1[a]);
        if (f0 != f1) {
            const double b = f0 > f1 ? f0 : f1;
            ts[nt++] = (b - u0[a]) / (u1[a] - u0[a]);
        }
    }
    ts[nt++] = 1.0;
    for (int i = 2; i < nt - 1; i++)
        for (int j = i; j > 1 && ts[j] < ts[j - 1]; j--) {
            const double t = ts[j];
            ts[j] = ts[j - 1];
            ts[j - 1] = t;
        }
    for (int sgi = 0; sgi + 1 < nt; sgi++) {
        const double ta = ts[sgi], tb = ts[sgi + 1];
        if (!(tb > ta)) continue;
        double m[3], Dd[3];
        int cell[3];
        for (int a = 0; a < 3; a++) {
            const double ua = u0[a] + ta * (u1[a] - u0[a]), ub = u0[a] + tb * (u1[a] - u0[a]);
            cell[a] = (int)floor(0.5 * (ua + ub));
            const double aa = ua - cell[a], bb = ub - cell[a];
            Dd[a] = bb - aa;
            m[a] = 0.5 * (aa + bb);
        }
        // every point of the piece's cell exists: cells -1..n (the path moves less
        // than a cell per axis from a physical position); out of range is recorded
        bool ok = true;
        for (int a = 0; a < 3; a++) ok = ok && cell[a] >= -1 && cell[a] + 2 < g.tot[a];
        if (!ok) continue;
        for (int a = 0; a < 3; a++) {
            const int jb = (a + 1) % 3, kb = (a + 2) % 3;
            const double w = coef * g.d[a] * Dd[a];
            const double cr = Dd[jb] * Dd[kb] / 12.0;
            const double W[4] = {w * ((1.0 - m[jb]) * (1.0 - m[kb]) + cr), w * (m[jb] * (1.0 - m[kb]) - cr),
                                 w * ((1.0 - m[jb]) * m[kb] - cr), w * (m[jb] * m[kb] + cr)};
            for (int e = 0; e < 4; e++) {
                int ii[3] = {cell[0] + 1, cell[1] + 1, cell[2] + 1};
                ii[jb] += e & 1;
                ii[kb] += e >> 1;
                atomicAdd(D.J[a] + gidx(g, ii[0], ii[1], ii[2]), W[e]);
            }
        }
    }
}

// The corrected policy's time-loop kernel: gather at the current position
// (the cell's own vertex), push, the charge-conserving current of the move,
// then the (periodic) boundaries.
// A move that ends beyond an absorbing wall removes the particle; its whole
// charge must cross the wall's vertex plane for continuity to hold there, so
// the path is continued along the wall's normal to the next vertex plane
// beyond the wall (x0 - d or x0 + L + d), a piece inside the ghost cell
// (corrected policy, as the oracle's absorbed_exit).
__device__ void absorbed_exit(const Geom &g, const BCTab &bc, const DepositPtrs &D, const double p1[3],
                              double coef) {
    double a[3] = {p1[0], p1[1], p1[2]};
    for (int d = 0; d < 3; d++) {
        double b[3] = {a[0], a[1], a[2]};
        if (bc.pbc[2 * d] == PBC_ABSORBING && a[d] < bc.xmin[d]) b[d] = bc.xmin[d] - g.d[d];
        else if (bc.pbc[2 * d + 1] == PBC_ABSORBING && a[d] > bc.xmax[d]) b[d] = bc.xmax[d] + g.d[d];
        else continue;
        vb_deposit(g, D, a, b, coef);
        a[d] = b[d];
    }
}

// The corrected policy's time-loop kernel. A particle that stays in its cell
// (no face crossed, no wall reached) makes one current piece, whose 12 terms
// go through the warp's run sums like any deposit. The others - a few lanes
// of nearly every warp - are put on a list of the block and worked off
// together by full warps: splitting their paths in place would make every
// warp issue the whole piece arithmetic on the FP64 pipe for them, and their
// pieces end in scattered atomics either way. Relativistic beams, 1,682,464
// particles in 49x37x29 unit cells: 1056 us a launch, FP64 pipe 84 % active,
// against 1877 us with every particle's pieces committed one by one (12
// atomics a piece) and the FP64 tests, conversions and divisions in place.
// A whole move's terms use fused adds and a product by 1 / 12: there is no
// reference to match bit for bit, and vb_deposit's are within rounding of them.
template <bool REL, int MODE>
__global__ void __launch_bounds__(FUSED_BLOCK) k_fused_vb(Geom g, SpeciesTab st, BCTab bc, GatherPtrs P, PState S,
                                                         int64_t np, DepositPtrs D, double dt,
                                                         DevCounters *ctr) {
    after_previous<false>();
    constexpr bool UNIT = MODE != ANY;
    __shared__ CommitTile tiles[FUSED_BLOCK / 32];
    __shared__ double s_move[6][FUSED_BLOCK];  // start and end of the listed moves
    __shared__ double s_coef[FUSED_BLOCK];
    __shared__ int s_n;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    bool active = false, listed = false;
    int64_t o = 0;
    int mask = 0;
    double c[12], coef = 0.0, p0[3] = {0.0, 0.0, 0.0}, p1[3] = {0.0, 0.0, 0.0};
    if (p < np) {
        double pos[3] = {S.x[p], S.y[p], S.z[p]};
        if (alive(pos[0])) {
            int s = species_of(st, p);
            int ci[3];
            locate<UNIT>(g, pos, ci);
            if (!cell_ok(g, ci[0], ci[1], ci[2])) {
                atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
            } else {
                double ds[3], e[3], b2[3], E12[12], S6[6];
                from_vertex<UNIT>(g, ci, pos, ds);
                o = gidx(g, ci[0], ci[1], ci[2]);
                gather_cell<UNIT>(g, P, o, ds, e, b2, E12, S6);
                double v[3] = {S.vx[p], S.vy[p], S.vz[p]};
#pragma unroll
                for (int a = 0; a < 3; a++) p0[a] = pos[a];
                if (REL) {
                    double ga = S.g[p];
                    VayStep vt;
                    vay_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v, ga, vt);
                    S.g[p] = ga;
                } else {
                    boris_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v);
                }
#pragma unroll
                for (int a = 0; a < 3; a++) p1[a] = pos[a];
                const bool hit = maybe_crossed(bc, pos);
                if (st.deposit[s] && dt > 0.0) {
                    coef = st.vbc[s];
                    double u0[3], u1[3];
                    listed = leaves_cell<UNIT>(g, ci, p0, p1, u0, u1) || hit;
                    if (!listed) {
                        active = true;
                        double m[3], Dd[3], n[3];
#pragma unroll
                        for (int a = 0; a < 3; a++) {
                            Dd[a] = u1[a] - u0[a];
                            m[a] = __fma_rn(0.5, Dd[a], UNIT ? ds[a] : u0[a] - f64_of_int(ci[a] - 1));
                            n[a] = 1.0 - m[a];
                        }
#pragma unroll
                        for (int a = 0; a < 3; a++) {
                            const int j = (a + 1) % 3, k = (a + 2) % 3;
                            const double w = UNIT ? coef * Dd[a] : coef * g.d[a] * Dd[a];
                            const double cr = Dd[j] * Dd[k] * (1.0 / 12.0);
                            c[4 * a] = w * __fma_rn(n[j], n[k], cr);
                            c[4 * a + 1] = w * __fma_rn(m[j], n[k], -cr);
                            c[4 * a + 2] = w * __fma_rn(m[j], m[k], cr);
                            c[4 * a + 3] = w * __fma_rn(n[j], m[k], -cr);
                        }
                    }
                }
                if (hit) {
                    mask = apply_bc(bc, pos, v);
                    if (mask & 64) pos[0] = __longlong_as_double(0x7ff8000000000000LL);
                }
                S.x[p] = pos[0]; S.y[p] = pos[1]; S.z[p] = pos[2];
                S.vx[p] = v[0]; S.vy[p] = v[1]; S.vz[p] = v[2];
            }
        }
    }
    if (__any_sync(0xffffffffu, mask & 63)) count_crossings(ctr, mask);
    const unsigned lm = __ballot_sync(0xffffffffu, listed);
    if (lm) {
        const int lane = threadIdx.x & 31;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_n, __popc(lm));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(lm & lanemask_lt());
        if (listed) {
#pragma unroll
            for (int a = 0; a < 3; a++) {
                s_move[a][at] = p0[a];
                s_move[3 + a][at] = p1[a];
            }
            s_coef[at] = coef;
        }
    }
    commit_deposit<12, 0>(g, D, tiles[threadIdx.x >> 5], active, o, c);
    __syncthreads();
    for (int i = threadIdx.x; i < s_n; i += FUSED_BLOCK) {
        const double a[3] = {s_move[0][i], s_move[1][i], s_move[2][i]};
        const double b[3] = {s_move[3][i], s_move[4][i], s_move[5][i]};
        vb_deposit(g, D, a, b, s_coef[i]);
        absorbed_exit(g, bc, D, b, s_coef[i]);
    }
}

// The fused time-loop kernel: gather at the current position (what
// InterpolateEB cached at the end of the previous step), push, the six
// boundaries, then the current deposit at the new position. Bound by the FP64
// pipe: some 230 FP64 instructions a particle (405 with tests, conversions and
// divisions on that pipe and the deposit summed in shuffle trees), 85 % active.
// Relativistic, 3,538,944 particles in 48^3 unit cells, sorted: 1513 us a
// launch against 2550 us.
template <bool REL, int MODE>
__global__ void __launch_bounds__(FUSED_BLOCK) k_fused(Geom g, SpeciesTab st, BCTab bc, GatherPtrs P, PState S,
                                                      int64_t np, DepositPtrs D, double dt, DevCounters *ctr) {
    after_previous<false>();
    constexpr bool UNIT = MODE != ANY;
    __shared__ CommitTile tiles[FUSED_BLOCK / 32];
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    bool active = false;
    int64_t o = 0;
    int mask = 0;
    double c[12];
    if (p < np) {
        double pos[3] = {S.x[p], S.y[p], S.z[p]};
        if (alive(pos[0])) {
            int s = species_of(st, p);
            int ci[3];
            locate<UNIT>(g, pos, ci);
            if (!cell_ok(g, ci[0], ci[1], ci[2])) {
                atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
            } else {
                double ds[3], e[3], b2[3], E12[12], S6[6];
                from_vertex<UNIT>(g, ci, pos, ds);
                gather_cell<UNIT>(g, P, gidx(g, ci[0], ci[1], ci[2]), ds, e, b2, E12, S6);
                double v[3] = {S.vx[p], S.vy[p], S.vz[p]};
                if (REL) {
                    double ga = S.g[p];
                    VayStep vt;
                    vay_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v, ga, vt);
                    S.g[p] = ga;
                } else {
                    boris_push<MODE>(st.qp[s], st.hqp[s], e, b2, dt, pos, v);
                }
                if (maybe_crossed(bc, pos)) mask = apply_bc(bc, pos, v);
                if (mask & 64) {
                    pos[0] = __longlong_as_double(0x7ff8000000000000LL);
                } else if (st.deposit[s]) {
                    locate<UNIT>(g, pos, ci);
                    if (cell_ok(g, ci[0], ci[1], ci[2])) {
                        active = true;
                        o = gidx(g, ci[0], ci[1], ci[2]);
                        from_vertex<UNIT>(g, ci, pos, ds);
                        deposit_terms_j<UNIT>(g, st.uq[s], ds, v, c);
                    } else {
                        atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
                    }
                }
                S.x[p] = pos[0]; S.y[p] = pos[1]; S.z[p] = pos[2];
                S.vx[p] = v[0]; S.vy[p] = v[1]; S.vz[p] = v[2];
            }
        }
    }
    if (__any_sync(0xffffffffu, mask & 63)) count_crossings(ctr, mask);
    commit_deposit<12, 0>(g, D, tiles[threadIdx.x >> 5], active, o, c);
}

// Per-block partial sums of the history's particle terms
// (src/IO/output.cpp:76-87): {sum 1/2 m v^2, sum m vx, sum m vy, sum m vz}.
__global__ void k_moments(SpeciesTab st, PState S, int64_t np, double *part) {
    after_previous();
    double acc[4] = {0, 0, 0, 0};
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        double vx = S.vx[p], vy = S.vy[p], vz = S.vz[p];
        if (!alive(S.x[p])) continue;
        double m = st.m[species_of(st, p)];
        acc[0] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        acc[1] += m * vx;
        acc[2] += m * vy;
        acc[3] += m * vz;
    }
    __shared__ double sh[32][4];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double total = warp_totals<4>(acc);
    const int at = total_index<4>(lane);
    if ((lane & 7) == 0) sh[w][at] = total;
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = 0.0;
        for (int ww = 0; ww < (int)(blockDim.x >> 5); ww++) v += sh[ww][threadIdx.x];
        part[blockIdx.x * 4 + threadIdx.x] = v;
    }
}

// Sort keys: species * ncell + reference cellID; removed particles get the
// largest key so they end up behind every live one.
__global__ void k_keys(Geom g, SpeciesTab st, PState S, int64_t np, uint32_t *key, uint32_t dead_key, DevCounters *ctr) {
    after_previous();
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    double x = S.x[p];
    if (!alive(x)) {
        key[p] = dead_key;
        return;
    }
    const double pos[3] = {x, S.y[p], S.z[p]};
    int ci[3];
    locate<false>(g, pos, ci);
    const int ix = ci[0], iy = ci[1], iz = ci[2];
    if (ix < 0 || iy < 0 || iz < 0 || ix >= g.n[0] + 2 || iy >= g.n[1] + 2 || iz >= g.n[2] + 2) {
        atomicOr(&ctr->err, (unsigned long long)ERR_BOUNDS);
        key[p] = dead_key - 1;
        return;
    }
    int s = species_of(st, p);
    key[p] = (uint32_t)((int64_t)s * g.ncell + cell_id(g, ix, iy, iz));
}

GatherPtrs gather_ptrs(emoo_handle *h) {
    GatherPtrs P;
    for (int c = 0; c < 3; c++) {
        P.E[c] = h->slot[EMOO_EX + c];
        P.B[c] = role_b(h, c);
        P.T[c] = role_t(h, c);
    }
    return P;
}

DepositPtrs deposit_ptrs(emoo_handle *h) {
    DepositPtrs D;
    for (int c = 0; c < 3; c++) D.J[c] = h->slot[EMOO_JX + c];
    D.rho = h->slot[EMOO_RHO];
    return D;
}

PState pstate(emoo_handle *h) { return PState{h->x, h->y, h->z, h->vx, h->vy, h->vz, h->gam}; }

int blocks_for(int64_t n, int t = 256) { return (int)std::max<int64_t>(1, (n + t - 1) / t); }

// ---- sensitivity probe (no reference counterpart) -------------------------

// Uniform in [-1, 1) from (seed, particle or point, component): splitmix64.
__device__ __forceinline__ double unit_noise(uint64_t seed, uint64_t i, uint64_t comp) {
    uint64_t z = seed + (i * 8u + comp + 1u) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 4503599627370496.0) - 1.0;  // 2^-52 steps over [-1, 1)
}

// Every live particle: v *= 1 + rel u, x += rel d u per component (u the
// noise above), a moved position kept only while it stays inside the box.
__global__ void k_perturb_particles(Geom g, PState S, int64_t np, uint64_t seed, double rel) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= np || S.x[p] != S.x[p]) return;
    double *pos[3] = {S.x, S.y, S.z}, *vel[3] = {S.vx, S.vy, S.vz};
    for (int c = 0; c < 3; c++) {
        vel[c][p] *= 1.0 + rel * unit_noise(seed, (uint64_t)p, c);
        const double x = pos[c][p] + rel * g.d[c] * unit_noise(seed, (uint64_t)p, 3 + c);
        if (x >= g.x0[c] && x < g.x0[c] + g.n[c] * g.d[c]) pos[c][p] = x;
    }
}

// f *= 1 + rel u at every point of one field (comp tells fields apart).
__global__ void k_perturb_field(double *f, int64_t n, uint64_t seed, uint64_t comp, double rel) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) f[i] *= 1.0 + rel * unit_noise(seed, (uint64_t)i, comp);
}

}  // namespace

void species_tab(emoo_handle *h, double dtp, SpeciesTab &st) {
    st.nspec = h->nspec;
    for (int s = 0; s <= h->nspec; s++) st.off[s] = h->off[s];
    for (int s = h->nspec + 1; s <= EMOO_NSPEC; s++) st.off[s] = h->off[h->nspec];
    const Geom &g = h->g;
    for (int s = 0; s < EMOO_NSPEC; s++) {
        double q = h->info.charge_ratio[s], m = h->info.mass_ratio[s];
        st.q[s] = q;
        st.m[s] = m;
        double qp = (0.5 * dtp * q) / m;
        qp *= UNIT_ACC;
        st.qp[s] = qp;
        st.hqp[s] = 0.5 * qp;
        st.uq[s] = UNIT_RHOJ * q;
        st.cr[s] = UNIT_RHOJ * (q / g.vol) / g.vol;
        st.vbc[s] = dtp > 0.0 ? st.uq[s] / g.vol / dtp : 0.0;
        st.deposit[s] = h->info.isTestParticle[s] ? 0 : 1;
    }
}

int interpolate_f64(emoo_handle *h) {
    if (h->np == 0) return EMOO_OK;
    if (!h->fcache) EMOO_CUDA(cudaMalloc(&h->fcache, sizeof(double) * 6 * (size_t)h->cap));
    h->launches++;
    k_interpolate<<<blocks_for(h->np), 256, 0, h->stream>>>(h->g, gather_ptrs(h), pstate(h), h->np, h->cap, h->fcache,
                                                            h->ctr);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int push_cached_f64(emoo_handle *h, double dtp) {
    if (h->np == 0) return EMOO_OK;
    if (!h->fcache) return EMOO_ERR_STATE;
    SpeciesTab st;
    species_tab(h, dtp, st);
    h->launches++;
    k_push_cached<<<blocks_for(h->np), 256, 0, h->stream>>>(st, pstate(h), h->np, h->cap, h->fcache, dtp,
                                                            h->info.relativity != 0);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int particle_bc_f64(emoo_handle *h) {
    if (h->np == 0) return EMOO_OK;
    h->launches++;
    k_particle_bc<<<blocks_for(h->np), 256, 0, h->stream>>>(h->bc, pstate(h), h->np, h->ctr);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int deposit_f64(emoo_handle *h, int with_rho) {
    size_t bytes = sizeof(double) * (size_t)h->g.npts;
    for (int c = 0; c < 3; c++) EMOO_CUDA(cudaMemsetAsync(h->slot[EMOO_JX + c], 0, bytes, h->stream));
    if (with_rho) EMOO_CUDA(cudaMemsetAsync(h->slot[EMOO_RHO], 0, bytes, h->stream));
    if (h->np == 0) return rho_background_f64(h, with_rho);
    SpeciesTab st;
    species_tab(h, h->dtp, st);
    h->launches++;
    launch_after(k_deposit, blocks_for(h->np, PART_BLOCK), PART_BLOCK, 0, h->stream)(h->g, st, pstate(h), h->np, deposit_ptrs(h), with_rho, h->ctr);
    EMOO_CUDA(cudaGetLastError());
    return rho_background_f64(h, with_rho);
}

// rho alone at the particles' current positions (J untouched), plus the
// background: the charge density the loop's last deposit would have left.
int deposit_rho_f64(emoo_handle *h) {
    EMOO_CUDA(cudaMemsetAsync(h->slot[EMOO_RHO], 0, sizeof(double) * (size_t)h->g.npts, h->stream));
    if (h->np > 0) {
        SpeciesTab st;
        species_tab(h, h->dtp, st);
        h->launches++;
        launch_after(k_deposit, blocks_for(h->np, PART_BLOCK), PART_BLOCK, 0, h->stream)(h->g, st, pstate(h), h->np, deposit_ptrs(h), 2, h->ctr);
        EMOO_CUDA(cudaGetLastError());
    }
    return rho_background_f64(h, 1);
}

template <bool REL, int MODE>
static void launch_fused(emoo_handle *h, const SpeciesTab &st, double dtp) {
    // Blocks of 128 leave a shorter last wave than blocks of 256: 131,072
    // relativistic particles, 10 steps, 1320 -> 1240 us, 442,368 2855 -> 2775,
    // 1.3 million 7260 -> 7180, 2.5 million 12770 -> 12700; at 1.0 and 3.5
    // million the same. Blocks of 64, whose lists of moves fill few warps, took
    // k_fused_vb 17 % longer at 1.7 million.
    const int blk = FUSED_BLOCK, nb = blocks_for(h->np, blk);
    if (h->policy == EMOO_POLICY_CORRECTED)
        launch_after(k_fused_vb<REL, MODE>, nb, blk, 0, h->stream)(h->g, st, h->bc, gather_ptrs(h), pstate(h), h->np,
                                                                   deposit_ptrs(h), dtp, h->ctr);
    else
        launch_after(k_fused<REL, MODE>, nb, blk, 0, h->stream)(h->g, st, h->bc, gather_ptrs(h), pstate(h), h->np,
                                                                deposit_ptrs(h), dtp, h->ctr);
}

int fused_step_f64(emoo_handle *h, double dtp) {
    size_t bytes = sizeof(double) * (size_t)h->g.npts;
    for (int c = 0; c < 3; c++) EMOO_CUDA(cudaMemsetAsync(h->slot[EMOO_JX + c], 0, bytes, h->stream));
    if (h->np == 0) return EMOO_OK;
    SpeciesTab st;
    species_tab(h, dtp, st);
    const bool timed = h->prof_on && h->policy != EMOO_POLICY_CORRECTED;
    h->launches++;
    if (timed) EMOO_CUDA(cudaEventRecord(h->prof_ev[0], h->stream));
    const int mode = !h->g.unit ? ANY : is_pow2(dtp) ? UNIT_DT2 : UNIT_CELLS;
    if (h->info.relativity) {
        if (mode == UNIT_DT2) launch_fused<true, UNIT_DT2>(h, st, dtp);
        else if (mode == UNIT_CELLS) launch_fused<true, UNIT_CELLS>(h, st, dtp);
        else launch_fused<true, ANY>(h, st, dtp);
    } else {
        if (mode == UNIT_DT2) launch_fused<false, UNIT_DT2>(h, st, dtp);
        else if (mode == UNIT_CELLS) launch_fused<false, UNIT_CELLS>(h, st, dtp);
        else launch_fused<false, ANY>(h, st, dtp);
    }
    EMOO_CUDA(cudaGetLastError());
    if (timed) {
        EMOO_CUDA(cudaEventRecord(h->prof_ev[1], h->stream));
        EMOO_TRY(prof_accumulate(h));
    }
    return EMOO_OK;
}

int particle_moments_f64(emoo_handle *h, double out4[4]) {
    for (int q = 0; q < 4; q++) out4[q] = 0.0;
    if (h->np == 0) return EMOO_OK;
    int nb = (int)std::min<int64_t>(blocks_for(h->np), 152 * 8);
    if (h->red_cap < (size_t)nb * 4) {
        if (h->red) cudaFree(h->red);
        EMOO_CUDA(cudaMalloc(&h->red, (size_t)nb * 4 * sizeof(double)));
        h->red_cap = (size_t)nb * 4;
    }
    SpeciesTab st;
    species_tab(h, h->dtp, st);
    h->launches++;
    launch_after(k_moments, nb, 256, 0, h->stream)(st, pstate(h), h->np, h->red);
    EMOO_CUDA(cudaGetLastError());
    std::vector<double> part((size_t)nb * 4);
    EMOO_CUDA(cudaMemcpyAsync(part.data(), h->red, part.size() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    EMOO_CUDA(cudaStreamSynchronize(h->stream));
    for (int b = 0; b < nb; b++)
        for (int q = 0; q < 4; q++) out4[q] += part[(size_t)b * 4 + q];
    return EMOO_OK;
}

// Compaction keys: the species index, nspec for removed particles (a stable
// sort by them drops the removed particles and keeps every species' order).
__global__ void k_compact_keys(SpeciesTab st, const double *x, int64_t np, uint32_t *key) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= np) return;
    key[p] = alive(x[p]) ? (uint32_t)species_of(st, p) : (uint32_t)st.nspec;
}

int compact_keys_f64(emoo_handle *h) {
    SpeciesTab st;
    species_tab(h, h->dtp, st);
    h->launches++;
    k_compact_keys<<<blocks_for(h->np), 256, 0, h->stream>>>(st, h->x, h->np, h->key[0]);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

int perturb_f64(emoo_handle *h, uint64_t seed, double rel) {
    if (h->np) {
        h->launches++;
        k_perturb_particles<<<blocks_for(h->np), 256, 0, h->stream>>>(h->g, pstate(h), h->np, seed, rel);
        EMOO_CUDA(cudaGetLastError());
    }
    const int ids[9] = {EMOO_EX, EMOO_EY, EMOO_EZ, EMOO_BX, EMOO_BY, EMOO_BZ, EMOO_BX_TM1, EMOO_BY_TM1, EMOO_BZ_TM1};
    for (int k = 0; k < 9; k++) {
        h->launches++;
        k_perturb_field<<<blocks_for(h->g.npts), 256, 0, h->stream>>>(h->slot[ids[k]], h->g.npts, seed, 8 + k, rel);
        EMOO_CUDA(cudaGetLastError());
    }
    return EMOO_OK;
}

int sort_keys_f64(emoo_handle *h) {
    SpeciesTab st;
    species_tab(h, h->dtp, st);
    uint32_t dead = (uint32_t)((int64_t)h->nspec * h->g.ncell + 1);
    h->launches++;
    launch_after(k_keys, blocks_for(h->np), 256, 0, h->stream)(h->g, st, pstate(h), h->np, h->key[0], dead, h->ctr);
    EMOO_CUDA(cudaGetLastError());
    return EMOO_OK;
}

}  // namespace emoo
