// step_kernels.cuh -- the kernels of one ISPH-DEM step.
//
// One kernel per fused pass, launched in the order of SOPHIA_single_ISPH
// (ISPH_Calc_seperate.cuh:13-503):
//
//   k_hash_* / sort / k_cells_gather_*   NNPS: cell key, stable sort by cell,
//                                        cell start/end + SoA permutation
//   k_build_list                         SPH neighbour list (kappa*h_i)
//   k_passA          mass_init + KGC + SPH porosity + prep_sph
//   k_dem_prep       DEM filters and porosity
//   k_passB          prep3D filter + advection forces
//   k_dem_contact    Hertz-Mindlin contact with tangential history
//   k_dem_coupling   Di Felice drag + pressure-gradient force + DEM predictor
//   k_sph_coupling   reaction force + SPH predictor
//   k_neumann        wall pressure/density/temperature extrapolation
//   k_ppe            one Jacobi sweep of the pressure Poisson equation
//   k_passC          pressure force + SPH corrector
//   k_dem_update     DEM corrector + cylinder/box/cone walls
//   k_open_bc        inlet/outlet ghost extrapolation
//   k_xsph           XSPH velocity/temperature smoothing
//
// Each kernel cites the reference kernels it replaces.  R is the field
// precision (float or double); positions, h and radii are always double.
#pragma once
#include "engine.cuh"

namespace sphdem {

// pair geometry in field precision from double positions
template <typename R>
struct Pair {
    R dx, dy, dz, r2, r;
};

template <typename R>
__device__ __forceinline__ Pair<R> make_pair(double xi, double yi, double zi, double xj, double yj, double zj) {
    Pair<R> g;
    g.dx = (R)(xi - xj);
    g.dy = (R)(yi - yj);
    g.dz = (R)(zi - zj);
    g.r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
    g.r = sqrt(g.r2);
    return g;
}

// Two-dimensional beds (dim 2) lie in a plane y = const and run this step
// with: the 2-D kernel normalisation; SPH particle volume (h / h_over_dx)^2;
// the gradient correction on the x-z block; a DEM sphere (centre in the
// plane; contact, drag and heat as for a sphere) in the porosity with its
// equatorial disc 3.14159 r^2, as the reference's 2-D coupling prep
// (KERNEL_clc_prep2D_coupling, functions_PREP2.cuh:2944-3033) -- the
// sphere's volume over a depth 4 r / 3 -- and its drag and heat acting on
// the fluid per unit depth (divided by that depth).
template <typename R>
__device__ __forceinline__ R dem_measure(const DevParams& P, R r) {
    return P.dim == 2 ? (R)3.14159 * r * r : (R)4.18879 * r * r * r;
}
template <typename R>
__device__ __forceinline__ R sph_volume(const DevParams& P, R th, R hd) {
    return P.dim == 2 ? (th / hd) * (th / hd) : (th / hd) * (th / hd) * (th / hd);
}

// One pair of a position + volume pass (nb_sum): displacement x_i - x_j, the
// volume of j in the pass's sums and in its Shepard sum.
template <typename R>
struct PairV {
    R dx, dy, dz, v, vs;
};
// prep step: SHEP: the Shepard sum takes only the marked types
template <typename R, bool SHEP>
__device__ __forceinline__ bool pv_prep(const DevParams& P, const PvRec<R>& qi, bool slow_i, const PvRec<R>& qj,
                                        PairV<R>& g) {
    const R v = pv_vol(qj);
    const Disp<R> d = pv_disp(P, qi, qj);
    g = PairV<R>{d.dx, d.dy, d.dz, (R)fabs(v), SHEP ? (v > (R)0 ? v : (R)0) : (R)fabs(v)};
    return slow_i || v != v;
}
// fix step of one pair: true when i or j is not usable from its record; the
// pair then comes from the double positions, and tag is the tag of j
template <typename R>
__device__ __forceinline__ bool pv_fix(const SphState<R>& S, const PosRec<R>* pos, const R* m, const R* rho,
                                       bool slow_i, const PvRec<R>& qj, int i, int j, PairV<R>& g, int& tag) {
    if (!slow_i && pv_vol(qj) == pv_vol(qj)) return false;
    const V4<R> s = pv_slow<R>(S.x, S.y, S.z, m, rho, i, j);
    g = PairV<R>{s.x, s.y, s.z, s.w, s.w};
    tag = ldr(pos + j).w;
    return true;
}

// 27-cell stencil in the reference order (z,y,x), calling f(j) for every
// slot j of every non-empty cell: the 9 rows in order, ascending slots
// inside a row.
template <typename F>
__device__ __forceinline__ void for_stencil_j(const DevParams& P, int ic, int jc, int kc,
                                              const int4* __restrict__ rows, const Cull& C, F f) {
    for_rows(P, ic, jc, kc, rows, C, [&](int a, int b) {
        for (int j = a; j < b; j++) f(j);
    });
}

// ---------------------------------------------------------------------------
// NNPS
// ---------------------------------------------------------------------------
// KERNEL_index_particle_to_cell_{sph,dem}: functions_NNPS.cuh:762-821
// The cell-sort count (cell_count, cell_sort.cuh) is fused in.
__global__ void k_hash(DevParams P, int n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ z, const int* __restrict__ itype, int* key, int* cnt) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int k = -1;
    if (i < n) {
        if (itype[i] == 3) k = P.num_cells;
        else {
            int ic, jc, kc;
            cell_ijk(P, x[i], y[i], z[i], ic, jc, kc);
            k = ic + P.NI * jc + P.NI * P.NJ * kc;
        }
        key[i] = k;
    }
    cell_count(cnt, k);
}

// per-cell stencil row table (for_rows), one thread per cell
__global__ void k_rows(DevParams P, const int* __restrict__ gs, const int* __restrict__ ge, int4* rows) {
    grid_dep_wait();
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int nc = P.NI * P.NJ * P.NK;
    if (c >= nc) return;
    int ic = c % P.NI, base = c - ic;
    rows[c] = row_bounds(gs, ge, P.NI, base, ic);
}

// reorder of every persistent SPH field, source of m/rho/pres/u/temp is
// the array that held the end-of-step value
template <typename R>
struct SphGatherSrc {
    const R *ux, *uy, *uz, *m, *rho, *pres, *temp;
};

template <typename R>
__global__ void k_cells_gather_sph(DevParams P, SphState<R> src, SphGatherSrc<R> gsrc, SphState<R> dst,
                                   SphRec<R> rec, const int* __restrict__ perm, int* wall_idx, int* buf_idx,
                                   int* counters, DevFlags* F) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    int p = perm[i];
    // all loads before the first store (see k_cells_gather_dem)
    double x = src.x[p], y = src.y[p], z = src.z[p], h = src.h[p];
    R ux = gsrc.ux[p], uy = gsrc.uy[p], uz = gsrc.uz[p], m = gsrc.m[p], rho = gsrc.rho[p], pr = gsrc.pres[p];
    const R temp = gsrc.temp[p], dd = src.dDEMpor[p], fs = src.flt_s[p], dp = src.dpres[p];
    int pt = src.ptype[p], bt = src.btype[p], it = src.itype[p];
    const int id = src.pid[p];
    dst.x[i] = x;
    dst.y[i] = y;
    dst.z[i] = z;
    dst.h[i] = h;
    dst.ux[i] = ux;
    dst.uy[i] = uy;
    dst.uz[i] = uz;
    dst.m[i] = m;
    dst.rho[i] = rho;
    dst.pres[i] = pr;
    dst.temp[i] = temp;
    dst.dDEMpor[i] = dd;
    dst.flt_s[i] = fs;
    dst.dpres[i] = dp;
    dst.ptype[i] = pt;
    dst.btype[i] = bt;
    dst.itype[i] = it;
    dst.pid[i] = id;
    const PosRec<R> q = make_pos<R>(P, x, y, z, pt, bt, it);
    store_pos(rec.pos, i, q);
    rec.mr0[i] = mk2<R>(m, rho);
    if (P.c2_passes) rec.pa[i] = pv_make(q, pv_code<R>(m / rho, q.w, pt == 1));
    rec.up[i] = mk4<R>(ux, uy, uz, pr);
    // walls and buffer particles of the step (parked slots excluded), up to
    // the launch bounds of their passes
    if (it != 3 && pt <= 0) {
        int k = atomicAdd(&counters[0], 1);
        if (k < P.nwall) wall_idx[k] = i;
        else atomicOr(&F->overflow, 4);
    }
    if (it != 3 && bt > 0 && pt < 1000) {
        int k = atomicAdd(&counters[1], 1);
        if (k < P.nbuf) buf_idx[k] = i;
        else atomicOr(&F->overflow, 4);
    }
}

// The same hand-over without NNPS, in place: the steps of one sphdem_step call
// after its first.  The step is Eulerian (SPH particles keep their positions
// and types), so the set is already in cell order and its grid, wall and
// buffer slots and neighbour list are those of the call's first step; only
// the end-of-step values become the state and the records are rebuilt.
template <typename R>
__global__ void k_refresh_sph(DevParams P, SphGatherSrc<R> g, SphState<R> S, SphRec<R> rec) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.ns) return;
    const R ux = g.ux[i], uy = g.uy[i], uz = g.uz[i], m = g.m[i], rho = g.rho[i], pr = g.pres[i];
    S.ux[i] = ux;
    S.uy[i] = uy;
    S.uz[i] = uz;
    S.m[i] = m;
    S.rho[i] = rho;
    S.pres[i] = pr;
    S.temp[i] = g.temp[i];
    rec.mr0[i] = mk2<R>(m, rho);
    rec.up[i] = mk4<R>(ux, uy, uz, pr);
    if (P.c2_passes) {
        const PosRec<R> q = ldr(rec.pos + i);
        rec.pa[i] = pv_make(q, pv_code<R>(m / rho, q.w, tag_ptype(q.w) == 1));
    }
}

template <typename R>
__global__ void k_cells_gather_dem(DevParams P, DemState<R> src, DemState<R> dst, const int* __restrict__ perm,
                                   DemWork<R> DW) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.nd;
    if (i >= n) return;
    int p = perm[i];
    // all loads before the first store: the sets may alias for all the compiler
    // knows, so a load waited behind each store, 26 latencies in a row.  20,000
    // spheres with their contact history: 27 -> 17 us
    const R x = src.x[p], y = src.y[p], z = src.z[p], h = src.h[p], rad = src.rad[p];
    const R ux = src.ux[p], uy = src.uy[p], uz = src.uz[p], wx = src.wx[p], wy = src.wy[p], wz = src.wz[p];
    const R m = src.m[p], rho = src.rho[p], ri = src.ri[p];
    const R t0 = src.temp[p], t1 = src.temp1[p], t2 = src.temp2[p], t3 = src.temp3[p];
    const R fx = src.Fdx_df[p], fy = src.Fdy_df[p], fz = src.Fdz_df[p], qs = src.Q_sd[p];
    const int pt = src.ptype[p], bt = src.btype[p], it = src.itype[p], id = src.pid[p], di = src.dem_idx[p];
    dst.x[i] = x; dst.y[i] = y; dst.z[i] = z; dst.h[i] = h; dst.rad[i] = rad;
    dst.ux[i] = ux; dst.uy[i] = uy; dst.uz[i] = uz;
    dst.wx[i] = wx; dst.wy[i] = wy; dst.wz[i] = wz;
    dst.m[i] = m; dst.rho[i] = rho; dst.ri[i] = ri;
    dst.temp[i] = t0; dst.temp1[i] = t1; dst.temp2[i] = t2; dst.temp3[i] = t3;
    dst.Fdx_df[i] = fx; dst.Fdy_df[i] = fy; dst.Fdz_df[i] = fz; dst.Q_sd[i] = qs;
    dst.ptype[i] = pt; dst.btype[i] = bt; dst.itype[i] = it; dst.pid[i] = id; dst.dem_idx[i] = di;
    // what the SPH passes read of a sphere
    DW.ra[i] = Dbl4{x, y, z, rad};
    DW.rb[i] = Dbl4{ux, uy, uz, m};
}

// SPH neighbour list: the candidate set and predicate of every SPH gather
// kernel (e.g. functions_PPE2.cuh:609-638): 27-cell stencil and
// sqrt(dx^2+dy^2+dz^2) + 1e-20 < kappa*h_i, decided exactly in FP64 (see
// test_pair).  Rows come out in ascending slot order, which is the
// reference's z,y,x cell visit order.  Column-major rows.  Threads of a
// warp are consecutive slots, mostly of one cell, so they walk the same
// candidate rows and their position-record loads coalesce.
template <typename R>
__global__ void __launch_bounds__(128) k_build_list(DevParams P, SphState<R> S, SphRec<R> rec,
                                                    const int4* __restrict__ rows,
                                                    int* __restrict__ nbr, int* __restrict__ ncnt, DevFlags* F) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.ns) return;
    double xi = S.x[i], yi = S.y[i], zi = S.z[i];
    double Rr = __dmul_rn(P.kappa, S.h[i]);
    Band bd = make_band(P, Rr);
    PosRec<R> qi = ldr(rec.pos + i);
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zi, ic, jc, kc);
    int c = 0, cap = P.nb_cap, n = P.ns;
    const Cull cu = make_cull(xi, yi, zi, Rr);
    for_rows(P, ic, jc, kc, rows, cu, [&](int a, int b) {
        for (int j = a; j < b; j++) {
            PosRec<R> qj = ldr(rec.pos + j);
            Disp<R> d;
            R r2;
            if (test_pair(P, qi, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, 1e-20, bd, d, r2)) {
                if (nbr && c < cap) nbr[nb_at(c, n, i)] = j;
                c++;
            }
        }
    });
    ncnt[i] = c;
    if (c > cap) atomicOr(&F->overflow, 1);
    // one atomic per converged group of threads for the largest count
    const unsigned am = __activemask();
    const int wmax = __reduce_max_sync(am, c);
    if ((threadIdx.x & 31) == __ffs(am) - 1) atomicMax(&F->max_ncnt, wmax);
}

// The 9 full stencil rows (z, y order) of cell (ic, jc, kc) for a whole
// warp: s[0..9] the prefix of the row lengths, s[10..18] the first slot of
// each row.  Returns the number of candidates; row_slot maps candidate t
// (0 <= t < that number) to its slot, in the reference's visit order.
__device__ __forceinline__ int stage_rows(const DevParams& P, int ic, int jc, int kc, const int4* __restrict__ rows,
                                          int* s, int lane) {
    int len = 0, lo = 0;
    if (lane < 9) {
        int kz = kc + lane / 3 - 1, jy = jc + lane % 3 - 1;
        if (kz >= 0 && kz <= P.NK - 1 && jy >= 0 && jy <= P.NJ - 1) {
            int4 r = __ldg(rows + ic + P.NI * jy + P.NI * P.NJ * kz);
            lo = r.x;
            len = max(r.w - r.x, 0);
        }
    }
    int inc = len;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane < 9) {
        s[lane + 1] = inc;
        s[10 + lane] = lo;
    }
    if (lane == 0) s[0] = 0;
    __syncwarp();
    return __shfl_sync(0xffffffffu, inc, 8);
}
__device__ __forceinline__ int row_slot(const int* s, int t) {
    int r = 0;
    while (t >= s[r + 1]) r++;
    return s[10 + r] + (t - s[r]);
}

// Relative FP32 coordinates of the cell-tiled passes.  A fixed-point
// position q is staged as (q - q0) x step, q0 a particle of the cell.  A
// position within Lk = 2 cell widths of q0 on every axis (all of a cell's
// stencil, unless a particle outside the box was clamped into a boundary
// cell) is 'near'; each staged coordinate then carries at most 2 x 2^-24 Lk
// of rounding (int -> float and x step), a difference at most 6 x 2^-24 Lk,
// and r^2 near Rr^2 moves by at most 2 sqrt(3) Rr (6 x 2^-24 L) + 3 FP32
// roundings, L = max Lk.  rel_band returns b with |r^2 error| < b Rr^2:
// 1.3e-6 L/Rr covers the rounding, q_abs/Rr the fixed-point quantisation
// of both positions, 1e-6 the rest.  A pair with a position outside the
// fixed-point range or not near takes the FP64 predicate.
struct RelFrame {
    int4 q0;
    int lx, ly, lz;         // 2 cell widths in steps per axis
    double L;               // max 2 cell widths (length)
    float sx, sy, sz;
    bool o_oor;             // q0 outside the fixed-point range: every pair exact
};
__device__ __forceinline__ RelFrame rel_frame(const DevParams& P, const int4& q0) {
    RelFrame F;
    F.q0 = q0;
    const double wx = (P.xmax - P.xmin) / P.NI, wy = (P.ymax - P.ymin) / P.NJ, wz = (P.zmax - P.zmin) / P.NK;
    F.lx = (int)fmin(2.0 * wx * P.q_inv[0] + 2.0, 2147483647.0);
    F.ly = (int)fmin(2.0 * wy * P.q_inv[1] + 2.0, 2147483647.0);
    F.lz = (int)fmin(2.0 * wz * P.q_inv[2] + 2.0, 2147483647.0);
    F.L = 2.0 * fmax(fmax(wx, wy), wz);
    F.sx = P.q_step[0];
    F.sy = P.q_step[1];
    F.sz = P.q_step[2];
    F.o_oor = (q0.w & TAG_OOR) != 0;
    return F;
}
// q outside the fixed-point range or not near q0.  In-range coordinates
// are below 2^30 in magnitude (quantize), so the int differences are exact.
__device__ __forceinline__ bool rel_slow(const RelFrame& F, const int4& q) {
    return (q.w & TAG_OOR) || abs(q.x - F.q0.x) > F.lx || abs(q.y - F.q0.y) > F.ly || abs(q.z - F.q0.z) > F.lz;
}
__device__ __forceinline__ float4 rel_coord(const RelFrame& F, const int4& q, int tagw) {
    return make_float4((float)(q.x - F.q0.x) * F.sx, (float)(q.y - F.q0.y) * F.sy, (float)(q.z - F.q0.z) * F.sz,
                       __int_as_float(tagw));
}
__device__ __forceinline__ double rel_band(const DevParams& P, const RelFrame& F, double Rr) {
    return 1e-6 + 1.3e-6 * F.L / Rr + P.q_abs / Rr;
}

// Cell-tiled list build (FP32 build).  One warp per cell: the particles of
// a cell share one stencil, so the warp stages the candidates of the 9 rows
// once, as FP32 coordinates relative to a particle of the cell, into shared
// memory (chunks of 128), and every lane -- one particle of the cell --
// tests them in the same order against its own radius.  All lanes read the
// same staged candidate (a broadcast) and run in lockstep; a pair costs a
// few FP32 operations instead of a global load and the fixed-point
// conversion.  Each lane appends its hits in staged order, which is the
// reference's z, y, x cell order with ascending slots, so the list equals
// the one-particle-per-thread build.  Prefilter: r^2 against Rr^2 (1 -/+ b)
// with b from rel_band.  Pairs in the band, or with a position outside the
// fixed-point range or not near the origin, take the reference predicate in
// FP64.
//
// The fast path forms r^2 as |c|^2 - 2 p.c + |p|^2: a candidate is staged
// with |c|^2, a lane holds -2p and compares |c|^2 - 2 p.c (three FMAs)
// against its threshold minus |p|^2.  Against the difference form this adds
// rounding of the magnitudes: |c|^2 (3 roundings), the three FMAs and |p|^2
// (3 more) and the threshold's subtraction, in all at most
// 6u (|c| + |p|)^2 + u hi^2 with u = 2^-24; both positions are near the
// origin (|c|, |p| <= sqrt(3) L), so dot_band widens the band by
// 80u (L / Rr)^2 + 2u of Rr^2.  Within the wider band the FP64 predicate
// decides, so the lists are unchanged.
// LW cells (warps) per block: 2, 4 or 8, picked per handle at commit with
// the one-thread-per-particle build (k_build_list) as the fourth candidate
// (list_build_mode, engine.cu); all four write the same lists.
constexpr int LT_CH = 128;
__device__ __forceinline__ double dot_band(const RelFrame& F, double Rr) {
    const double u = 5.9604644775390625e-08, q = F.L / Rr;
    return 80.0 * u * q * q + 2.0 * u;
}
template <int LW>
__global__ void __launch_bounds__(LW * 32) k_build_list_tiled(DevParams P, SphState<float> S,
                                                                      SphRec<float> rec,
                                                                      const int* __restrict__ gs,
                                                                      const int* __restrict__ ge,
                                                                      const int4* __restrict__ rows,
                                                                      int* __restrict__ nbr,
                                                                      int* __restrict__ ncnt, DevFlags* F) {
    grid_dep_wait();
    __shared__ float4 sc[LW][LT_CH + 4];   // relative x, y, z and |c|^2
    __shared__ int sj[LW][LT_CH + 4];      // slot, bit 31: not near the origin
    __shared__ int srow[LW][20];   // prefix[10] | start[9]
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * LW + w;
    const int ncell = P.NI * P.NJ * P.NK;
    if (c >= ncell) return;
    const int a0 = __ldg(gs + c);
    if (a0 < 0) return;
    const int e0 = __ldg(ge + c);
    const int ic = c % P.NI, jc = (c / P.NI) % P.NJ, kc = c / (P.NI * P.NJ);
    const int tot = stage_rows(P, ic, jc, kc, rows, srow[w], lane);
    const RelFrame Fr = rel_frame(P, ldr(rec.pos + a0));   // origin of the relative coordinates
    const int n = P.ns, cap = P.nb_cap;
    for (int p0 = a0; p0 < e0; p0 += 32) {
        const int i = p0 + lane;
        const bool act = i < e0;
        double xi = 0, yi = 0, zi = 0, Rr = 0;
        float lo2 = 0, hi2 = 0, fx = 0, fy = 0, fz = 0;
        float ax = 0, ay = 0, az = 0, tlo = 0, thi = 0;   // -2p and the thresholds of the fast path
        bool slow = true;
        if (act) {
            xi = S.x[i];
            yi = S.y[i];
            zi = S.z[i];
            Rr = __dmul_rn(P.kappa, S.h[i]);
            const double b = rel_band(P, Fr, Rr), r2 = Rr * Rr, bd = b + dot_band(Fr, Rr);
            lo2 = (float)(r2 * (1.0 - b));
            hi2 = (float)(r2 * (1.0 + b));
            const int4 qi = ldr(rec.pos + i);
            slow = Fr.o_oor || rel_slow(Fr, qi);
            const float4 f = rel_coord(Fr, qi, 0);
            fx = f.x;
            fy = f.y;
            fz = f.z;
            ax = -2.f * fx;
            ay = -2.f * fy;
            az = -2.f * fz;
            const float pp = fmaf(fz, fz, fmaf(fy, fy, fx * fx));
            tlo = (float)(r2 * (1.0 - bd)) - pp;
            thi = (float)(r2 * (1.0 + bd)) - pp;
        }
        int cnt = 0;
        // entry cnt of particle i at pw: +1 inside a block of 8 entries, to
        // the particle's next block (8n further) after the eighth
        int* pw = nbr ? nbr + nb_at(0, n, i) : nullptr;
        const ptrdiff_t next_block = 8 * (ptrdiff_t)n - 7;
        auto push = [&](int j) {
            if (pw && cnt < cap) *pw = j;
            pw += ((cnt & 7) == 7) ? next_block : 1;
            cnt++;
        };
        const bool lanes_slow = __any_sync(0xffffffffu, act && slow);
        // Candidates that no lane of this group can reach are not staged: the
        // lanes' box [bl, bh] and their largest prefilter radius hb.  The box
        // distance is formed like a lane's r^2 from differences that are no
        // larger, and FP32 rounding is monotone, so a candidate with box
        // distance^2 > hb (1 + 2^-20) has r^2 > hi2 for every lane.  Off while
        // a lane takes the FP64 path; a candidate outside the fixed-point
        // range is always staged.
        float blx = act ? fx : 3e38f, bly = act ? fy : 3e38f, blz = act ? fz : 3e38f;
        float bhx = act ? fx : -3e38f, bhy = act ? fy : -3e38f, bhz = act ? fz : -3e38f;
        float hb = act ? hi2 : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            blx = fminf(blx, __shfl_xor_sync(0xffffffffu, blx, o));
            bly = fminf(bly, __shfl_xor_sync(0xffffffffu, bly, o));
            blz = fminf(blz, __shfl_xor_sync(0xffffffffu, blz, o));
            bhx = fmaxf(bhx, __shfl_xor_sync(0xffffffffu, bhx, o));
            bhy = fmaxf(bhy, __shfl_xor_sync(0xffffffffu, bhy, o));
            bhz = fmaxf(bhz, __shfl_xor_sync(0xffffffffu, bhz, o));
            hb = fmaxf(hb, __shfl_xor_sync(0xffffffffu, hb, o));
        }
        hb *= 1.f + 9.5367431640625e-07f;
        const unsigned lt = (1u << lane) - 1u;
        int t = 0;
        while (t < tot) {
            // stage the next candidates that pass the box test, in order
            int tn = 0;
            bool any_oor = false;
            while (t < tot && tn <= LT_CH - 32) {
                const int tl = t + lane;
                bool keep = false;
                float4 v;
                int jt = 0;
                if (tl < tot) {
                    const int j = row_slot(srow[w], tl);
                    const int4 qj = ldr(rec.pos + j);
                    const bool oor = rel_slow(Fr, qj);
                    v = rel_coord(Fr, qj, 0);
                    v.w = fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x));
                    jt = j | (oor ? (int)0x80000000 : 0);
                    const float dx = fmaxf(fmaxf(blx - v.x, v.x - bhx), 0.f);
                    const float dy = fmaxf(fmaxf(bly - v.y, v.y - bhy), 0.f);
                    const float dz = fmaxf(fmaxf(blz - v.z, v.z - bhz), 0.f);
                    keep = oor || lanes_slow || dx * dx + dy * dy + dz * dz <= hb;
                    any_oor |= keep && oor;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int pos = tn + __popc(m & lt);
                    sc[w][pos] = v;
                    sj[w][pos] = jt;
                }
                tn += __popc(m);
                t += 32;
            }
            // padded to whole groups of four; the padding (|c|^2 = inf) fails every test
            const int tp = (tn + 3) & ~3;
            if (lane < tp - tn) {
                sc[w][tn + lane] = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7f800000));
                sj[w][tn + lane] = 0;
            }
            const bool slow_chunk = lanes_slow || __any_sync(0xffffffffu, any_oor);
            __syncwarp();
            if (act && !slow_chunk) {
                // fast path: the FP32 prefilter of 32 candidates into two masks
                // without a branch (in reach; certain), FP64 only inside the
                // band, then the lane's hits in order.  Appending where a
                // candidate was found ran the append for nearly every one, a
                // few lanes at a time: bench bed 182 -> 166 us.  (Blocks of 8
                // queued in shared memory, 171 us, and 64 registers, 171 us,
                // were no better.)
                for (int u = 0; u < tp; u += 32) {
                    unsigned in = 0, sure = 0;
#pragma unroll
                    for (int k = 0; k < 32; k += 4) {
                        if (u + k < tp) {
#pragma unroll
                            for (int v = k; v < k + 4; v++) {
                                const float4 cv = sc[w][u + v];
                                const float tv = fmaf(az, cv.z, fmaf(ay, cv.y, fmaf(ax, cv.x, cv.w)));
                                if (tv <= thi) in |= 1u << v;
                                if (tv < tlo) sure |= 1u << v;
                            }
                        }
                    }
                    for (unsigned b = in & ~sure; b; b &= b - 1) {
                        const int k = __ffs(b) - 1, j = sj[w][u + k];
                        if (!(__dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < Rr)) in &= ~(1u << k);
                    }
                    for (; in; in &= in - 1) push(sj[w][u + __ffs(in) - 1]);
                }
            } else if (act) {
                // a particle or candidate outside the fixed-point range: FP64 where needed
                for (int u = 0; u < tn; u++) {
                    const float4 cj = sc[w][u];
                    const float dx = fx - cj.x, dy = fy - cj.y, dz = fz - cj.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    const int jb = sj[w][u];
                    const int j = jb & 0x7fffffff;
                    bool hit;
                    if (!slow && jb >= 0) {
                        if (r2 < lo2) hit = true;
                        else if (r2 > hi2) hit = false;
                        else hit = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < Rr;
                    } else {
                        hit = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < Rr;
                    }
                    if (hit) push(j);
                }
            }
            __syncwarp();
        }
        if (act) {
            ncnt[i] = cnt;
            if (cnt > cap) atomicOr(&F->overflow, 1);
        }
        // one atomic per warp for the largest count
        const int wmax = __reduce_max_sync(0xffffffffu, act ? cnt : 0);
        if (lane == 0 && wmax > 0) atomicMax(&F->max_ncnt, wmax);
    }
}

// SPH -> DEM candidate list.  The SPH kernels that sum over DEM spheres
// (pass A's porosity, the reaction force of k_sph_coupling) visit the DEM
// slots of the 27-cell stencil in the reference's order and keep those
// with |x_i - x_j| < kappa h_i.  About one stencil candidate in ten is
// inside, so this pass finds them once per step and the two kernels walk
// the short list (same slots, same order) and repeat their own test on it.
// The list holds every j with pair_dist < kappa h_i, the add = 0 form of
// the predicate; the 1e-20 form of pass A keeps a subset of it.
//
// One warp per cell, as k_build_list_tiled: the cell's DEM candidates
// (p_type > 1000) are staged compacted in shared memory as FP32 coordinates
// relative to the cell's first SPH particle, and each lane -- one SPH
// particle of the cell -- tests them in order.  A coordinate within
// Lb = 4 cells of the origin is rounded by at most e = 2^-24 Lb, a
// difference by 4 e, so r^2 moves by at most 2 sqrt(3) Rr (4 e) + 3 (4 e)^2
// near the radius, plus a few FP32 roundings; the band below is wider and
// pairs inside it take the FP64 predicate.  A particle or sphere farther
// than Lb from the origin (one clamped into a boundary cell) always takes
// the FP64 predicate.  ncntd holds the exact count; a particle with more
// than cap hits keeps only its count, and the consumers walk its stencil
// instead.
constexpr int DL_WARPS = 4, DL_CH = 128;
// one cell of k_build_dlist (scw, srw: the warp's shared staging)
__device__ __forceinline__ void dlist_cell(int c, DevParams P, const double* __restrict__ sx,
                                                                 const double* __restrict__ sy,
                                                                 const double* __restrict__ sz,
                                                                 const double* __restrict__ sh,
                                                                 const int* __restrict__ gs, const int* __restrict__ ge,
                                                                 const int4* __restrict__ drows,
                                                                 const double* __restrict__ dx,
                                                                 const double* __restrict__ dy,
                                                                 const double* __restrict__ dz,
                                                                 const int* __restrict__ dptype, int* __restrict__ nbrd,
                                                                 int* __restrict__ ncntd, int cap, DevFlags* F, float4* scw, int* srw, int lane) {    const int a0 = __ldg(gs + c);
    if (a0 < 0) return;
    const int e0 = __ldg(ge + c);
    const int ic = c % P.NI, jc = (c / P.NI) % P.NJ, kc = c / (P.NI * P.NJ);
    const int tot = stage_rows(P, ic, jc, kc, drows, srw, lane);
    const int n = P.ns;
    const double x0 = sx[a0], y0 = sy[a0], z0 = sz[a0];
    const double Lb = 4.0 * fmax(fmax((P.xmax - P.xmin) / P.NI, (P.ymax - P.ymin) / P.NJ), (P.zmax - P.zmin) / P.NK);
    const double e4 = 4.0 * 5.9604644775390625e-08 * Lb;   // 4 x 2^-24 x Lb
    const unsigned lt = (1u << lane) - 1u;
    for (int p0 = a0; p0 < e0; p0 += 32) {
        const int i = p0 + lane;
        const bool act = i < e0;
        double xi = 0, yi = 0, zi = 0, Rr = 0;
        float lo2 = 0, hi2 = 0, fx = 0, fy = 0, fz = 0;
        bool slow = false;
        if (act) {
            xi = sx[i];
            yi = sy[i];
            zi = sz[i];
            Rr = P.kappa * sh[i];
            const double r2 = Rr * Rr, d = 3.5 * Rr * e4 + 3.0 * e4 * e4 + 2e-6 * r2;
            lo2 = (float)(r2 - d);
            hi2 = (float)(r2 + d);
            const double ux = xi - x0, uy = yi - y0, uz = zi - z0;
            slow = !(fabs(ux) <= Lb && fabs(uy) <= Lb && fabs(uz) <= Lb);
            fx = (float)ux;
            fy = (float)uy;
            fz = (float)uz;
        }
        const bool lanes_slow = __any_sync(0xffffffffu, act && slow);
        int cnt = 0;
        int* pw = nbrd ? nbrd + i : nullptr;   // entry cnt of row i at pw (pw += n per hit)
        int t = 0;
        while (t < tot) {
            int ns = 0;
            bool any_far = false;
            while (t < tot && ns <= DL_CH - 32) {
                const int tl = t + lane;
                int j = 0;
                bool keep = false;
                if (tl < tot) {
                    j = row_slot(srw, tl);
                    keep = __ldg(dptype + j) > 1000;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const double ux = dx[j] - x0, uy = dy[j] - y0, uz = dz[j] - z0;
                    const bool far = !(fabs(ux) <= Lb && fabs(uy) <= Lb && fabs(uz) <= Lb);
                    any_far |= far;
                    scw[ns + __popc(m & lt)] =
                        make_float4((float)ux, (float)uy, (float)uz, __int_as_float(j | (far ? (int)0x80000000 : 0)));
                }
                ns += __popc(m);
                t += 32;
            }
            // whole groups of four; the padding (r^2 = inf) fails every test
            const int np = (ns + 3) & ~3;
            if (lane < np - ns) scw[ns + lane] = make_float4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);
            const bool slow_chunk = lanes_slow || __any_sync(0xffffffffu, any_far);
            __syncwarp();
            auto push = [&](int j) {
                if (pw && cnt < cap) *pw = j;
                pw += n;
                cnt++;
            };
            if (act && !slow_chunk) {
                // masks of 32 candidates, as in k_build_list_tiled: bench bed
                // 42 -> 32 us, 200,000 spheres 340 -> 255 us
                for (int u = 0; u < np; u += 32) {
                    unsigned in = 0, sure = 0;
#pragma unroll
                    for (int k = 0; k < 32; k += 4) {
                        if (u + k < np) {
#pragma unroll
                            for (int v = k; v < k + 4; v++) {
                                const float4 cj = scw[u + v];
                                const float ex = fx - cj.x, ey = fy - cj.y, ez = fz - cj.z;
                                const float r2 = ex * ex + ey * ey + ez * ez;
                                if (!(r2 > hi2)) in |= 1u << v;
                                if (r2 < lo2) sure |= 1u << v;
                            }
                        }
                    }
                    for (unsigned b = in & ~sure; b; b &= b - 1) {
                        const int k = __ffs(b) - 1, j = __float_as_int(scw[u + k].w);
                        if (!(pair_dist(xi, yi, zi, dx[j], dy[j], dz[j]) < Rr)) in &= ~(1u << k);
                    }
                    for (; in; in &= in - 1) push(__float_as_int(scw[u + __ffs(in) - 1].w));
                }
            } else if (act) {
                for (int u = 0; u < ns; u++) {
                    const float4 cj = scw[u];
                    const int jb = __float_as_int(cj.w), j = jb & 0x7fffffff;
                    bool hit;
                    if (!slow && jb >= 0) {
                        const float ex = fx - cj.x, ey = fy - cj.y, ez = fz - cj.z;
                        const float r2 = ex * ex + ey * ey + ez * ez;
                        if (r2 > hi2) continue;
                        hit = r2 < lo2 || pair_dist(xi, yi, zi, dx[j], dy[j], dz[j]) < Rr;
                    } else {
                        hit = pair_dist(xi, yi, zi, dx[j], dy[j], dz[j]) < Rr;
                    }
                    if (hit) push(j);
                }
            }
            __syncwarp();
        }
        if (act) ncntd[i] = cnt;
        const int wmax = __reduce_max_sync(0xffffffffu, act ? cnt : 0);
        if (lane == 0 && wmax > 0) atomicMax(&F->max_ncntd, wmax);
    }
}

// The same list with one thread per SPH particle over the DEM slots of its
// stencil rows (the exact predicate for every candidate): the same entries
// in the same order.  Picked per handle at commit where it is faster (2-D
// beds, whose cells hold a few particles each); parked slots (i_type 3) keep
// their count, as the warp-per-cell build leaves them.
__global__ void __launch_bounds__(128) k_build_dlist_pp(DevParams P, const double* __restrict__ sx,
                                                        const double* __restrict__ sy,
                                                        const double* __restrict__ sz,
                                                        const double* __restrict__ sh,
                                                        const int* __restrict__ itype,
                                                        const int4* __restrict__ drows,
                                                        const double* __restrict__ dx,
                                                        const double* __restrict__ dy,
                                                        const double* __restrict__ dz,
                                                        const int* __restrict__ dptype, int* __restrict__ nbrd,
                                                        int* __restrict__ ncntd, int cap, DevFlags* F) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = P.ns;
    const bool act = i < n && itype[i] != 3;
    int cnt = 0;
    if (act) {
        const double xi = sx[i], yi = sy[i], zi = sz[i], Rr = P.kappa * sh[i];
        int ic, jc, kc;
        cell_ijk(P, xi, yi, zi, ic, jc, kc);
        int* pw = nbrd ? nbrd + i : nullptr;   // entry cnt of row i at pw (pw += n per hit)
        for_stencil_j(P, ic, jc, kc, drows, make_cull(xi, yi, zi, Rr), [&](int j) {
            if (__ldg(dptype + j) <= 1000) return;
            if (pair_dist(xi, yi, zi, dx[j], dy[j], dz[j]) < Rr) {
                if (pw && cnt < cap) *pw = j;
                pw += n;
                cnt++;
            }
        });
        ncntd[i] = cnt;
    }
    const int wmax = __reduce_max_sync(0xffffffffu, act ? cnt : 0);
    if ((threadIdx.x & 31) == 0 && wmax > 0) atomicMax(&F->max_ncntd, wmax);
}

template <bool OCC>
__global__ void __launch_bounds__(DL_WARPS * 32) k_build_dlist(DevParams P, const double* __restrict__ sx,
                                                                 const double* __restrict__ sy,
                                                                 const double* __restrict__ sz,
                                                                 const double* __restrict__ sh,
                                                                 const int* __restrict__ gs, const int* __restrict__ ge,
                                                                 const int4* __restrict__ drows,
                                                                 const double* __restrict__ dx,
                                                                 const double* __restrict__ dy,
                                                                 const double* __restrict__ dz,
                                                                 const int* __restrict__ dptype, int* __restrict__ nbrd,
                                                                 int* __restrict__ ncntd, int cap, DevFlags* F,
                                                                 const int* __restrict__ occ, const int* __restrict__ occ_n) {
    grid_dep_wait();
    __shared__ float4 sc[DL_WARPS][DL_CH + 32];
    __shared__ int srow[DL_WARPS][20];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (OCC) {   // a sparse grid: the occupied cells, grid-stride
        const int no = *occ_n;
        for (int q = blockIdx.x * DL_WARPS + w; q < no; q += gridDim.x * DL_WARPS) {
            dlist_cell(occ[q], P, sx, sy, sz, sh, gs, ge, drows, dx, dy, dz, dptype, nbrd, ncntd, cap, F, sc[w], srow[w], lane);
            __syncwarp();
        }
    } else {
        const int c = blockIdx.x * DL_WARPS + w;
        if (c < P.NI * P.NJ * P.NK)
            dlist_cell(c, P, sx, sy, sz, sh, gs, ge, drows, dx, dy, dz, dptype, nbrd, ncntd, cap, F, sc[w], srow[w], lane);
    }
}

// A walk over the SPH -> DEM list of particle i, two entries at a time: the
// list entries and the spheres' records (load(j)) of both are in flight before
// either is summed; one dependent chain per entry made this most of pass A on
// beds whose spheres are small against the kernel.  Sums in list order.
template <typename T, typename L, typename C>
__device__ __forceinline__ void dem_walk(const int* __restrict__ nbrd, int cd, int n, int i, L load, C comp) {
    int j0 = 0, j1 = 0;
    if (cd > 0) j0 = nbrd[i];
    if (cd > 1) j1 = nbrd[(size_t)n + i];
    int k = 0;
    for (; k + 2 <= cd; k += 2) {
        const T r0 = load(j0), r1 = load(j1);
        const int a = j0, b = j1;
        if (k + 2 < cd) j0 = nbrd[(size_t)(k + 2) * n + i];
        if (k + 3 < cd) j1 = nbrd[(size_t)(k + 3) * n + i];
        comp(a, r0);
        comp(b, r1);
    }
    if (k < cd) comp(j0, load(j0));
}
struct DemAB {
    Dbl4 a, b;
};
// KERNEL_clc_prep3D_coupling_sph (functions_PREP2.cuh:3190-3364): the sums of
// particle i over its spheres
template <typename R, int L, typename K>
__device__ __forceinline__ void sph_dem_porosity(const DevParams& P, const SphWork<R>& W, const DemState<double>& D,
                                                 const DemWork<double>& DW, const int4* __restrict__ drows,
                                                 const LaneGroup<L>& g, double xi, double yi, double zi, double hi,
                                                 const K& Kn, R& por, R& dfx, R& dfy, R& dfz) {
    const double Rr = P.kappa * hi;
    const float r2l = r2_lo(Rr), r2h = r2_hi(Rr);
    const int n = P.ns, i = g.i;
    struct T {
        R w, v, ax, ay, az;
    };
    auto load = [&](int j) { return DemAB{ldr(DW.ra + j), ldr(DW.rb + j)}; };
    auto terms = [&](int, const DemAB& q, T& t) {
        PairT<R> g = pair_test<R>(xi, yi, zi, q.a.x, q.a.y, q.a.z, Rr, 1e-20, r2l, r2h);
        if (!g.in) return false;
        R r = g.r + (R)1e-20, ir = rcp(r);
        t.w = kw(Kn, r);
        R dw = kdw(Kn, r);
        R rj = (R)q.a.w;
        t.v = dem_measure(P, rj);
        t.ax = dw * g.dx * ir * (R)q.b.x;
        t.ay = dw * g.dy * ir * (R)q.b.y;
        t.az = dw * g.dz * ir * (R)q.b.z;
        return true;
    };
    auto add = [&](const T& t) {
        por += t.w * t.v;
        dfx += t.ax * t.v;
        dfy += t.ay * t.v;
        dfz += t.az * t.v;
    };
    auto one = [&](int j, const DemAB& q) {
        T t;
        if (terms(j, q, t)) add(t);
    };
    const int cd = W.ncntd[i];
    if (cd <= P.nbd_cap) {
        if constexpr (L == 1) dem_walk<DemAB>(W.nbrd, cd, n, i, load, one);
        else ordered_walk<L, DemAB, T>(g, cd, [&](int k) { return W.nbrd[(size_t)k * n + i]; }, load, terms, add);
    } else {
        int ic, jc, kc;
        cell_ijk(P, xi, yi, zi, ic, jc, kc);
        for_stencil_j(P, ic, jc, kc, drows, make_cull(xi, yi, zi, Rr), [&](int j) {
            if (D.ptype[j] > 1000) one(j, load(j));
        });
    }
}

// ---------------------------------------------------------------------------
// pass A: KERNEL_clc_mass_init_sph (functions_MASS.cuh:24-43),
// KERNEL_clc_correction_KGC_3D_sph (functions_PREP2.cuh:452-568),
// KERNEL_clc_prep3D_coupling_sph (functions_PREP2.cuh:3190-3364),
// KERNEL_clc_prep3D_prep_sph (functions_PREP2.cuh:1623-1679).
// Neighbours read the start-of-step m, rho; the new m, rho go to m_new,
// rho_new so that no thread sees a half-updated neighbour.
// ---------------------------------------------------------------------------
// A pair adds V (x x^T) kg to the six moments and V kws to the Shepard sum
// (V = m / rho of the record, constant factors after the loop).  Registers in
// FP32 are held to 7 blocks per SM: 91 us on the bench bed at 8 blocks
// (spills), 86 at 7, 92 at 6.
template <typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 7 : 1) k_passA(DevParams P, SphState<R> S, SphWork<R> W, DemState<double> D,
                                               DemWork<double> DW, const int4* __restrict__ drows) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i];
    R mo = S.m[i], ro = S.rho[i];
    if (it > 2) {
        W.m_new[i] = mo;
        W.rho_new[i] = ro;
        rec.f1[i] = mk4<R>(mo, ro, S.temp[i], W.DEMpor[i]);
        return;
    }
    R dprev = S.dDEMpor[i];
    W.dDEMpor_prev[i] = dprev;
    double xi = S.x[i], yi = S.y[i], zi = S.z[i], hi = S.h[i];
    R th = (R)hi;
    const C2Sum<R> K = c2_sum<R>(P, th);
    const PvRec<R> qi = ldr(rec.pa + i);
    const bool slow_i = pv_vol(qi) != pv_vol(qi);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R txx = 0, tyy = 0, tzz = 0, txy = 0, tyz = 0, tzx = 0, sflt = 0;
    const int* __restrict__ nb = W.nbr;
    const bool kgc = P.kgc == 1;
    nb_sum<NbP<R>, PairV<R>>(
        cnt, nb, n, i,
        [&](int j) {
            NbP<R> t;
            t.q = ldr(rec.pa + j);
            return t;
        },
        [&](const NbP<R>& t, PairV<R>& g) { return pv_prep<R, true>(P, qi, slow_i, t.q, g); },
        [&](int j, NbP<R>& t, PairV<R>& g) {
            int tag;
            if (!pv_fix(S, rec.pos, S.m, S.rho, slow_i, t.q, i, j, g, tag)) return;
            if (tag_ptype(tag) > 1000) g.v = 0;
            if (tag_ptype(tag) != 1) g.vs = 0;
        },
        [&](int, const NbP<R>&, const PairV<R>& g) {
            const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
            const R rinv = rsq_floor(r2), r = r2 * rinv;
            sflt += g.vs * c2_w(K, r);
            const R w = g.v * c2_g(K, r);
            const R wx = w * g.dx, wy = w * g.dy, wz = w * g.dz;
            txx += wx * g.dx;
            txy += wx * g.dy;
            tzx += wx * g.dz;
            tyy += wy * g.dy;
            tyz += wy * g.dz;
            tzz += wz * g.dz;
        });
    sflt *= K.wn;
    if (kgc) {
        const R sc = -K.gn;
        txx *= sc; txy *= sc; tzx *= sc; tyy *= sc; tyz *= sc; tzz *= sc;
        Cm6<R> C{1, 0, 0, 1, 0, 1};
        if (P.dim == 2) {
            // a bed in a plane y = const: the x-z block of the moment matrix
            const R det = txx * tzz - tzx * tzx;
            if (fabs(det) > (R)1e-4) {
                const R rr = (R)1 / det;
                C.xx = tzz * rr;
                C.xz = -tzx * rr;
                C.zz = txx * rr;
            }
        } else {
            R det = txx * (tyy * tzz - tyz * tyz);
            det -= txy * (txy * tzz - tyz * tzx);
            det += tzx * (txy * tyz - tyy * tzx);
            if (fabs(det) > (R)1e-4) {
                R rr = (R)1 / det;
                C.xx = (tyy * tzz - tyz * tyz) * rr;
                C.xy = (tzx * tyz - txy * tzz) * rr;
                C.xz = (txy * tyz - tzx * tyy) * rr;
                C.yy = (txx * tzz - tzx * tzx) * rr;
                C.yz = (tzx * txy - txx * tyz) * rr;
                C.zz = (txx * tyy - txy * txy) * rr;
            }
        }
        W.Cm[i] = C.xx;
        W.Cm[(size_t)n + i] = C.xy;
        W.Cm[(size_t)2 * n + i] = C.xz;
        W.Cm[(size_t)3 * n + i] = C.yy;
        W.Cm[(size_t)4 * n + i] = C.yz;
        W.Cm[(size_t)5 * n + i] = C.zz;
    }
    R por = 0, dfx = 0, dfy = 0, dfz = 0;
    if (P.nd > 0) {
        const Knl<R, 3> Kd = knl_make<R, 3>(P, th);
        sph_dem_porosity<R, 1>(P, W, D, DW, drows, LaneGroup<1>(), xi, yi, zi, hi, Kd, por, dfx, dfy, dfz);
    }
    R isf = rcp(sflt + (R)1e-20);
    R pori = (R)1 - por * isf;
    W.DEMpor[i] = pori;
    S.dDEMpor[i] = (dfx + dfy + dfz) * isf;
    // prep_sph
    R hd = (R)P.h_over_dx;
    R v = sph_volume(P, th, hd);
    R mref;
    if (pt == 9) mref = (R)P.rho_liquid * v * pori;
    else if (pt == -3 || pt == 0 || pt == 3 || pt == 1) mref = (R)P.rho_gas * v * pori;
    else mref = (R)P.rho_liquid * v * pori;
    if (pt == 9 && zi < 0.05) mref = (R)P.rho_gas * v * pori;
    R rref = (P.dim == 2) ? mref / ((th / hd) * (th / hd)) : mref / v;
    W.rho_ref[i] = rref;
    R mn = mo, rn = ro;
    if (P.rho_type == 1) {
        rn = mref / v;
        mn = mref;
    }
    W.rho_new[i] = rn;
    W.m_new[i] = mn;
    rec.f1[i] = mk4<R>(mn, rn, S.temp[i], pori);
    const PosRec<R> q = ldr(rec.pos + i);
    rec.pb[i] = pv_make(q, pv_code<R>(mn / rn, q.w, pt == 1 || pt == 3));
    rec.rp[i] = pori * rn;
}

// contact history permutation, one thread per (slot, sphere): the writes of
// a slot plane are coalesced
__global__ void k_gather_history(int n, const int* __restrict__ perm, const int* __restrict__ hid_src,
                                 const double* __restrict__ hds_src, int* hid_dst, double* hds_dst) {
    grid_dep_wait();
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n * SPHDEM_NSLOT) return;
    int s = q / n, i = q - s * n;
    int p = perm[i];
    hid_dst[(size_t)s * n + i] = hid_src[(size_t)s * n + p];
#pragma unroll
    for (int c = 0; c < 3; c++) hds_dst[(size_t)(s * 3 + c) * n + i] = hds_src[(size_t)(s * 3 + c) * n + p];
}

// KERNEL_clc_prep3D_coupling_dem: functions_PREP2.cuh:3367-3523.
// One warp per DEM sphere; lanes stride over the candidate rows.
// G = 32: a warp per sphere; G = 1: a thread per sphere (2-D beds with many
// spheres); dem_thread_per_sphere in engine.cu.
template <typename R, int G>
__global__ void __launch_bounds__(128) k_dem_prep(DevParams P, SphState<R> S, SphRec<R> rec, DemState<double> D,
                                                  DemWork<double> DW, const int4* __restrict__ srows, const int4* __restrict__ drows) {
    static_assert(G == 32 || G == 1, "a warp or a thread per sphere");
    grid_dep_wait();
    const int i = G == 32 ? (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5)
                          : (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const int lane = G == 32 ? (int)(threadIdx.x & 31) : 0;
    __shared__ int s_rows[4][20];   // 128 threads = 4 warps
    int* sm = s_rows[threadIdx.x >> 5];
    if (i >= P.nd) return;
    if (D.itype[i] > 2) return;
    int pti = D.ptype[i];
    double xi = D.x[i], yi = D.y[i], zi = D.z[i], hi = D.h[i];
    R th = (R)hi;
    Knl<R> K = knl_make<R>(P, th);
    double Rr = P.kappa * hi;
    Band bd = make_band(P, Rr);
    float r2l = r2_lo(Rr), r2h = r2_hi(Rr);
    PosRec<R> qp = make_pos<R>(P, xi, yi, zi, 0, 0, 0);
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zi, ic, jc, kc);
    R f1 = 0, f3 = 0, por = 0;
    const Cull cu = make_cull(xi, yi, zi, Rr);
    // the sphere's SPH neighbours (p_type <= 1000, |x_i - x_j| < kappa h_i,
    // the add = 0 form that k_dem_coupling uses) into DW.nbs in visit order,
    // ranked by a ballot per round; the filter sums take their own subset
    // (p_type 1 or 3, the 1e-20 form)
    const unsigned lt = (1u << lane) - 1u;
    int cs = 0;
    auto dem_por = [&](int j) {
        if (D.ptype[j] <= 1000) return;
        PairT<R> g = pair_test<R>(xi, yi, zi, D.x[j], D.y[j], D.z[j], Rr, 1e-20, r2l, r2h);
        if (!g.in) return;
        R w = kw(K, g.r);
        R rj = (R)D.rad[j];
        por += w * dem_measure(P, rj);
    };
    if constexpr (G == 1) {
        // in visit order, one candidate after another
        for_stencil_j(P, ic, jc, kc, srows, cu, [&](int j) {
            const PosRec<R> qj = ldr(rec.pos + j);
            const int ptj = tag_ptype(qj.w);
            if (ptj > 1000) return;
            bool in = false, in20 = false;
            Disp<R> d;
            R r2 = 0;
            test_pair2(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, bd, d, r2, in, in20);
            if (in) {
                if (cs < DEM_SPH_CAP) DW.nbs[(size_t)i * DEM_SPH_CAP + cs] = j;
                cs++;
            }
            if (!in20 || (ptj != 1 && ptj != 3)) return;
            R r, rinv;
            rdist(r2, r, rinv);
            V2<R> mr = ldr(rec.mr0 + j);
            R c = mr.x * rcp(mr.y) * kw(K, r);
            if (ptj == 1) f1 += c;
            else f3 += c;
        });
        DW.ncs[i] = cs;
        for_stencil_j(P, ic, jc, kc, drows, cu, dem_por);
    } else {
    auto pos = [&](int j) { return ldr(rec.pos + j); };
    for_rows_warp_pre<PosRec<R>>(P, ic, jc, kc, srows, cu, sm, lane, pos, [&](int j, const PosRec<R>& qj) {
        bool in = false, in20 = false;
        int ptj = 0;
        Disp<R> d;
        R r2 = 0;
        if (j >= 0) {
            ptj = tag_ptype(qj.w);
            if (ptj <= 1000) test_pair2(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, bd, d, r2, in, in20);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int pos = cs + __popc(m & lt);
            if (pos < DEM_SPH_CAP) DW.nbs[(size_t)i * DEM_SPH_CAP + pos] = j;
        }
        cs += __popc(m);
        if (!in20 || (ptj != 1 && ptj != 3)) return;
        R r, rinv;
        rdist(r2, r, rinv);
        V2<R> mr = ldr(rec.mr0 + j);
        R c = mr.x * rcp(mr.y) * kw(K, r);
        if (ptj == 1) f1 += c;
        else f3 += c;
    });
    if (lane == 0) DW.ncs[i] = cs;
    for_rows_warp(P, ic, jc, kc, drows, cu, sm, lane, dem_por);
    f1 = warp_sum(f1);
    f3 = warp_sum(f3);
    por = warp_sum(por);
    }
    if (lane == 0 && pti > 1000) {
        DW.flt_s[i] = f3;
        DW.flt_sd[i] = f1;
        DW.flt_sd2[i] = f1;
        DW.DEMpor[i] = (R)1 - (por / (f3 + f1 + (R)1.0e-20));
    }
}

// The same for Wendland C2, a warp per sphere: the scan of the ~620 SPH
// stencil candidates only lists the ~60 within the radius, and the Shepard sums
// run over that list (two rounds of the warp); summing inside the scan ran the
// kernel in nearly every round with a few lanes on.  The porosity sum takes
// the spheres from k_dem_near's list where the kernel's radius lies inside its
// range.  78 -> 66 us on the bench bed, 0.66 -> 0.57 ms on
// 200,000 spheres: bound by the scan.  The list in shared memory is longer than
// the one k_dem_coupling reads, so that spheres with up to DEM_LIST SPH
// neighbours are scanned once (20,000 with 300 each: 180 us, 276 with a second
// scan, 196 summing inside the scan).
constexpr int DEM_LIST = 512;
template <typename R>
__global__ void __launch_bounds__(128) k_dem_prep_c2(DevParams P, SphState<R> S, SphRec<R> rec, DemState<double> D,
                                                     DemWork<double> DW, const int4* __restrict__ srows,
                                                     const int4* __restrict__ drows) {
    grid_dep_wait();
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    __shared__ int s_rows[4][20];
    __shared__ int s_list[4][DEM_LIST];
    int* sm = s_rows[threadIdx.x >> 5];
    int* list = s_list[threadIdx.x >> 5];
    if (i >= P.nd) return;
    const int it = D.itype[i];
    if (it > 2) return;
    const int pti = D.ptype[i];
    const double xi = D.x[i], yi = D.y[i], zi = D.z[i], hi = D.h[i], Rr = P.kappa * hi;
    const Knl<R, 3> K = knl_make<R, 3>(P, (R)hi);
    const Band bd = make_band(P, Rr);
    const PosRec<R> qp = make_pos<R>(P, xi, yi, zi, 0, 0, 0);
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zi, ic, jc, kc);
    const Cull cu = make_cull(xi, yi, zi, Rr);
    const unsigned lt = (1u << lane) - 1u;
    // the sphere's SPH neighbours (p_type <= 1000, the add = 0 form of the
    // predicate, which k_dem_coupling uses), in visit order
    int cs = 0;
    auto pos = [&](int j) { return ldr(rec.pos + j); };
    for_rows_warp_pre<PosRec<R>>(P, ic, jc, kc, srows, cu, sm, lane, pos, [&](int j, const PosRec<R>& qj) {
        bool in = false;
        if (j >= 0) {
            Disp<R> d;
            R r2;
            in = tag_ptype(qj.w) <= 1000 && test_pair(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, 0.0, bd, d, r2);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int pos = cs + __popc(m & lt);
            if (pos < DEM_LIST) list[pos] = j;
        }
        cs += __popc(m);
    });
    if (lane == 0) DW.ncs[i] = cs;
    __syncwarp();
    R f1 = 0, f3 = 0, por = 0;
    auto shep = [&](int j) {   // p_type 1 and 3, the 1e-20 form (add = 0 admits no other pair of non-zero weight)
        const PosRec<R> qj = ldr(rec.pos + j);
        const V2<R> mr = ldr(rec.mr0 + j);
        const int ptj = tag_ptype(qj.w);
        const Disp<R> d = disp_pt(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j);
        R r, rinv;
        rdist(d.dx * d.dx + d.dy * d.dy + d.dz * d.dz, r, rinv);
        const R c = mr.x * rcp(mr.y) * kw(K, r);
        f1 += ptj == 1 ? c : (R)0;
        f3 += ptj == 3 ? c : (R)0;
    };
    if (cs <= DEM_LIST) {
        int* __restrict__ nbs = DW.nbs + (size_t)i * DEM_SPH_CAP;
        for (int k = lane; k < cs; k += 32) {
            const int j = list[k];
            if (k < DEM_SPH_CAP) nbs[k] = j;
            shep(j);
        }
    } else {   // more than the list holds: the stencil again
        for_rows_warp(P, ic, jc, kc, srows, cu, sm, lane, [&](int j) {
            const PosRec<R> qj = ldr(rec.pos + j);
            Disp<R> d;
            R r2;
            if (tag_ptype(qj.w) <= 1000 && test_pair(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, 0.0, bd, d, r2)) shep(j);
        });
    }
    const float r2l = r2_lo(Rr), r2h = r2_hi(Rr);
    auto dem_por = [&](int j) {
        if (D.ptype[j] <= 1000) return;
        const PairT<R> g = pair_test<R>(xi, yi, zi, D.x[j], D.y[j], D.z[j], Rr, 1e-20, r2l, r2h);
        if (g.in) por += kw(K, g.r) * dem_measure(P, (R)D.rad[j]);
    };
    const int cd = it == 1 && pti > 1000 && Rr <= P.r_search * D.rad[i] ? DW.ncd[i] : DEM_DEM_CAP + 1;
    if (cd <= DEM_DEM_CAP) {
        // the list leaves out the sphere itself (and any at its very centre)
        const int* __restrict__ nbd = DW.nbd + (size_t)i * DEM_DEM_CAP;
        for (int k = lane; k < cd; k += 32) dem_por(__ldg(nbd + k));
        if (lane == 0) dem_por(i);
    } else {
        for_rows_warp(P, ic, jc, kc, drows, cu, sm, lane, dem_por);
    }
    f1 = warp_sum(f1);
    f3 = warp_sum(f3);
    por = warp_sum(por);
    if (lane == 0 && pti > 1000) {
        DW.flt_s[i] = f3;
        DW.flt_sd[i] = f1;
        DW.flt_sd2[i] = f1;
        DW.DEMpor[i] = (R)1 - (por / (f3 + f1 + (R)1.0e-20));
    }
}

// ---------------------------------------------------------------------------
// Sub-particle-scale eddy viscosity, the strain-rate branch of
// KERNEL_clc_prep3D_sph (functions_PREP2.cuh:2113-2118, 2166-2171), run
// with fv_solve and the SPS turbulence model only:
//   S_i = sum_j -m_j (rho_i + rho_j) |u_i - u_j|^2 / (2 rho_i rho_j r^2) (x_ij . grad W_ij)
// with the uncorrected kernel slope, and vis_t_i = (C_s L h_i)^2 max(S_i, 1e-20) rho_i
// (C_s = 0.12, L = 0.01, Parameters.cuh:102-104).  Pass B's viscous term
// reads vis_t of both particles of a pair, so this runs as its own pass
// just before it.
// ---------------------------------------------------------------------------
template <typename R, int KT>
__global__ void __launch_bounds__(128) k_sps(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    if (S.itype[i] > 2 || S.ptype[i] > 1000) {
        W.vist[i] = 0;
        return;
    }
    const SphRec<R> rec = W.rec;
    R th = (R)S.h[i];
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    PosRec<R> qi = ldr(rec.pos + i);
    V4<R> upi = rec.up[i];
    V4<R> fi = rec.f1[i];
    R uxi = upi.x, uyi = upi.y, uzi = upi.z, rhoi = fi.y;
    R irhoi = rcp(rhoi);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R sr = 0;
    nb_walk<4, NbQ44<R>>(
        cnt, W.nbr, n, i,
        [&](int j) {
            NbQ44<R> t;
            t.q = ldr(rec.pos + j);
            t.a = ldr(rec.f1 + j);
            t.b = ldr(rec.up + j);
            return t;
        },
        [&](int j, const NbQ44<R>& t) {
            Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
            R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
            rdist(r2, r, rinv);
            R dw = kdw(K, r) * rinv;
            R ux = uxi - t.b.x, uy = uyi - t.b.y, uz = uzi - t.b.z;
            R v = (R)-0.5 * t.a.x * (rhoi + t.a.y) * (ux * ux + uy * uy + uz * uz) * irhoi * rcp(t.a.y) * rinv * rinv;
            sr += v * r2 * dw;   // v (x_ij . x_ij) W'/r
        });
    sr = sr > (R)1e-20 ? sr : (R)1e-20;
    R cl = (R)0.12 * (th * (R)0.01);
    W.vist[i] = cl * cl * sr * rhoi;
}

// ---------------------------------------------------------------------------
// pass B: KERNEL_clc_prep3D_sph (functions_PREP2.cuh:1985-2227, Shepard
// filter) + KERNEL_advection_force3D_sph (functions_PPE2.cuh:1251-1607).
// The delta-SPH density gradient of prep3D is not formed: no kernel of the
// ISPH step reads it.
// ---------------------------------------------------------------------------
// The pair terms with G = dW/dr / r (C2Sum), d = x_i - x_j, V = m_j / rho_j,
// C the symmetric gradient correction and du = u_i - u_j:
//   pressure          (p_i + p_j) V G (C d)          C and factors after the loop
//   viscous           du V G c_v (d . C d) / r^2
//   Eulerian advection du V G (u_i . C d) = du V G (w . d), w = C u_i
// The viscous and advection sums share du, so a pair adds one scalar times
// du; heat conduction and advection share T_i - T_j the same way.  (The
// reference multiplies C into every pair's gradient and divides by r; that
// form took 118 instructions per pair, this one about 60.)
// The forces that need m_j and rho_j themselves (interface sharpness,
// repulsive boundary, SPS eddy viscosity, inter-particle surface tension,
// artificial viscosity) run in k_passB_any.  HEAT: conduction (con_solve).
template <typename R, bool HEAT>
__global__ void __launch_bounds__(128) k_passB(DevParams P, SphState<R> S, SphWork<R> W, const DevFlags* F) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    // Shepard filter every freq_filt*decouple_stride steps (functions_PREP2.cuh:2120)
    const int filt = (F->step_count % P.filt_period) == 0;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    W.ftx[i] = 0; W.fty[i] = 0; W.ftz[i] = 0; W.ftot[i] = 0;
    W.pgfx[i] = 0; W.pgfy[i] = 0; W.pgfz[i] = 0;
    W.dtemp[i] = 0;
    if (it > 2 || pt > 1000) return;
    bool adv = !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (!filt && !adv) return;
    R th = (R)S.h[i];
    const C2Sum<R> K = c2_sum<R>(P, th);
    const PvRec<R> qi = ldr(rec.pb + i);
    const bool slow_i = pv_vol(qi) != pv_vol(qi);
    V4<R> upi = rec.up[i];
    V4<R> fi = rec.f1[i];
    R uxi = upi.x, uyi = upi.y, uzi = upi.z, pi = upi.w;
    R rhoi = fi.y, tempi = fi.z, pori = fi.w;
    R irhoi = rcp(rhoi);
    const Cm6<R> C = cm6_load(W.Cm, n, i, P.kgc == 1);
    const R vis = (R)P.mu_gas, vis_h = (vis * vis) / (vis + vis), kc = (R)P.k_sph;
    // per-particle factors of the pair terms
    const R cv_i = P.fv ? vis_h * (R)4 * pori * irhoi : (R)0;
    const R ch_i = (R)4 * pori * kc * kc * irhoi / (kc + kc) / (R)P.cp_sph * (R)(pt != -1);
    Disp<R> w = cm6_mul(C, uxi, uyi, uzi);
    if (P.sph_lagrangian) w = Disp<R>{0, 0, 0};
    int cnt = min(W.ncnt[i], P.nb_cap);
    R flt = 0, tx = 0, ty = 0, tz = 0, px = 0, py = 0, pz = 0, et = 0;
    const int* __restrict__ nb = W.nbr;
    using Rec = std::conditional_t<HEAT, NbP4S<R>, NbP4<R>>;
    if (!adv) {   // a filter step of a row without forces: the Shepard sum alone
        nb_sum<NbP<R>, PairV<R>>(
            cnt, nb, n, i, [&](int j) { return NbP<R>{ldr(rec.pb + j)}; },
            [&](const NbP<R>& t, PairV<R>& g) { return pv_prep<R, false>(P, qi, slow_i, t.q, g); },
            [&](int j, NbP<R>& t, PairV<R>& g) {
                int tag;
                pv_fix(S, rec.pos, W.m_new, W.rho_new, slow_i, t.q, i, j, g, tag);
            },
            [&](int, const NbP<R>&, const PairV<R>& g) {
                const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
                flt += g.vs * c2_w(K, r2 * rsq_floor(r2));
            });
        S.flt_s[i] = flt * K.wn;
        return;
    }
    nb_sum<Rec, PairV<R>>(
        cnt, nb, n, i,
        [&](int j) {
            Rec t;
            t.q = ldr(rec.pb + j);
            t.b = ldr(rec.up + j);
            if constexpr (HEAT) t.s = ldr(S.temp + j);
            return t;
        },
        [&](const Rec& t, PairV<R>& g) { return pv_prep<R, false>(P, qi, slow_i, t.q, g); },
        [&](int j, Rec& t, PairV<R>& g) {
            int tag;
            if (!pv_fix(S, rec.pos, W.m_new, W.rho_new, slow_i, t.q, i, j, g, tag) || tag_ptype(tag) < 1000) return;
            // not a neighbour of the forces; the filter counts its volume
            g.v = 0;
            t.b = mk4<R>(uxi, uyi, uzi, pi);
            if constexpr (HEAT) t.s = tempi;
        },
        [&](int, const Rec& t, const PairV<R>& g) {
            const V4<R>& uj = t.b;
            const R v = g.v;
            const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
            const R rinv = rsq_floor(r2), r = r2 * rinv;
            if (filt) flt += g.vs * c2_w(K, r);
            const R G = c2_g(K, r), vg = v * G;
            const R s = vg * (pi + uj.w);
            px += s * g.dx;
            py += s * g.dy;
            pz += s * g.dz;
            const R dux = uxi - uj.x, duy = uyi - uj.y, duz = uzi - uj.z;
            const Disp<R> y = cm6_mul(C, g.dx, g.dy, g.dz);
            const R quad = g.dx * y.dx + g.dy * y.dy + g.dz * y.dz;
            const R wd = w.dx * g.dx + w.dy * g.dy + w.dz * g.dz;
            const R a = vg * (cv_i * quad * rinv * rinv + wd);
            tx += a * dux;
            ty += a * duy;
            tz += a * duz;
            if constexpr (HEAT) et += vg * (ch_i * r * rcp(r + (R)1e-10) + wd) * (tempi - t.s);
        });
    if (filt) S.flt_s[i] = flt * K.wn;
    tx *= K.gn;
    ty *= K.gn;
    tz *= K.gn;
    if (P.fg) tz += -(R)P.g_sph;
    W.ftx[i] = tx;
    W.fty[i] = ty;
    W.ftz[i] = tz;
    W.ftot[i] = sqrt(tx * tx + ty * ty + tz * tz);
    if (P.fp) {
        // rho_i/eps_i * (-eps_i / rho_i) and the kernel's factor
        const R cp = -pori * irhoi * (rhoi / pori) * K.gn;
        const Disp<R> a = cm6_mul(C, px, py, pz);
        W.pgfx[i] = cp * a.dx;
        W.pgfy[i] = cp * a.dy;
        W.pgfz[i] = cp * a.dz;
    }
    if (HEAT) W.dtemp[i] = et * K.gn;
}

// ---------------------------------------------------------------------------
// The spheres within the search range of each sphere (r_search r_i, the
// candidates of KERNEL_DEM_interaction3D_dem), in visit order, for
// k_dem_contact.  A warp per sphere scans the stencil's ~160 slots and keeps
// ~18: the contact pass then runs its pair terms (about 450 instructions) over
// the short list only, with 8 lanes per sphere; scanning and summing in one
// warp-per-sphere kernel ran them with 11 of 32 lanes busy at 128 registers.
// The squared distance decides outside a band of 4e-15 around the range (its
// FP64 rounding is below 1e-15), the reference's square root inside it.
// ncd holds the exact count; a sphere with more than the list holds is walked
// by its stencil.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_dem_near(DevParams P, DemState<double> D, DemWork<double> DW,
                                                  const int4* __restrict__ drows) {
    grid_dep_wait();
    const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    __shared__ int s_rows[4][20];
    if (i >= P.nd || D.itype[i] != 1 || D.ptype[i] <= 1000) return;
    const double xi = D.x[i], yi = D.y[i], zi = D.z[i], R = P.r_search * D.rad[i];
    const double lo = R * R * (1.0 - 4e-15), hi = R * R * (1.0 + 4e-15);
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zi, ic, jc, kc);
    const unsigned lt = (1u << lane) - 1u;
    int c = 0;
    struct Cand {
        Dbl4 a;
        int pt;
    };
    auto load = [&](int j) { return Cand{ldr(DW.ra + j), __ldg(D.ptype + j)}; };
    for_rows_warp_pre<Cand>(P, ic, jc, kc, drows, make_cull(xi, yi, zi, R), s_rows[threadIdx.x >> 5], lane, load,
                            [&](int j, const Cand& q) {
        bool in = false;
        if (j >= 0 && q.pt > 1000) {
            const double xj = q.a.x, yj = q.a.y, zj = q.a.z;
            const double dx = xi - xj, dy = yi - yj, dz = zi - zj, d2 = dx * dx + dy * dy + dz * dz;
            in = d2 < lo;
            if (!in && !(d2 > hi)) in = pair_dist(xi, yi, zi, xj, yj, zj) < R;
            in = in && d2 > 0.0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int pos = c + __popc(m & lt);
            if (pos < DEM_DEM_CAP) DW.nbd[(size_t)i * DEM_DEM_CAP + pos] = j;
        }
        c += __popc(m);
    });
    if (lane == 0) DW.ncd[i] = c;
}

// ---------------------------------------------------------------------------
// DEM contact: KERNEL_DEM_interaction3D_dem (functions_DEM_INTERACTION2.cuh:
// 888-1766).  The history lookup compares against the start-of-step slot
// ids held in registers; inserts pick the first slot that was free at the
// start of the step (so two new partners in one step share a slot, as in
// the reference).  Spring increments and overlap are FP64.
// ---------------------------------------------------------------------------
// G = 8: eight lanes per sphere over the list of k_dem_near; G = 1: one
// thread per sphere over its stencil in visit order (2-D beds with many
// spheres: a few candidates, which a warp would leave mostly idle).  The
// launch picks G from the configuration (dem_thread_per_sphere in engine.cu),
// so a bed always runs one form.
template <typename R, int G>
// 4 blocks of 128 per SM (128 registers)
__global__ void __launch_bounds__(128, 4) k_dem_contact(DevParams P, DemState<double> D, DemWork<double> DW,
                                                     const int4* __restrict__ drows,
                                                     DevFlags* F) {
    static_assert(G == 8 || G == 1, "eight lanes or a thread per sphere");
    grid_dep_wait();
    // G = 8: lanes take entries l, l+8, ... of the list, which is in visit
    // order, and the pair terms are reduced with shuffles.
    // History writes keep the sequential semantics: lookups use the
    // start-of-step ids, a release clears only the partner's own slot, and
    // every new contact targets the first slot free at the start of the
    // step, so the new contact visited last wins that slot.
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int lane = (int)(threadIdx.x % G);
    const unsigned gm = G == 1 ? 0u : ((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));   // the group's lanes
    const int n = P.nd;
    if (i >= n) return;
    if (lane == 0) {
        DW.ftx[i] = 0; DW.fty[i] = 0; DW.ftz[i] = 0;
        DW.tqx[i] = 0; DW.tqy[i] = 0; DW.tqz[i] = 0;
        DW.dtemp[i] = 0; DW.dtemp1[i] = 0; DW.dtemp2[i] = 0; DW.dtemp3[i] = 0;
    }
    if (D.itype[i] != 1 || D.ptype[i] <= 1000) return;
    // the contact mechanics run in FP64 in both builds (the state is FP64 and
    // stiff colliding contacts amplify rounding; 0.01 ms per step against R);
    // the radiation heat rate below is formed in R
    using Q = double;
    double xi = D.x[i], yi = D.y[i], zi = D.z[i], radi = D.rad[i];
    Q uxi = D.ux[i], uyi = D.uy[i], uzi = D.uz[i], wxi = D.wx[i], wyi = D.wy[i], wzi = D.wz[i];
    Q mi = D.m[i], rii = D.ri[i], rhoi = D.rho[i], tempi = D.temp[i];
    Q pri = (Q)P.nu_p, Gi = (Q)P.G, ymi = Gi * ((Q)2 * ((Q)1 + pri));
    Q ymij = (Q)1 / ((((Q)1 - pri * pri) / ymi) + (((Q)1 - pri * pri) / ymi));
    Q Gij = (Q)1 / ((((Q)2 - pri) / Gi) + (((Q)2 - pri) / Gi));
    Q cdamp = sqrt((Q)3.333333333) * (Q)P.damp;
    Q kci = (Q)P.k_dem, cpi = (Q)P.cp_dem;
    const R tiR = (R)tempi;
    const R emiR = (tiR >= (R)700) ? ((R)0.505586 + (R)7.92943e-4 * tiR - (R)5.228643e-7 * tiR * tiR +
                                      (R)1.10479e-10 * tiR * tiR * tiR)
                                   : (R)0.842337;
    Q radiR = (Q)radi;
    const Q imi = (Q)1 / mi, iradi = (Q)1 / radiR;   // hoisted reciprocals of the sphere's own terms
    Q dr2 = ((Q)1 / (Q)6) * radiR;
    Q volm = ((Q)4 / (Q)3) * (Q)3.141592 * (radiR * radiR * radiR - (radiR - dr2) * (radiR - dr2) * (radiR - dr2));
    int oid[SPHDEM_NSLOT];
    int free_slot = -1;
#pragma unroll
    for (int s = 0; s < SPHDEM_NSLOT; s++) {
        oid[s] = D.hid[s * n + i];
        if (free_slot < 0 && oid[s] < 1) free_slot = s;
    }
    // every lane of the group holds the start-of-step ids before one releases a slot
    if constexpr (G > 1) __syncwarp(gm);
    Q tx = 0, ty = 0, tz = 0, tqx = 0, tqy = 0, tqz = 0, dtr = 0, dtc = 0;
    const double kdt = P.dt;
    // this lane's last new contact (visit order t) and its spring
    int new_t = -1, new_id = 0;
    double new_dx = 0, new_dy = 0, new_dz = 0;
    int t_visit = -1;   // place of the pair in visit order
    auto pair = [&](int j) {
        if (G == 1) t_visit++;
        if (D.ptype[j] <= 1000) return;
        double xj = D.x[j], yj = D.y[j], zj = D.z[j], radj = D.rad[j];
        double td = pair_dist(xi, yi, zi, xj, yj, zj);
        if (!(td < P.r_search * radi && td > 0.0)) return;
        double ovlp = radi + radj - td;
        int demj = D.dem_idx[j];
        Q radjR = (Q)radj;
        Q radij = (Q)1 / (iradi + (Q)1 / radjR);
        Q tdR = (Q)td;
        if (P.con) {
            // radiation between spheres within the search range (functions_DEM_INTERACTION2.cuh:
            // 1080-1194): a heat rate, formed in the field precision R
            const R ti = (R)tempi, tj = (R)D.temp[j];
            const R riR = (R)radiR, rjR = (R)radjR, rijR = (R)radij, tdF = (R)tdR;
            R emj = (tj >= (R)700) ? ((R)0.505586 + (R)7.92943e-4 * tj - (R)5.228643e-7 * tj * tj +
                                      (R)1.10479e-10 * tj * tj * tj)
                                   : (R)0.842337;
            const R itdF = rcp(tdF);
            R ai = riR * itdF, aj = rjR * itdF, dij = aj - ai;
            R dc_r = (R)0.56 * ((R)2 * rijR);
            R dc_ar = (R)3.14159 * dc_r * dc_r;
            R dmax = (R)0.5 * (sqrt((R)1 + (R)4 * dc_ar / ((R)3.14159 * tdF * tdF * ((R)1 - dij * dij))) - dij);
            R ci = ((R)1 - dij * dij) / ((R)2 * dmax) - dij;
            R cj = ((R)1 - dij * dij) / ((R)2 * (dmax + dij)) + dij;
            R si = sqrt((R)1 - ci * ci), sj = sqrt((R)1 - cj * cj);
            R ri_cr = riR * si, rj_cr = rjR * sj;
            R td_cr = tdF - riR * ci - rjR * cj;
            R z_cr = (R)1 + ((R)4 * rj_cr * rj_cr + td_cr * td_cr) / (ri_cr * ri_cr);
            R F_cr = (R)0.5 * (z_cr - sqrt(z_cr * z_cr - (R)4 * rj_cr * rj_cr / (ri_cr * ri_cr)));
            R F_ij = ((R)1 + ci) * F_cr * (R)0.5;
            R ar_i = (R)2 * (R)3.14159 * riR * riR * ((R)1 - ci);
            R ar_j = (R)2 * (R)3.14159 * rjR * rjR * ((R)1 - cj);
            R arr = ar_j / ar_i;
            R Y = F_ij + ((R)1 - F_ij) * (arr / ((R)1 + arr));
            R einv = ((R)1 - emiR) / (emiR * ar_i) + ((R)1 - emj) / (emj * ar_j) + (R)1 / (Y * ar_i);
            // Ti^4 - Tj^4; in FP32 as (Ti - Tj)(Ti + Tj)(Ti^2 + Tj^2), which keeps the
            // relative precision of a difference of nearly equal temperatures
            R d4;
            if constexpr (sizeof(R) == 4) d4 = (ti - tj) * (ti + tj) * (ti * ti + tj * tj);
            else d4 = ti * ti * ti * ti - tj * tj * tj * tj;
            dtr += (Q)(-(R)5.6704e-8 * d4 / (einv * ((R)rhoi * (R)volm) * (R)cpi));
        }
        if (!(td < P.r_contact * radi)) return;
        int slot = -1;
#pragma unroll
        for (int s = 0; s < SPHDEM_NSLOT; s++)
            if (slot < 0 && oid[s] == demj) slot = s;
        if (td > 0 && ovlp > 0) {
            Q tov = (Q)ovlp;
            if (P.con) {
                Q kij = (Q)1 / ((Q)1 / kci + (Q)1 / kci);
                dtc += -(Q)4 * kij * sqrt(((Q)2 * tov) * (radij - (Q)0.5 * tov)) * (tempi - D.temp[j]) /
                       ((rhoi * volm) * cpi);
            }
            double dsx = 0, dsy = 0, dsz = 0;
            if (slot >= 0) {
                dsx = D.hds[(slot * 3 + 0) * n + i];
                dsy = D.hds[(slot * 3 + 1) * n + i];
                dsz = D.hds[(slot * 3 + 2) * n + i];
            }
            Q mj = D.m[j];
            const Q itd = (Q)1 / (Q)td;
            Q nx = (Q)(xj - xi) * itd, ny = (Q)(yj - yi) * itd, nz = (Q)(zj - zi) * itd;
            Q li = radiR - (Q)0.5 * tov, lj = radjR - (Q)0.5 * tov;
            Q rcxi = li * nx, rcyi = li * ny, rczi = li * nz;
            Q rcxj = -lj * nx, rcyj = -lj * ny, rczj = -lj * nz;
            Q wxj = D.wx[j], wyj = D.wy[j], wzj = D.wz[j];
            Q urxi = wyi * rczi - wzi * rcyi, uryi = wzi * rcxi - wxi * rczi, urzi = wxi * rcyi - wyi * rcxi;
            Q urxj = wyj * rczj - wzj * rcyj, uryj = wzj * rcxj - wxj * rczj, urzj = wxj * rcyj - wyj * rcxj;
            Q urx = (D.ux[j] + urxj) - (uxi + urxi);
            Q ury = (D.uy[j] + uryj) - (uyi + uryi);
            Q urz = (D.uz[j] + urzj) - (uzi + urzi);
            Q unm = nx * urx + ny * ury + nz * urz;
            Q unx = unm * nx, uny = unm * ny, unz = unm * nz;
            Q usx = urx - unx, usy = ury - uny, usz = urz - unz;
            dsx += (double)usx * kdt;
            dsy += (double)usy * kdt;
            dsz += (double)usz * kdt;
            const Q iusm = (Q)1 / (sqrt(usx * usx + usy * usy + usz * usz) + (Q)1e-20);
            Q sx = usx * iusm, sy = usy * iusm, sz = usz * iusm;
            Q mij = (Q)1 / (imi + (Q)1 / mj);
            Q sq = sqrt(radij * tov);   // sqrt(R* delta): also stands for sqrt(R*) sqrt(delta)
            Q Cspr = (Q)1.33333 * ymij * sq * tov * imi;
            Q Cspr_s = (Q)8 * Gij * sq * imi;
            Q Kn = (Q)2 * ymij * sq;
            Q Cd = cdamp * sqrt(mij * Kn) * imi;
            Q Cds = cdamp * sqrt(mij * Cspr_s * mi) * imi;
            tx += Cspr * -nx;
            ty += Cspr * -ny;
            tz += Cspr * -nz;
            tx += Cd * unx;
            ty += Cd * uny;
            tz += Cd * unz;
            Q fssx = Cspr_s * (Q)dsx + Cds * usx;
            Q fssy = Cspr_s * (Q)dsy + Cds * usy;
            Q fssz = Cspr_s * (Q)dsz + Cds * usz;
            Q sgx = (fssx >= (Q)0) ? (Q)1 : (Q)-1;
            Q sgy = (fssy >= (Q)0) ? (Q)1 : (Q)-1;
            Q sgz = (fssz >= (Q)0) ? (Q)1 : (Q)-1;
            // stick while |f_spring| < |f_friction| (the squares compare the same way)
            Q mfss2 = fssx * fssx + fssy * fssy + fssz * fssz;
            Q fr = (Q)P.fric * Cspr;
            Q ffx = fr * sx, ffy = fr * sy, ffz = fr * sz;
            Q mfsf2 = ffx * ffx + ffy * ffy + ffz * ffz;
            bool stick = mfss2 < mfsf2;
            Q fsx = stick ? fssx : sgx * fabs(ffx);
            Q fsy = stick ? fssy : sgy * fabs(ffy);
            Q fsz = stick ? fssz : sgz * fabs(ffz);
            tx += fsx;
            ty += fsy;
            tz += fsz;
            tqx += mi * (rcyi * fsz - rczi * fsy);
            tqy += mi * (rczi * fsx - rcxi * fsz);
            tqz += mi * (rcxi * fsy - rcyi * fsx);
            if (slot >= 0) {
                // existing partner: its own slot, no other pair touches it
                D.hid[slot * n + i] = demj;
                D.hds[(slot * 3 + 0) * n + i] = dsx;
                D.hds[(slot * 3 + 1) * n + i] = dsy;
                D.hds[(slot * 3 + 2) * n + i] = dsz;
            } else {
                new_t = t_visit;
                new_id = demj;
                new_dx = dsx;
                new_dy = dsy;
                new_dz = dsz;
            }
        } else if (slot >= 0) {
            D.hds[(slot * 3 + 0) * n + i] = 0.0;
            D.hds[(slot * 3 + 1) * n + i] = 0.0;
            D.hds[(slot * 3 + 2) * n + i] = 0.0;
            D.hid[slot * n + i] = 0;
        }
    };
    const int cd = G == 1 ? 0 : DW.ncd[i];
    if (G > 1 && cd <= DEM_DEM_CAP) {
        const int* __restrict__ nbd = DW.nbd + (size_t)i * DEM_DEM_CAP;
        for (int k = lane; k < cd; k += G) {
            t_visit = k;
            pair(__ldg(nbd + k));
        }
    } else {
        int ic, jc, kc, t = 0;
        cell_ijk(P, xi, yi, zi, ic, jc, kc);
        for_stencil_j(P, ic, jc, kc, drows, make_cull(xi, yi, zi, P.r_search * radi), [&](int j) {
            if constexpr (G == 1) {
                pair(j);
            } else {
                if (t % G == lane) {
                    t_visit = t;
                    pair(j);
                }
                t++;
            }
        });
    }
    // the new contact visited last takes the first slot free at the start
    int last_t = new_t;
    if constexpr (G > 1) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) last_t = max(last_t, __shfl_xor_sync(gm, last_t, o));
    }
    if (last_t >= 0 && new_t == last_t) {
        // no free slot (a 17th partner): flag it; the new contact acted this
        // step and is not recorded (the reference writes through an unset
        // slot index here, functions_DEM_INTERACTION2.cuh:1567)
        const int slot = free_slot;
        if (slot < 0) {
            atomicOr(&F->overflow, 2);
        } else {
            D.hid[slot * n + i] = new_id;
            D.hds[(slot * 3 + 0) * n + i] = new_dx;
            D.hds[(slot * 3 + 1) * n + i] = new_dy;
            D.hds[(slot * 3 + 2) * n + i] = new_dz;
        }
    }
    if constexpr (G > 1) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            tx += __shfl_xor_sync(gm, tx, o); ty += __shfl_xor_sync(gm, ty, o); tz += __shfl_xor_sync(gm, tz, o);
            tqx += __shfl_xor_sync(gm, tqx, o); tqy += __shfl_xor_sync(gm, tqy, o); tqz += __shfl_xor_sync(gm, tqz, o);
            dtr += __shfl_xor_sync(gm, dtr, o); dtc += __shfl_xor_sync(gm, dtc, o);
        }
    }
    if (lane != 0) return;
    if (P.fg) tz += -(Q)P.g_dem;
    if (P.con) {
        Q temp1i = D.temp1[i], temp2i = D.temp2[i], temp3i = D.temp3[i];
        Q a0 = kci / (rhoi * cpi);
        Q dr1 = ((Q)5 / (Q)6) * radiR / (Q)3;
        Q A = ((Q)2 * kci / dr1) / ((Q)2 * kci / dr1 + kci / dr2), B = (Q)1 - A;
        Q ts = A * temp1i + B * tempi;
        Q d0 = (Q)2 * (a0 / radiR) * (tempi - ts) / ((Q)2 * dr2) + a0 * (tempi - (Q)2 * tempi + ts) / (dr2 * dr2);
        Q d1 = ((Q)2 * a0 / ((Q)2.5 * dr1)) * ((Q)2 * ts - temp1i - temp2i) / ((Q)2 * dr1) +
               a0 * ((Q)2 * ts - (Q)3 * temp1i + temp2i) / (dr1 * dr1);
        Q d2 = (Q)2 * (a0 / ((Q)1.5 * dr1)) * (temp1i - temp3i) / ((Q)2 * dr1) +
               a0 * (temp1i - (Q)2 * temp2i + temp3i) / (dr1 * dr1);
        Q d3 = (Q)2 * (a0 / ((Q)0.5 * dr1)) * ((temp2i - temp3i) / ((Q)2 * dr1)) + a0 * (temp2i - temp3i) / (dr1 * dr1);
        DW.dtemp[i] = d0 + dtr + dtc;
        DW.dtemp1[i] = d1;
        DW.dtemp2[i] = d2;
        DW.dtemp3[i] = d3;
    }
    DW.ftx[i] = tx;
    DW.fty[i] = ty;
    DW.ftz[i] = tz;
    DW.tqx[i] = tqx / rii;
    DW.tqy[i] = tqy / rii;
    DW.tqz[i] = tqz / rii;
}

// ---------------------------------------------------------------------------
// KERNEL_DEM_coupling3D_dem (functions_SPH_DEM_COUPLING2.cuh:627-1129) with
// KERNEL_clc_projection_dem (functions_TIME_ISPH2.cuh:206-308) fused into its
// epilogue (the predictor only needs this particle's force).  The pair sums
// of one sphere over its SPH neighbours (dc_pair) are formed by a warp --
// lanes over the candidates, partial sums reduced with shuffles -- and one
// lane runs the drag closure and the predictor (dem_coupling_finish).
// ---------------------------------------------------------------------------
template <typename R>
struct DcSums {
    R tx, ty, tz, ufx, ufy, ufz, uax, uay, uaz, por, ttf, tta;
    R wtf, wta;   // the weights of ttf/tta: their SPH temperatures are stored as T - t_ref
    int has_f, has_a;
};

// one SPH neighbour j of sphere i at distance r (the pair already passed the
// kappa h_i test): Shepard sums of fluid/air velocity, temperature and
// porosity, and the pressure-gradient force
template <typename R, int KT>
__device__ __forceinline__ void dc_pair_at(const Knl<R, KT>& K, R ff, R fa, R pgc, const V4<R>& fj, const V4<R>& uj,
                                           R gx, R gy, R gz, int ptj, R r, DcSums<R>& a) {
    const R porj = fj.w;
    if (!(porj < (R)1)) return;
    R w = kw(K, r);
    R mj = fj.x, rhoj = fj.y, c = mj * w * rcp(rhoj);
    if ((ptj == 1 && ff > (R)0.000001) || (ptj == 3 && fa > (R)0.000001)) {
        if (ptj == 1) {
            a.has_f = 1;
            a.ufx += uj.x * c; a.ufy += uj.y * c; a.ufz += uj.z * c;
            a.ttf += fj.z * c;
            a.wtf += c;
        } else {
            a.has_a = 1;
            a.uax += uj.x * c; a.uay += uj.y * c; a.uaz += uj.z * c;
            a.tta += fj.z * c;
            a.wta += c;
        }
        a.por += porj * c;
    }
    if (ptj != 0 && ptj != 9 && ptj != -3 && ptj != 3 && ff > (R)0.01) {
        R q = c * pgc;
        a.tx += gx * q;
        a.ty += gy * q;
        a.tz += gz * q;
    }
}
template <typename R, int KT>
__device__ __forceinline__ void dc_pair(const SphWork<R>& W, const Knl<R, KT>& K, R ff, R fa, R pgc, int j, int ptj, R r,
                                        DcSums<R>& a) {
    const V4<R> fj = ldr(W.rec.f1 + j);
    const R porj = fj.w;
    if (!(porj < (R)1)) return;
    R w = kw(K, r);
    R mj = fj.x, rhoj = fj.y, c = mj * w * rcp(rhoj);
    if ((ptj == 1 && ff > (R)0.000001) || (ptj == 3 && fa > (R)0.000001)) {
        V4<R> uj = ldr(W.rec.up + j);
        if (ptj == 1) {
            a.has_f = 1;
            a.ufx += uj.x * c; a.ufy += uj.y * c; a.ufz += uj.z * c;
            a.ttf += fj.z * c;
            a.wtf += c;
        } else {
            a.has_a = 1;
            a.uax += uj.x * c; a.uay += uj.y * c; a.uaz += uj.z * c;
            a.tta += fj.z * c;
            a.wta += c;
        }
        a.por += porj * c;
    }
    if (ptj != 0 && ptj != 9 && ptj != -3 && ptj != 3 && ff > (R)0.01) {
        R q = c * pgc;
        a.tx += W.pgfx[j] * q;
        a.ty += W.pgfy[j] * q;
        a.tz += W.pgfz[j] * q;
    }
}

template <typename R>
__device__ __forceinline__ void dc_warp_sum(DcSums<R>& a) {
    a.tx = warp_sum(a.tx); a.ty = warp_sum(a.ty); a.tz = warp_sum(a.tz);
    a.ufx = warp_sum(a.ufx); a.ufy = warp_sum(a.ufy); a.ufz = warp_sum(a.ufz);
    a.uax = warp_sum(a.uax); a.uay = warp_sum(a.uay); a.uaz = warp_sum(a.uaz);
    a.por = warp_sum(a.por); a.ttf = warp_sum(a.ttf); a.tta = warp_sum(a.tta);
    a.wtf = warp_sum(a.wtf); a.wta = warp_sum(a.wta);
    a.has_f = __any_sync(0xffffffffu, a.has_f);
    a.has_a = __any_sync(0xffffffffu, a.has_a);
}

// drag closure on the reduced sums (when coupled) and the DEM predictor
template <typename R>
__device__ void dem_coupling_finish(const DevParams& P, DemState<double>& D, DemWork<double>& DW, int i, bool coupled,
                                    const DcSums<R>& a) {
    using Q = double;   // the DEM set is FP64: the closure and the predictor run in FP64
    const int pt = D.ptype[i];
    Q uxi = D.ux[i], uyi = D.uy[i], uzi = D.uz[i];
    Q ftx = DW.ftx[i], fty = DW.fty[i], ftz = DW.ftz[i];
    if (coupled) {
        Q radi = (Q)D.rad[i], di = (Q)2 * radi;
        Q mi = D.m[i], rhoi = D.rho[i], tempi = D.temp[i];
        Q fa = DW.flt_s[i], ff = DW.flt_sd[i];
        const Q tx = a.tx, ty = a.ty, tz = a.tz, ufx = a.ufx, ufy = a.ufy, ufz = a.ufz;
        const Q uax = a.uax, uay = a.uay, uaz = a.uaz, por = a.por, ttf = a.ttf, tta = a.tta;
        const int has_f = a.has_f, has_a = a.has_a;
        Q rho_f = has_f ? (Q)P.rho_gas : (Q)0, rho_a = has_a ? (Q)P.rho_gas : (Q)0;
        Q ki = (radi < (Q)0.0012) ? (Q)55.0 : (Q)0.84;
        Q ali = (radi < (Q)0.0012) ? (Q)1.77e-5 : (Q)2.5e-6;
        Q cpi = ki / (ali * rhoi);
        Q eps = (Q)1.0e-15;
        Q pori = por / (ff + eps);
        Q ux_f = ufx / (ff + eps) - uxi, uy_f = ufy / (ff + eps) - uyi, uz_f = ufz / (ff + eps) - uzi;
        // the SPH temperatures in ttf/tta are stored as T - t_ref: absolute sums
        const Q tr = (Q)P.t_ref;
        const Q ttfa = ttf + tr * (Q)a.wtf, ttaa = tta + tr * (Q)a.wta;
        Q tf = ttfa / (ff + eps) - tempi;
        Q ux_a = uax / (fa + eps) - uxi, uy_a = uay / (fa + eps) - uyi, uz_a = uaz / (fa + eps) - uzi;
        Q ta = ttaa / (fa + eps) - tempi;
        Q ux_fa = (ufx + uax) / (ff + fa + eps) - uxi, uy_fa = (ufy + uay) / (ff + fa + eps) - uyi,
          uz_fa = (ufz + uaz) / (ff + fa + eps) - uzi;
        Q tfa = (ttfa + ttaa) / (ff + fa + eps) - tempi;
        Q f_fluid = ff / (ff + fa + eps), f_air = fa / (ff + fa + eps);
        Q mf = sqrt(ux_f * ux_f + uy_f * uy_f + uz_f * uz_f);
        DW.magf[i] = mf;
        Q ma = sqrt(ux_a * ux_a + uy_a * uy_a + uz_a * uz_a);
        Q mfa = sqrt(ux_fa * ux_fa + uy_fa * uy_fa + uz_fa * uz_fa);
        Q dfx = 0, dfy = 0, dfz = 0, dax = 0, day = 0, daz = 0, dq = 0;
        Q a_ht = (Q)6 / di;
        Q nu = (Q)P.nu_gas;
        DW.DEMpor[i] = pori;
        // the Di Felice closure (functions_SPH_DEM_COUPLING2.cuh:979-1009) in the
        // field precision R: an empirical coefficient, applied to the FP64 slip
        const R diR = (R)di, poriR = (R)pori, miR = (R)mi, nuR = (R)nu, epsR = (R)1.0e-15;
        const R mfR = (R)mf, maR = (R)ma, mfaR = (R)mfa, kiR = (R)ki, ahtR = (R)a_ht;
        if (mf > (Q)1.0e-8 && (ff + fa) > (Q)0.00001 && f_fluid > (Q)0.65) {
            R Re = diR * mfR * poriR / (nuR + epsR);
            R q = (R)0.63 + (R)4.8 / sqrt(Re);
            R Cdf = q * q;
            R lr = (R)1.5 - log10(Re);
            R bf = (R)3.7 - (R)0.65 * exp(-lr * lr / (R)2);
            R c = ((R)1 / (R)8) * Cdf * (R)rho_f * (R)3.14159 * diR * diR * mfR * pow(poriR, (R)2 - bf) / miR;
            dfx = c * ux_f; dfy = c * uy_f; dfz = c * uz_f;
            dq = (Q)(((R)2 + (R)0.6 * sqrt(Re)) * (R)0.0518 / diR * ahtR) * tf;
            D.Fdx_df[i] = dfx;
            D.Fdy_df[i] = dfy;
            D.Fdz_df[i] = dfz;
        }
        if (ma > (Q)1.0e-8 && (ff + fa) > (Q)0.00001 && f_air > (Q)0.65) {
            R Re = diR * poriR * maR / (nuR + epsR);
            R q = (R)0.63 + (R)4.8 / sqrt(Re);
            R lr = (R)1.5 - log10(Re);
            R b = (R)2.65 * ((R)1 + poriR) - ((R)5.3 - (R)3.5 * poriR) * poriR * poriR * exp(-lr * lr / (R)2);
            R c = ((R)1 / (R)8) * q * q * (R)rho_a * (R)3.14159 * diR * diR * maR * pow(poriR, (R)-1 - b) / miR;
            dax = c * ux_a; day = c * uy_a; daz = c * uz_a;
            dq = (Q)(((R)2 + (R)0.6 * sqrt(Re)) * kiR / diR * ahtR) * ta;
        }
        if ((ma > (Q)1.0e-8 || mf > (Q)1.0e-8) && (ff + fa) > (Q)0.00001 && f_air <= (Q)0.65 && f_fluid <= (Q)0.65) {
            R rfa = (R)P.rho_gas * (R)f_air + (R)P.rho_liquid * (R)f_fluid;
            R vfa = (R)P.mu_gas * (R)f_air + (R)P.mu_liquid * (R)f_fluid;
            R vk = vfa / (rfa + epsR);
            R Re = diR * poriR * mfaR / (vk + epsR);
            R q = (R)0.63 + (R)4.8 / sqrt(Re);
            R lr = (R)1.5 - log10(Re);
            R b = (R)2.65 * ((R)1 + poriR) - ((R)5.3 - (R)3.5 * poriR) * poriR * poriR * exp(-lr * lr / (R)2);
            R c = ((R)1 / (R)8) * q * q * rfa * (R)3.14159 * diR * diR * mfaR * pow(poriR, (R)-1 - b) / miR;
            dax = c * ux_fa; day = c * uy_fa; daz = c * uz_fa;
            dq = (Q)(((R)2 + (R)0.6 * sqrt(Re)) * kiR / diR * ahtR) * tfa;
        }
        ftx = ftx + dfx / pori + tx;
        fty = fty + dfy / pori + ty;
        ftz = ftz + dfz / pori + tz;
        DW.ftx[i] = ftx;
        DW.fty[i] = fty;
        DW.ftz[i] = ftz;
        if (P.con) {
            DW.dtemp[i] = dq / (rhoi * cpi);
            D.Q_sd[i] = dq * mi / rhoi;
        }
        DW.Fdx_da[i] = dax; DW.Fdy_da[i] = day; DW.Fdz_da[i] = daz;
        DW.Fdx_b[i] = tx; DW.Fdy_b[i] = ty; DW.Fdz_b[i] = tz;
    }
    // predictor (DEM): u* = u + f dt
    DW.ux0[i] = uxi; DW.uy0[i] = uyi; DW.uz0[i] = uzi;
    if (pt == 9) {
        D.ux[i] = (Q)P.ball_vel; D.uy[i] = (Q)0; D.uz[i] = (Q)0;
        DW.ux0[i] = (Q)P.ball_vel; DW.uy0[i] = (Q)0; DW.uz0[i] = (Q)0;
    } else if (pt >= 0) {
        Q b = (Q)(D.btype[i] == 0);
        Q dt = (Q)P.dt;
        D.ux[i] = uxi + ftx * b * dt;
        D.uy[i] = uyi + fty * b * dt;
        D.uz[i] = uzi + ftz * b * dt;
    }
    if (P.con && pt > 0) DW.temp0[i] = D.temp[i];
}

// G = 32: a warp per sphere; G = 1: a thread per sphere (2-D beds with many
// spheres, ~20 SPH neighbours each); dem_thread_per_sphere in engine.cu.
template <typename R, int KT, int G>
__global__ void __launch_bounds__(128) k_dem_coupling(DevParams P, SphState<R> S, SphWork<R> W, DemState<double> D,
                                                      DemWork<double> DW, const int4* __restrict__ srows) {
    static_assert(G == 32 || G == 1, "a warp or a thread per sphere");
    grid_dep_wait();
    const int i = G == 32 ? (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5)
                          : (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const int lane = G == 32 ? (int)(threadIdx.x & 31) : 0;
    __shared__ int s_rows[4][20];   // 128 threads = 4 warps
    int* sm = s_rows[threadIdx.x >> 5];
    if (i >= P.nd) return;
    int it = D.itype[i], pt = D.ptype[i];
    if (it > 2) {
        if (lane == 0) DW.dcf[i] = -1;   // k_dem_finish skips it
        return;
    }
    DcSums<R> a{};
    const bool coupled = it == 1 && pt > 1000;
    if (coupled) {
        const SphRec<R> rec = W.rec;
        double xi = D.x[i], yi = D.y[i], zi = D.z[i], hi = D.h[i];
        R radi = (R)D.rad[i], voli = ((R)4 / (R)3) * (R)3.14159 * radi * radi * radi;
        R mi = D.m[i];
        R fa = DW.flt_s[i], ff = DW.flt_sd[i];
        R th = (R)hi;
        Knl<R, KT> K = knl_make<R, KT>(P, th);
        double Rr = P.kappa * hi;
        Band bd = make_band(P, Rr);
        PosRec<R> qp = make_pos<R>(P, xi, yi, zi, 0, 0, 0);
        int ic, jc, kc;
        cell_ijk(P, xi, yi, zi, ic, jc, kc);
        R pgc = voli / (mi * ff + (R)1.0e-15);
        auto pair = [&](int j) {
            PosRec<R> qj = ldr(rec.pos + j);
            int ptj = tag_ptype(qj.w);
            if (ptj > 1000) return;
            Disp<R> d;
            R r2;
            if (!test_pair(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j, Rr, 0.0, bd, d, r2)) return;
            R r, rinv;
            rdist(r2, r, rinv);
            dc_pair(W, K, ff, fa, pgc, j, ptj, r, a);
        };
        // the neighbours k_dem_prep listed (same positions, same predicate);
        // a sphere with more than the list holds walks its stencil
        const int cs = DW.ncs[i];
        if (KT == 3 && G == 32 && cs <= DEM_SPH_CAP) {
            // the listed pairs are inside: all of a pair's records load
            // together instead of one after another's test (56 -> 48 us on the
            // bench bed, where the pass waits on loads)
            const int* __restrict__ nbs = DW.nbs + (size_t)i * DEM_SPH_CAP;
            for (int k = lane; k < cs; k += G) {
                const int j = __ldg(nbs + k);
                const PosRec<R> qj = ldr(rec.pos + j);
                const V4<R> fj = ldr(rec.f1 + j), uj = ldr(rec.up + j);
                const R gx = ldr(W.pgfx + j), gy = ldr(W.pgfy + j), gz = ldr(W.pgfz + j);
                const Disp<R> d = disp_pt(P, qp, qj, xi, yi, zi, S.x, S.y, S.z, j);
                R r, rinv;
                rdist(d.dx * d.dx + d.dy * d.dy + d.dz * d.dz, r, rinv);
                dc_pair_at(K, ff, fa, pgc, fj, uj, gx, gy, gz, tag_ptype(qj.w), r, a);
            }
        } else if (cs <= DEM_SPH_CAP) {
            const int* __restrict__ nbs = DW.nbs + (size_t)i * DEM_SPH_CAP;
            for (int k = lane; k < cs; k += G) pair(__ldg(nbs + k));
        } else {
            const Cull cu = make_cull(xi, yi, zi, Rr);
            if constexpr (G == 32) for_rows_warp(P, ic, jc, kc, srows, cu, sm, lane, pair);
            else for_stencil_j(P, ic, jc, kc, srows, cu, pair);
        }
        if constexpr (G == 32) dc_warp_sum(a);
    }
    if (lane != 0) return;
    // the closure and the predictor run in k_dem_finish (thread per sphere),
    // so this pair pass keeps the registers of the FP32 sums only
    const int nd = P.nd;
    double* o = DW.dcs;
    o[0 * nd + i] = a.tx; o[1 * nd + i] = a.ty; o[2 * nd + i] = a.tz;
    o[3 * nd + i] = a.ufx; o[4 * nd + i] = a.ufy; o[5 * nd + i] = a.ufz;
    o[6 * nd + i] = a.uax; o[7 * nd + i] = a.uay; o[8 * nd + i] = a.uaz;
    o[9 * nd + i] = a.por; o[10 * nd + i] = a.ttf; o[11 * nd + i] = a.tta;
    o[12 * nd + i] = a.wtf; o[13 * nd + i] = a.wta;
    DW.dcf[i] = (coupled ? 1 : 0) | (a.has_f ? 2 : 0) | (a.has_a ? 4 : 0);
}

// the drag closure and the DEM predictor of every sphere the pair pass
// reached (dcf >= 0), on the sums it left in DW.dcs
template <typename R>
__global__ void __launch_bounds__(128) k_dem_finish(DevParams P, DemState<double> D, DemWork<double> DW) {
    grid_dep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nd = P.nd;
    if (i >= nd) return;
    const int f = DW.dcf[i];
    if (f < 0) return;
    const double* o = DW.dcs;
    DcSums<R> a;
    a.tx = (R)o[0 * nd + i]; a.ty = (R)o[1 * nd + i]; a.tz = (R)o[2 * nd + i];
    a.ufx = (R)o[3 * nd + i]; a.ufy = (R)o[4 * nd + i]; a.ufz = (R)o[5 * nd + i];
    a.uax = (R)o[6 * nd + i]; a.uay = (R)o[7 * nd + i]; a.uaz = (R)o[8 * nd + i];
    a.por = (R)o[9 * nd + i]; a.ttf = (R)o[10 * nd + i]; a.tta = (R)o[11 * nd + i];
    a.wtf = (R)o[12 * nd + i]; a.wta = (R)o[13 * nd + i];
    a.has_f = (f >> 1) & 1;
    a.has_a = (f >> 2) & 1;
    dem_coupling_finish(P, D, DW, i, (f & 1) != 0, a);
    // what the reaction force reads of a sphere
    DW.rc[i] = Dbl4{D.Fdx_df[i], D.Fdy_df[i], D.Fdz_df[i], D.Q_sd[i]};
    DW.rd[i] = make_double2(DW.flt_sd2[i], DW.flt_s[i]);
}

// ---------------------------------------------------------------------------
// KERNEL_SPH_coupling3D_sph (functions_SPH_DEM_COUPLING2.cuh:1815-2019) +
// KERNEL_clc_projection_sph (functions_TIME_ISPH2.cuh:104-204).
// ---------------------------------------------------------------------------
// L lanes per particle (small sets, small_set_lanes in engine.cu)
template <typename R, int KT, int L>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 6 : 1) k_sph_coupling(DevParams P, SphState<R> S, SphWork<R> W, DemState<double> D,
                                                      DemWork<double> DW, const int4* __restrict__ drows, int time_zero) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    int it = S.itype[i], pt = S.ptype[i];
    if (it > 2) return;
    R ftx = W.ftx[i], fty = W.fty[i], ftz = W.ftz[i];
    if (it == 1 && pt <= 1000) {
        double xi = S.x[i], yi = S.y[i], zi = S.z[i], hi = S.h[i];
        R rhoi = W.rho_new[i], tempi = S.temp[i];
        // heat_capacity(ptypei, tempi): the reference passes the arguments
        // swapped (functions_SPH_DEM_COUPLING2.cuh:1860)
        R cpi = (abs((int)(tempi + (R)P.t_ref)) > 1000) ? (R)P.cp_dem : (R)P.cp_sph;   // stored T - t_ref
        R th = (R)hi;
        Knl<R, KT> K = knl_make<R, KT>(P, th);
        double Rr = P.kappa * hi;
        R tx = 0, ty = 0, tz = 0, tt = 0;
        if (P.nd > 0 && (pt == 1 || pt == 3)) {
            float r2l = r2_lo(Rr), r2h = r2_hi(Rr);
            struct Rec {
                Dbl4 a, c;
                double2 f;
                double m;
            };
            auto load = [&](int j) { return Rec{ldr(DW.ra + j), ldr(DW.rc + j), ldr(DW.rd + j), ldr(&DW.rb[j].w)}; };
            struct T {
                R c, ax, ay, az, at;
            };
            auto terms = [&](int, const Rec& q, T& t) {
                PairT<R> g = pair_test<R>(xi, yi, zi, q.a.x, q.a.y, q.a.z, Rr, 0.0, r2l, r2h);
                if (!g.in) return false;
                R ffj = (R)q.f.x + (R)q.f.y;
                if (!(ffj > (R)0)) return false;
                R w = kw(K, g.r);
                if (P.dim == 2) w *= (R)0.75 / (R)q.a.w;   // per unit depth (depth 4 r / 3)
                t.c = w / (ffj + (R)1.0e-20);
                R mr = (R)q.m / rhoi;
                t.ax = -mr * (R)q.c.x;
                t.ay = -mr * (R)q.c.y;
                t.az = -mr * (R)q.c.z;
                t.at = -(R)q.c.w / (rhoi * cpi);
                return true;
            };
            auto add = [&](const T& t) {
                tx += t.ax * t.c;
                ty += t.ay * t.c;
                tz += t.az * t.c;
                tt += t.at * t.c;
            };
            auto one = [&](int j, const Rec& q) {
                T t;
                if (terms(j, q, t)) add(t);
            };
            const int cd = W.ncntd[i];
            if (cd <= P.nbd_cap) {
                if constexpr (L == 1) dem_walk<Rec>(W.nbrd, cd, n, i, load, one);
                else ordered_walk<L, Rec, T>(grp, cd, [&](int k) { return W.nbrd[(size_t)k * n + i]; }, load, terms, add);
            } else {
                int ic, jc, kc;
                cell_ijk(P, xi, yi, zi, ic, jc, kc);
                for_stencil_j(P, ic, jc, kc, drows, make_cull(xi, yi, zi, Rr), [&](int j) {
                    if (D.ptype[j] > 1000) one(j, load(j));
                });
            }
        }
        if (grp.lane) return;
        ftx += tx;
        fty += ty;
        ftz += tz;
        W.ftx[i] = ftx;
        W.fty[i] = fty;
        W.ftz[i] = ftz;
        W.ftot[i] = sqrt(ftx * ftx + fty * fty + ftz * ftz);
        if (P.con) W.dtemp[i] += tt;
    }
    if (grp.lane) return;
    // predictor (SPH), KERNEL_clc_projection_sph; eps u* also goes to the
    // {eps u*, p} record the PPE reads
    R uxi = S.ux[i], uyi = S.uy[i], uzi = S.uz[i];
    W.ux0[i] = uxi; W.uy0[i] = uyi; W.uz0[i] = uzi;
    R usx = uxi, usy = uyi, usz = uzi;
    if (pt == 9) {
        usx = (R)P.ball_vel; usy = (R)0; usz = (R)0;
        W.ux0[i] = (R)P.ball_vel; W.uy0[i] = (R)0; W.uz0[i] = (R)0;
    } else if (pt >= 0) {
        R b = (R)(S.btype[i] == 0);
        R dt = (R)P.sdt;
        usx = uxi + ftx * b * dt;
        usy = uyi + fty * b * dt;
        usz = uzi + ftz * b * dt;
    }
    S.ux[i] = usx; S.uy[i] = usy; S.uz[i] = usz;
    if (P.c2_passes) {
        const R pori = W.DEMpor[i];
        W.rec.pu[i] = mk4<R>(pori * usx, pori * usy, pori * usz, S.pres[i]);
    } else {
        W.rec.up[i] = mk4<R>(usx, usy, usz, S.pres[i]);
    }
    if (time_zero) W.rho_ref[i] = W.rho_new[i];
    if (P.con && pt > 0) W.temp0[i] = S.temp[i];
}

// a wall's pressure and density into the state and the records of the passes
// that follow (patch_p: its pressure too, before the pressure equation)
template <typename R>
__device__ __forceinline__ void wall_store(const DevParams& P, const SphWork<R>& W, R* pres, int i, R pw, R rw,
                                           int patch_p) {
    const SphRec<R> rec = W.rec;
    pres[i] = pw;
    W.rho_new[i] = rw;
    *comp<R>(rec.f1, i, 1) = rw;
    if (P.c2_passes) {
        pv_set_vol(rec.pb, i, pv_code<R>(*comp<R>(rec.f1, i, 0) / rw, ldr(rec.pos + i).w, false));
        if (patch_p) {
            rec.rp[i] = rec.f1[i].w * rw;
            *comp<R>(rec.pu, i, 3) = pw;
        }
    } else if (patch_p) {
        *comp<R>(rec.up, i, 3) = pw;
    }
}

// ---------------------------------------------------------------------------
// KERNEL_Neumann_boundary3D_sph (functions_BC.cuh:139-274): wall particles
// take the Shepard average over fluid within 2*kappa*h (W evaluated with
// 2h) inside the 27-cell stencil.  pres is the array the walls write into.
// One warp per wall particle (W.wall_idx lists the walls of this step).
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(128) k_neumann(DevParams P, SphState<R> S, SphWork<R> W, R* pres,
                                                 const int4* __restrict__ rows,
                                                 int patch_up) {
    grid_dep_wait();
    int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    __shared__ int s_rows[4][20];   // 128 threads = 4 warps
    int* sm = s_rows[threadIdx.x >> 5];
    if (w >= P.nwall || w >= W.counters[0]) return;
    const SphRec<R> rec = W.rec;
    int i = W.wall_idx[w];
    double xi = S.x[i], yi = S.y[i], zi = S.z[i], hi = S.h[i];
    R th2 = (R)2 * (R)hi;
    Knl<R> K = knl_make<R>(P, (R)hi);
    K.ih = rcp(th2);
    K.th = th2;
    double R2 = 2.0 * (P.kappa * hi);
    Band bd = make_band(P, R2);
    PosRec<R> qi = ldr(rec.pos + i);
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zi, ic, jc, kc);
    R tp = 0, flt = 0, tt = 0, tr = 0;
    const Cull cu = make_cull(xi, yi, zi, R2);
    for_rows_warp(P, ic, jc, kc, rows, cu, sm, lane, [&](int j) {
        PosRec<R> qj = ldr(rec.pos + j);
        int ptj = tag_ptype(qj.w);
        if (ptj < 1 || ptj >= 1000) return;
        Disp<R> d;
        R r2;
        if (!test_pair(P, qi, qj, xi, yi, zi, S.x, S.y, S.z, j, R2, 1e-20, bd, d, r2)) return;
        R r, rinv;
        rdist(r2, r, rinv);
        R wk = kw(K, r);
        V4<R> fj = ldr(rec.f1 + j);
        R mj = fj.x, rj = fj.y;
        R mr = mj * rcp(rj) * wk;
        tp += mr * pres[j];
        flt += mr;
        tt += mr * fj.z;
        tr += rj * rcp(fj.w) * wk * mj * rcp(rj);
    });
    tp = warp_sum(tp);
    flt = warp_sum(flt);
    tt = warp_sum(tt);
    tr = warp_sum(tr);
    if (lane != 0) return;
    R pw, rw;
    if (flt < (R)1e-6) {
        rw = W.rho_ref[i];
        pw = (R)0;
    } else {
        pw = tp / flt;
        S.temp[i] = tt / flt;
        rw = rec.f1[i].w * tr / flt;
    }
    wall_store<R>(P, W, pres, i, pw, rw, patch_up);
}

// Cell-tiled Neumann pass (FP32 build): one warp per cell that holds wall
// particles.  The fluid candidates of the cell's 9 stencil rows are staged
// (compacted in order) in shared memory with the factors the sums need
// ({x, y, z relative to a particle of the cell, slot} and {m/rho, p, T,
// m/eps}); each lane -- one wall particle of the cell -- runs over them in
// order with its own 2 kappa h radius, FP32 prefilter and the FP64
// reference predicate inside the band.  Same sums as k_neumann in candidate
// order per wall, so the FP32 results differ from it by rounding only.
constexpr int NT_WARPS = 4, NT_CH = 128;
// one cell of k_neumann_tiled (saw, sbw, srw: the warp's shared staging)
template <int KT>   // 5: Wendland C6; -1: the others
__device__ __forceinline__ void neumann_cell(int c, DevParams P, SphState<float> S, SphWork<float> W,
                                                                   float* pres, const int* __restrict__ gs,
                                                                   const int* __restrict__ ge,
                                                                   const int4* __restrict__ rows, int patch_up, float4* saw, float4* sbw, int* srw, int lane,
                                             int part = 0, int parts = 1) {
    const int a0 = __ldg(gs + c);
    if (a0 < 0) return;
    const int e0 = __ldg(ge + c);
    const SphRec<float> rec = W.rec;
    if (a0 + 32 * part >= e0) return;
    bool any_wall = false;
    for (int i = a0 + lane; i < e0; i += 32) any_wall |= S.ptype[i] <= 0;
    if (!__any_sync(0xffffffffu, any_wall)) return;
    const int ic = c % P.NI, jc = (c / P.NI) % P.NJ, kc = c / (P.NI * P.NJ);
    const int tot = stage_rows(P, ic, jc, kc, rows, srw, lane);
    const RelFrame Fr = rel_frame(P, ldr(rec.pos + a0));
    const unsigned lt = (1u << lane) - 1u;
    for (int p0 = a0 + 32 * part; p0 < e0; p0 += 32 * parts) {
        const int i = p0 + lane;
        const bool act = i < e0 && S.ptype[i] <= 0;
        if (!__any_sync(0xffffffffu, act)) continue;
        double xi = 0, yi = 0, zi = 0, R2 = 0;
        float lo2 = 0, hi2 = 0, fx = 0, fy = 0, fz = 0;
        float scale = 1.f;   // the sums times scale are the normalised sums
        Knl<float> K{};
        bool slow = false;
        if (act) {
            xi = S.x[i];
            yi = S.y[i];
            zi = S.z[i];
            const double hi = S.h[i];
            const float th2 = 2.f * (float)hi;
            K = knl_make<float>(P, (float)hi);
            K.ih = rcp(th2);
            K.th = th2;
            if (KT != 5 && K.kt == 3) {   // every chunk's sums leave out tA
                scale = K.tA;
                K.tA = 1.f;
            }
            R2 = 2.0 * (P.kappa * hi);
            const double b = rel_band(P, Fr, R2), r2 = R2 * R2;
            lo2 = (float)(r2 * (1.0 - b));
            hi2 = (float)(r2 * (1.0 + b));
            const int4 qi = ldr(rec.pos + i);
            slow = Fr.o_oor || rel_slow(Fr, qi);
            const float4 f = rel_coord(Fr, qi, 0);
            fx = f.x;
            fy = f.y;
            fz = f.z;
        }
        const bool lanes_slow = __any_sync(0xffffffffu, act && slow);
        float tp = 0.f, flt = 0.f, tt = 0.f, tr = 0.f;
        int t = 0;   // next raw candidate
        while (t < tot) {
            // stage fluid candidates in order until the chunk is full
            int ns = 0;
            bool any_oor = false;
            while (t < tot && ns <= NT_CH - 32) {
                const int tl = t + lane;
                bool keep = false;
                int4 qj = make_int4(0, 0, 0, 0);
                int j = 0;
                if (tl < tot) {
                    j = row_slot(srw, tl);
                    qj = ldr(rec.pos + j);
                    const int ptj = tag_ptype(qj.w);
                    keep = ptj >= 1 && ptj < 1000;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int pos = ns + __popc(m & lt);
                    const bool oor = rel_slow(Fr, qj);
                    any_oor |= oor;
                    const float4 fj = ldr(rec.f1 + j);
                    const float mr = fj.x * rcp(fj.y);
                    saw[pos] = rel_coord(Fr, qj, j | (oor ? (int)0x80000000 : 0));
                    sbw[pos] = make_float4(mr, pres[j], fj.z, fj.x * rcp(fj.w));
                }
                ns += __popc(m);
                t += 32;
            }
            const bool slow_chunk = lanes_slow || __any_sync(0xffffffffu, any_oor);
            __syncwarp();
            const int np = (ns + 3) & ~3;
            if constexpr (KT == 5) {   // padded to whole groups of four with candidates out of reach
                if (lane < np - ns) {
                    saw[ns + lane] = make_float4(1e18f, 1e18f, 1e18f, 0.f);
                    sbw[ns + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                __syncwarp();
            }
            if (KT != 5 && act && !slow_chunk && K.kt == 3) {
                // every candidate on the FP32 frame: the kernel is evaluated
                // for all of them and the pairs outside the radius add
                // nothing, so the lanes do not diverge (only a pair in the
                // rounding band takes the FP64 predicate).  Wendland C2 in
                // line without its normalisation tA, which cancels in the
                // ratios below (only the empty-support test scales by it).
                const float hq = 0.5f * K.ih;
#pragma unroll 4
                for (int u = 0; u < ns; u++) {
                    const float4 cj = saw[u];
                    const float dx = fx - cj.x, dy = fy - cj.y, dz = fz - cj.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    bool in = r2 < lo2;
                    if (!in && r2 <= hi2) {
                        const int j = __float_as_int(cj.w);
                        in = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                    }
                    const float q = r2 * rsqrtf(fmaxf(r2, 1e-30f)) * hq;
                    const float a = 1.f - q, a2 = a * a;
                    const float wk = a2 * a2 * (1.f + 4.f * q);
                    const float4 bj = sbw[u];
                    if (in && q < 1.f) {
                        const float mr = bj.x * wk;
                        tp += mr * bj.y;
                        flt += mr;
                        tt += mr * bj.z;
                        tr += bj.w * wk;
                    }
                }
            } else if (KT == 5 && act && !slow_chunk) {
                // Wendland C6, four candidates at a time without branches
                // between them (the band's FP64 predicate: one branch per
                // four): the wall pass of the gas-spouted beds waits on its
                // own arithmetic, 194 -> 174 us.  C2's shorter loop is faster
                // one by one (46 against 50).
                const Knl<float, 5> K5{K.kt, K.tA, K.ih, K.th};
                for (int u0 = 0; u0 < np; u0 += 4) {
                    float r2[4], w[4];
                    bool in[4], band = false;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float4 cj = saw[u0 + u];
                        const float dx = fx - cj.x, dy = fy - cj.y, dz = fz - cj.z;
                        r2[u] = dx * dx + dy * dy + dz * dz;
                        in[u] = r2[u] < lo2;
                        band |= !in[u] && r2[u] <= hi2;
                    }
                    if (band) {
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (!in[u] && r2[u] <= hi2) {
                                const int j = __float_as_int(saw[u0 + u].w);
                                in[u] = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                            }
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        float r, rinv;
                        rdist(r2[u], r, rinv);
                        w[u] = kw(K5, r);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const float4 bj = sbw[u0 + u];
                        const float wk = w[u];
                        if (in[u]) {
                            const float mr = bj.x * wk;
                            tp += mr * bj.y;
                            flt += mr;
                            tt += mr * bj.z;
                            tr += bj.w * wk;
                        }
                    }
                }
            } else if (act && !slow_chunk) {
                // as above, any kernel
#pragma unroll 2
                for (int u = 0; u < ns; u++) {
                    const float4 cj = saw[u];
                    const float dx = fx - cj.x, dy = fy - cj.y, dz = fz - cj.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    bool in = r2 < lo2;
                    if (!in && r2 <= hi2) {
                        const int j = __float_as_int(cj.w);
                        in = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                    }
                    float r, rinv;
                    rdist(r2, r, rinv);
                    const float wk = kw(K, r);
                    const float4 bj = sbw[u];
                    if (in) {
                        const float mr = bj.x * wk;
                        tp += mr * bj.y;
                        flt += mr;
                        tt += mr * bj.z;
                        tr += bj.w * wk;
                    }
                }
            } else if (act) {
                for (int u = 0; u < ns; u++) {
                    const float4 cj = saw[u];
                    const float dx = fx - cj.x, dy = fy - cj.y, dz = fz - cj.z;
                    const float r2 = dx * dx + dy * dy + dz * dz;
                    bool in;
                    if (!slow_chunk) {
                        if (r2 > hi2) continue;
                        in = r2 < lo2;
                        if (!in) {
                            const int j = __float_as_int(cj.w);
                            in = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                        }
                    } else {
                        const int jb = __float_as_int(cj.w), j = jb & 0x7fffffff;
                        if (!slow && jb >= 0) {
                            if (r2 > hi2) continue;
                            in = r2 < lo2 ||
                                 __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                        } else {
                            in = __dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2;
                        }
                    }
                    if (!in) continue;
                    float r, rinv;
                    if (!slow_chunk || (!slow && __float_as_int(cj.w) >= 0)) {
                        rdist(r2, r, rinv);
                    } else {
                        const int j = __float_as_int(cj.w) & 0x7fffffff;
                        const float ex = (float)(xi - S.x[j]), ey = (float)(yi - S.y[j]), ez = (float)(zi - S.z[j]);
                        rdist(ex * ex + ey * ey + ez * ez, r, rinv);
                    }
                    const float wk = kw(K, r);
                    const float4 bj = sbw[u];
                    const float mr = bj.x * wk;
                    tp += mr * bj.y;
                    flt += mr;
                    tt += mr * bj.z;
                    tr += bj.w * wk;
                }
            }
            __syncwarp();
        }
        if (!act) continue;
        float pw, rw;
        if (flt * scale < 1e-6f) {
            rw = W.rho_ref[i];
            pw = 0.f;
        } else {
            pw = tp / flt;
            S.temp[i] = tt / flt;
            rw = rec.f1[i].w * tr / flt;
        }
        wall_store<float>(P, W, pres, i, pw, rw, patch_up);
    }
}

template <bool OCC, int KT>
__global__ void __launch_bounds__(NT_WARPS * 32, 8) k_neumann_tiled(DevParams P, SphState<float> S, SphWork<float> W,
                                                                   float* pres, const int* __restrict__ gs,
                                                                   const int* __restrict__ ge,
                                                                   const int4* __restrict__ rows, int patch_up, int parts,
                                                                   const int* __restrict__ occ, const int* __restrict__ occ_n) {
    grid_dep_wait();
    __shared__ float4 sa[NT_WARPS][NT_CH + 32];
    __shared__ float4 sb[NT_WARPS][NT_CH + 32];
    __shared__ int srow[NT_WARPS][20];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (OCC) {   // a sparse grid: the occupied cells, grid-stride
        const int no = *occ_n;
        for (int q = blockIdx.x * NT_WARPS + w; q < no; q += gridDim.x * NT_WARPS) {
            neumann_cell<KT>(occ[q], P, S, W, pres, gs, ge, rows, patch_up, sa[w], sb[w], srow[w], lane);
            __syncwarp();
        }
    } else {
        // parts warps per cell, every parts-th group of 32 of its particles each
        const int q = blockIdx.x * NT_WARPS + w, c = q / parts;
        if (c < P.NI * P.NJ * P.NK)
            neumann_cell<KT>(c, P, S, W, pres, gs, ge, rows, patch_up, sa[w], sb[w], srow[w], lane, q % parts, parts);
    }
}

// The tiled pass in double (Wendland C2): a warp per cell that holds walls,
// the fluid candidates staged with their factors, a lane per wall.  The squared
// distance decides outside a band of 4e-15 around the radius (its rounding is
// below 1e-15), the reference's square root inside it.  A warp per wall
// (k_neumann) evaluated a square root per candidate and reduced four sums per
// wall: 331 -> 143 us on the bench bed.
constexpr int N64_CH = 96;
__device__ __forceinline__ void neumann_cell64(int c, const DevParams& P, SphState<double>& S, SphWork<double>& W,
                                               double* pres, const int* __restrict__ gs, const int* __restrict__ ge,
                                               const int4* __restrict__ rows, int patch_p, double2 (*sa)[4], int* sj,
                                               int* srw, int lane) {
    const int a0 = __ldg(gs + c);
    if (a0 < 0) return;
    const int e0 = __ldg(ge + c);
    const SphRec<double> rec = W.rec;
    bool any_wall = false;
    for (int i = a0 + lane; i < e0; i += 32) any_wall |= S.ptype[i] <= 0;
    if (!__any_sync(0xffffffffu, any_wall)) return;
    const int ic = c % P.NI, jc = (c / P.NI) % P.NJ, kc = c / (P.NI * P.NJ);
    const int tot = stage_rows(P, ic, jc, kc, rows, srw, lane);
    const unsigned lt = (1u << lane) - 1u;
    for (int p0 = a0; p0 < e0; p0 += 32) {
        const int i = p0 + lane;
        const bool act = i < e0 && S.ptype[i] <= 0;
        if (!__any_sync(0xffffffffu, act)) continue;
        double xi = 0, yi = 0, zi = 0, R2 = 0, hq = 0, scale = 1;
        if (act) {
            xi = S.x[i];
            yi = S.y[i];
            zi = S.z[i];
            const double hi = S.h[i];
            R2 = 2.0 * (P.kappa * hi);
            hq = 0.25 / hi;   // 1 / (2 (2h))
            scale = knl_tmpA<double>(3, P.dim, hi);
        }
        const double lo = R2 * R2 * (1.0 - 4e-15), hi2 = R2 * R2 * (1.0 + 4e-15);
        double tp = 0, flt = 0, tt = 0, tr = 0;
        int t = 0;
        while (t < tot) {
            int ns = 0;
            while (t < tot && ns <= N64_CH - 32) {
                const int tl = t + lane;
                bool keep = false;
                int j = 0;
                if (tl < tot) {
                    j = row_slot(srw, tl);
                    const int ptj = S.ptype[j];
                    keep = ptj >= 1 && ptj < 1000;
                }
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) {
                    const int pos = ns + __popc(m & lt);
                    const Dbl4 fj = ldr(rec.f1 + j);
                    sa[pos][0] = make_double2(S.x[j], S.y[j]);
                    sa[pos][1] = make_double2(S.z[j], fj.x / fj.y);
                    sa[pos][2] = make_double2(pres[j], fj.z);
                    sa[pos][3] = make_double2(fj.x / fj.w, 0.0);
                    sj[pos] = j;
                }
                ns += __popc(m);
                t += 32;
            }
            __syncwarp();
            if (act) {
#pragma unroll 2
                for (int u = 0; u < ns; u++) {
                    const double2 xy = sa[u][0], zm = sa[u][1];
                    const double dx = xi - xy.x, dy = yi - xy.y, dz = zi - zm.x;
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    if (r2 > hi2) continue;
                    if (!(r2 < lo)) {
                        const int j = sj[u];
                        if (!(__dadd_rn(pair_dist(xi, yi, zi, S.x[j], S.y[j], S.z[j]), 1e-20) < R2)) continue;
                    }
                    const double q = r2 * rsq_floor(r2) * hq;
                    if (!(q < 1.0)) continue;
                    const double a = 1.0 - q, a2 = a * a, wk = a2 * a2 * (1.0 + 4.0 * q);
                    const double2 pt = sa[u][2], me = sa[u][3];
                    const double mr = zm.y * wk;
                    tp += mr * pt.x;
                    flt += mr;
                    tt += mr * pt.y;
                    tr += me.x * wk;
                }
            }
            __syncwarp();
        }
        if (!act) continue;
        double pw, rw;
        if (flt * scale < 1e-6) {
            rw = W.rho_ref[i];
            pw = 0.0;
        } else {
            pw = tp / flt;
            S.temp[i] = tt / flt;
            rw = rec.f1[i].w * tr / flt;
        }
        wall_store<double>(P, W, pres, i, pw, rw, patch_p);
    }
}

template <bool OCC>
__global__ void __launch_bounds__(64) k_neumann_tiled64(DevParams P, SphState<double> S, SphWork<double> W,
                                                        double* pres, const int* __restrict__ gs,
                                                        const int* __restrict__ ge, const int4* __restrict__ rows,
                                                        int patch_p, const int* __restrict__ occ,
                                                        const int* __restrict__ occ_n) {
    grid_dep_wait();
    __shared__ double2 sa[2][N64_CH][4];
    __shared__ int sj[2][N64_CH];
    __shared__ int srow[2][20];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (OCC) {   // a sparse grid: the occupied cells, grid-stride
        const int no = *occ_n;
        for (int q = blockIdx.x * 2 + w; q < no; q += gridDim.x * 2) {
            neumann_cell64(occ[q], P, S, W, pres, gs, ge, rows, patch_p, sa[w], sj[w], srow[w], lane);
            __syncwarp();
        }
    } else {
        const int c = blockIdx.x * 2 + w;
        if (c < P.NI * P.NJ * P.NK) neumann_cell64(c, P, S, W, pres, gs, ge, rows, patch_p, sa[w], sj[w], srow[w], lane);
    }
}

// ---------------------------------------------------------------------------
// KERNEL_PPE3D_sph + KERNEL_PPE3D_calc_sph (functions_PPE2.cuh:542-698,
// 868-878): one Jacobi sweep; p_new = (b + sum A_ij p_j) / sum A_ij for
// fluid, every other particle keeps its pressure.
// ---------------------------------------------------------------------------
// With G = dW/dr / r, d = x_i - x_j, V = m_j / rho_j and C the symmetric
// gradient correction: A_ij = -(eps_i rho_i + eps_j rho_j) / rho_i V G (d . C d) / r^2
// and the divergence sum takes V G (eps_i u_i - eps_j u_j) . C d; eps u*, p and
// eps rho come from their records, G's factor and 1 / rho_i leave the sums.
template <typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 5 : 1) k_ppe(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    bool solve = it <= 2 && !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (!solve) {
        W.p_new[i] = S.pres[i];
        return;
    }
    const V4<R> pui = rec.pu[i];
    R th = (R)S.h[i];
    const C2Sum<R> K = c2_sum<R>(P, th);
    const PvRec<R> qi = ldr(rec.pb + i);
    const bool slow_i = pv_vol(qi) != pv_vol(qi);
    const R prhoi = rec.rp[i];
    const Cm6<R> C = cm6_load(W.Cm, n, i, P.kgc == 1);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R b = 0, A = 0, AP = 0;
    const int* __restrict__ nb = W.nbr;
    nb_sum<NbP4S<R>, PairV<R>>(
        cnt, nb, n, i,
        [&](int j) {
            NbP4S<R> t;
            t.q = ldr(rec.pb + j);
            t.b = ldr(rec.pu + j);
            t.s = ldr(rec.rp + j);
            return t;
        },
        [&](const NbP4S<R>& t, PairV<R>& g) { return pv_prep<R, false>(P, qi, slow_i, t.q, g); },
        [&](int j, NbP4S<R>& t, PairV<R>& g) {
            int tag;
            if (!pv_fix(S, rec.pos, W.m_new, W.rho_new, slow_i, t.q, i, j, g, tag)) return;
            if (tag_ptype(tag) >= 1000) {   // no neighbour of this sum
                g.v = 0;
                t.b = pui;
                t.s = prhoi;
            }
        },
        [&](int, const NbP4S<R>& t, const PairV<R>& g) {
            const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
            const R rinv = rsq_floor(r2), r = r2 * rinv;
            const R v = g.v;
            const R vg = v * c2_g(K, r);
            const Disp<R> y = cm6_mul(C, g.dx, g.dy, g.dz);
            b += vg * ((pui.x - t.b.x) * y.dx + (pui.y - t.b.y) * y.dy + (pui.z - t.b.z) * y.dz);
            const R quad = g.dx * y.dx + g.dy * y.dy + g.dz * y.dz;
            const R a = vg * (prhoi + t.s) * (quad * rinv * rinv);
            A += a;
            AP += a * t.b.w;
        });
    const R sc = -K.gn * rcp(rec.f1[i].y);
    const R bs = (R)P.rho_gas * (K.gn * b + (R)2 * S.dDEMpor[i] - W.dDEMpor_prev[i]) / (R)P.sdt;
    W.p_new[i] = (bs + sc * AP) / (sc * A);
}

// ---------------------------------------------------------------------------
// pass C: KERNEL_pressureforce3D_sph (functions_PPE2.cuh:2154-2335) and
// KERNEL_time_update_projection_sph (functions_TIME_ISPH2.cuh:467-620).
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 7 : 1) k_passC(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    W.fpx[i] = 0; W.fpy[i] = 0; W.fpz[i] = 0;
    if (it > 2) {
        rec.ut[i] = mk4<R>(S.ux[i], S.uy[i], S.uz[i], S.temp[i]);
        return;
    }
    R fx = 0, fy = 0, fz = 0;
    bool pf = !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (pf && P.fp) {
        // sum of V (p_i + p_j) G d; the gradient correction and the factors after it
        R th = (R)S.h[i];
        const C2Sum<R> K = c2_sum<R>(P, th);
        const PvRec<R> qi = ldr(rec.pb + i);
        const bool slow_i = pv_vol(qi) != pv_vol(qi);
        const R pi = W.p_new[i];
        int cnt = min(W.ncnt[i], P.nb_cap);
        const int* __restrict__ nb = W.nbr;
        const R* __restrict__ pn = W.p_new;
        nb_sum<NbPS<R>, PairV<R>>(
            cnt, nb, n, i,
            [&](int j) {
                NbPS<R> t;
                t.q = ldr(rec.pb + j);
                t.s = ldr(pn + j);
                return t;
            },
            [&](const NbPS<R>& t, PairV<R>& g) { return pv_prep<R, false>(P, qi, slow_i, t.q, g); },
            [&](int j, NbPS<R>& t, PairV<R>& g) {
                int tag;
                if (!pv_fix(S, rec.pos, W.m_new, W.rho_new, slow_i, t.q, i, j, g, tag)) return;
                if (tag_ptype(tag) >= 1000) {   // no neighbour of this sum
                    g.v = 0;
                    t.s = pi;
                }
            },
            [&](int, const NbPS<R>& t, const PairV<R>& g) {
                const R v = g.v;
                const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
                const R rinv = rsq_floor(r2), r = r2 * rinv;
                const R s = v * c2_g(K, r) * (pi + t.s);
                fx += s * g.dx;
                fy += s * g.dy;
                fz += s * g.dz;
            });
        const Cm6<R> C = cm6_load(W.Cm, n, i, P.kgc == 1);
        const R cpi = -rec.f1[i].w * rcp(W.rho_new[i]) * K.gn;
        const Disp<R> a = cm6_mul(C, fx, fy, fz);
        fx = cpi * a.dx;
        fy = cpi * a.dy;
        fz = cpi * a.dz;
        W.fpx[i] = fx; W.fpy[i] = fy; W.fpz[i] = fz;
    }
    if (pt == 9) {
        rec.ut[i] = mk4<R>(S.ux[i], S.uy[i], S.uz[i], S.temp[i]);
        return;
    }
    R ux0, uy0, uz0, ax, ay, az;
    if (pt > 0) {
        ux0 = S.ux[i]; uy0 = S.uy[i]; uz0 = S.uz[i];
        R b = (R)(bt == 0);
        ax = fx * b; ay = fy * b; az = fz * b;
    } else {
        ux0 = W.ux0[i]; uy0 = W.uy0[i]; uz0 = W.uz0[i];
        ax = ay = az = (R)0;
    }
    R dt = (R)P.sdt;
    R uxc = ux0 + ax * dt, uyc = uy0 + ay * dt, uzc = uz0 + az * dt;
    R lim = (R)P.u_limit;
    if ((uxc * uxc + uyc * uyc + uzc * uzc) >= lim * lim) {
        uxc = ux0; uyc = uy0; uzc = uz0;
    }
    if (!P.xsph && P.sph_lagrangian && pt > 0) {
        S.x[i] += ((double)W.ux0[i] + (double)uxc) / 2.0 * P.sdt;
        S.y[i] += ((double)W.uy0[i] + (double)uyc) / 2.0 * P.sdt;
        S.z[i] += ((double)W.uz0[i] + (double)uzc) / 2.0 * P.sdt;
    }
    S.ux[i] = uxc; S.uy[i] = uyc; S.uz[i] = uzc;
    R tn = S.temp[i];
    if (P.con && pt > 0) {
        tn = W.temp0[i] + W.dtemp[i] * dt * (R)(pt != -1);
        S.temp[i] = tn;
    }
    rec.ut[i] = mk4<R>(uxc, uyc, uzc, tn);
}

// ---------------------------------------------------------------------------
// DEM corrector (KERNEL_time_update_projection_dem, functions_TIME_ISPH2.cuh:
// 622-776) followed by KERNEL_treat_DEM_{cylinder_z,box_z,truncated_cone_z}_dem
// (functions_DEM_BC.cuh:491-718, 1770-2027, 4485-4722) on the same particle.
// ---------------------------------------------------------------------------
template <typename R>
__device__ void dem_wall_response(const DevParams& P, DemState<R>& D, DemWork<R>& DW, int i, R nx, R ny, R nz) {
    R kdt = (R)P.dt;
    R ux = D.ux[i], uy = D.uy[i], uz = D.uz[i], wx = D.wx[i], wy = D.wy[i], wz = D.wz[i];
    R m = D.m[i], ri = D.ri[i], rad = (R)D.rad[i];
    R ftx = DW.ftx[i], fty = DW.fty[i], ftz = DW.ftz[i];
    R ucx = ux - rad * (wy * nz - wz * ny), ucy = uy - rad * (wz * nx - wx * nz), ucz = uz - rad * (wx * ny - wy * nx);
    R cwx = -rad * (wy * nz - wz * ny), cwy = -rad * (wz * nx - wx * nz), cwz = -rad * (wx * ny - wy * nx);
    R unm = ux * nx + uy * ny + uz * nz;
    R ucn = ucx * nx + ucy * ny + ucz * nz, cwn = cwx * nx + cwy * ny + cwz * nz;
    R usx = ucx - ucn * nx, usy = ucy - ucn * ny, usz = ucz - ucn * nz;
    R uwx = cwx - cwn * nx, uwy = cwy - cwn * ny, uwz = cwz - cwn * nz;
    const R tiny = (R)1e-10;
    if (fabs(usx) < tiny) usx = 0;
    if (fabs(usy) < tiny) usy = 0;
    if (fabs(usz) < tiny) usz = 0;
    if (fabs(uwx) < tiny) uwx = 0;
    if (fabs(uwy) < tiny) uwy = 0;
    if (fabs(uwz) < tiny) uwz = 0;
    R usm = sqrt(usx * usx + usy * usy + usz * usz), uwm = sqrt(uwx * uwx + uwy * uwy + uwz * uwz);
    R sx = usx / (usm + (R)1e-20), sy = usy / (usm + (R)1e-20), sz = usz / (usm + (R)1e-20);
    R swx = uwx / (uwm + (R)1e-20), swy = uwy / (uwm + (R)1e-20), swz = uwz / (uwm + (R)1e-20);
    if (fabs(unm) < (R)50 * kdt) {
        R fn = ftx * nx + fty * ny + ftz * nz;
        R a = (R)P.mu_s * m * fn, b = (R)P.mu_rs * m * fn;
        R ffx = a * sx, ffy = a * sy, ffz = a * sz, frx = b * swx, fry = b * swy, frz = b * swz;
        if (fn > (R)0) { ffx = ffy = ffz = frx = fry = frz = 0; }
        DW.ftx[i] = ftx + ffx / m;
        DW.fty[i] = fty + ffy / m;
        DW.ftz[i] = ftz + ffz / m;
        R q = rad / ri;
        DW.tqx[i] += -q * (ny * (ffz + frz) - nz * (ffy + fry));
        DW.tqy[i] += -q * (nz * (ffx + frx) - nx * (ffz + frz));
        DW.tqz[i] += -q * (nx * (ffy + fry) - ny * (ffx + frx));
        R uxc = ux + (ffx / m) * kdt, uyc = uy + (ffy / m) * kdt, uzc = uz + (ffz / m) * kdt;
        R ucn2 = uxc * nx + uyc * ny + uzc * nz;
        D.ux[i] = uxc - ucn2 * nx;
        D.uy[i] = uyc - ucn2 * ny;
        D.uz[i] = uzc - ucn2 * nz;
        D.wx[i] = wx - q * (ny * (ffz + frz) - nz * (ffy + fry)) * kdt;
        D.wy[i] = wy - q * (nz * (ffx + frx) - nx * (ffz + frz)) * kdt;
        D.wz[i] = wz - q * (nx * (ffy + fry) - ny * (ffx + frx)) * kdt;
    } else {
        R cn = -m * ((R)1 + (R)P.rest_n) * ucn;
        R cs = -(R)1 / (((R)1 / m) + (rad * rad / ri)) * ((R)1 + (R)P.rest_s) * usm;
        R Jx = cn * nx + cs * sx, Jy = cn * ny + cs * sy, Jz = cn * nz + cs * sz;
        R q = rad / ri;
        D.ux[i] = ux + ((R)1 / m) * Jx;
        D.uy[i] = uy + ((R)1 / m) * Jy;
        D.uz[i] = uz + ((R)1 / m) * Jz;
        D.wx[i] = wx - q * (ny * Jz - nz * Jy);
        D.wy[i] = wy - q * (nz * Jx - nx * Jz);
        D.wz[i] = wz - q * (nx * Jy - ny * Jx);
    }
}

template <typename R>
__global__ void __launch_bounds__(128) k_dem_update(DevParams P, DemState<R> D, DemWork<R> DW) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.nd) return;
    int it = D.itype[i], pt = D.ptype[i];
    if (it > 2) return;
    if (pt != 9) {
        R ux0, uy0, uz0;
        if (pt > 0) { ux0 = D.ux[i]; uy0 = D.uy[i]; uz0 = D.uz[i]; }
        else { ux0 = DW.ux0[i]; uy0 = DW.uy0[i]; uz0 = DW.uz0[i]; }
        // fp and fb are zero for DEM particles: the corrector keeps u*
        R lim = (R)P.u_limit;
        R uxc = ux0, uyc = uy0, uzc = uz0;
        if ((uxc * uxc + uyc * uyc + uzc * uzc) >= lim * lim) { uxc = ux0; uyc = uy0; uzc = uz0; }
        if (pt > 0) {
            D.x[i] += ((double)DW.ux0[i] + (double)uxc) / 2.0 * P.dt;
            D.y[i] += ((double)DW.uy0[i] + (double)uyc) / 2.0 * P.dt;
            D.z[i] += ((double)DW.uz0[i] + (double)uzc) / 2.0 * P.dt;
        }
        D.ux[i] = uxc; D.uy[i] = uyc; D.uz[i] = uzc;
    }
    if (P.con && pt > 0) D.temp[i] = DW.temp0[i] + DW.dtemp[i] * (R)P.dt * (R)(pt != -1);
    if (it != 1 || pt <= 1000) return;
    // cylinder_z
    if (P.wall_mask & 1) {
        double xc = P.cyl_cx, yc = P.cyl_cy, Rc = P.cyl_r;
        double x = D.x[i], y = D.y[i], z = D.z[i], rad = D.rad[i];
        double F = (x - xc) * (x - xc) + (y - yc) * (y - yc) - (Rc - rad) * (Rc - rad);
        if (F > 0) {
            double rr = sqrt((x - xc) * (x - xc) + (y - yc) * (y - yc));
            double cpx = xc + (Rc - rad) * (x - xc) / rr, cpy = yc + (Rc - rad) * (y - yc) / rr;
            D.x[i] = cpx; D.y[i] = cpy; D.z[i] = z;
            double nx = -(cpx - xc) / (Rc - rad), ny = -(cpy - yc) / (Rc - rad);
            if (!(sqrt(nx * nx + ny * ny) < 0.5)) dem_wall_response<R>(P, D, DW, i, (R)nx, (R)ny, (R)0);
        }
    }
    // box_z
    if (P.wall_mask & 2) {
        double xc = P.box_c[0], yc = P.box_c[1], zc = P.box_c[2];
        double hx = 0.5 * P.box_L[0], hy = 0.5 * P.box_L[1], hz = 0.5 * P.box_L[2];
        double x = D.x[i], y = D.y[i], z = D.z[i], rad = D.rad[i];
        double F = fmax(fmax(fabs(x - xc) - (hx - rad), fabs(y - yc) - (hy - rad)), fabs(z - zc) - (hz - rad));
        if (F > 0) {
            double cpx = xc + fmin(hx - rad, fmax(-(hx - rad), x - xc));
            double cpy = yc + fmin(hy - rad, fmax(-(hy - rad), y - yc));
            double cpz = zc + fmin(hz - rad, fmax(-(hz - rad), z - zc));
            D.x[i] = cpx; D.y[i] = cpy; D.z[i] = cpz;
            double sgx = (cpx - x) / (fabs(cpx - x) + 1e-20);
            double sgy = (cpy - y) / (fabs(cpy - y) + 1e-20);
            double sgz = (cpz - z) / (fabs(cpz - z) + 1e-20);
            if (fabs(cpy - y) < 1e-12) sgy = 0.0;
            if (fabs(cpy - x) < 1e-12) sgx = 0.0;  // the reference tests cpy-x here (functions_DEM_BC.cuh:1846)
            if (fabs(cpz - z) < 1e-12) sgz = 0.0;
            double nn = sqrt(sgx * sgx + sgy * sgy + sgz * sgz) + 1e-20;
            double nx = sgx / nn, ny = sgy / nn, nz = sgz / nn;
            if (!(sqrt(nx * nx + ny * ny + nz * nz) < 0.5)) dem_wall_response<R>(P, D, DW, i, (R)nx, (R)ny, (R)nz);
        }
    }
    // truncated_cone_z
    if (P.wall_mask & 4) {
        double xc = P.cone_c[0], yc = P.cone_c[1], r1 = P.cone_r1, r2 = P.cone_r2, hc = P.cone_h;
        double x = D.x[i], y = D.y[i], z = D.z[i], rad = D.rad[i];
        if (!(z <= -hc + rad)) {
            double L = sqrt((r1 - r2) * (r1 - r2) + hc * hc);
            double st = hc / L, ct = fabs(r1 - r2) / L, tt = st / ct;
            double rr = r2 + (hc + z) / tt - rad / st;
            double rxy = sqrt((x - xc) * (x - xc) + (y - yc) * (y - yc));
            double F = (x - xc) * (x - xc) + (y - yc) * (y - yc) - rr * rr;
            if (F > 0) {
                double cpz = tt * (rxy + rad / st - r2) - hc;
                D.z[i] = cpz;
                double nx = -st * (x - xc) / rxy, ny = -st * (y - yc) / rxy, nz = ct;
                dem_wall_response<R>(P, D, DW, i, (R)nx, (R)ny, (R)nz);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// KERNEL_open_boundary_extrapolation3D_1{,_calc}_sph (functions_BC.cuh:
// 787-984, 1204-1218): buffer particles take Shepard averages of the fluid
// around their mirror point.  Only non-buffer fluid is read, so the update
// is done in place.  One warp per buffer particle (W.buf_idx).
// ---------------------------------------------------------------------------
constexpr int OB_Q = 8;   // queued hits per lane
template <typename R, int KT>
__global__ void __launch_bounds__(128) k_open_bc(DevParams P, SphState<R> S, SphWork<R> W, const int4* __restrict__ rows) {
    grid_dep_wait();
    int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    __shared__ int s_rows[4][20];   // 128 threads = 4 warps
    int* sm = s_rows[threadIdx.x >> 5];
    if (w >= P.nbuf || w >= W.counters[1]) return;
    int i = W.buf_idx[w];
    int bt = S.btype[i];
    double xi = S.x[i], yi = S.y[i], zi = S.z[i], hi = S.h[i];
    const BedObc ob = bed_obc(P, yi);
    double zg = zi;
    if (bt == 1) zg = 2 * ob.L2 - zi;
    else if (bt == 2) zg = 2 * ob.L3 - zi;
    R th = (R)hi;
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    double Rr = P.kappa * hi;
    const Band bd = make_band(P, Rr);
    const PosRec<R> qp = make_pos<R>(P, xi, yi, zg, 0, 0, 0);   // the mirror point
    int ic, jc, kc;
    cell_ijk(P, xi, yi, zg, ic, jc, kc);
    R hd = (R)P.h_over_dx;
    R trho = 0, tp = 0, tux = 0, tuy = 0, tuz = 0, tt = 0, flt = 0;
    const Cull cu = make_cull(xi, yi, zg, Rr);
    // the candidate's type and the prefilter from its packed record (one
    // load); the FP64 predicate only inside the band.  A lane queues its hits
    // and the warp sums them when a queue is full and at the end, all lanes
    // together: summed where they were found, a few lanes at a time ran the
    // seven sums in nearly every round.  Each lane's sums keep their order.
    __shared__ int s_q[4][OB_Q][32];
    int(*qu)[32] = s_q[threadIdx.x >> 5];
    int nq = 0;
    auto flush = [&]() {
        const int m = __reduce_max_sync(0xffffffffu, nq);
        for (int k = 0; k < m; k++) {
            if (k >= nq) continue;
            const int j = qu[k][lane];
            const PosRec<R> qj = ldr(W.rec.pos + j);
            const Disp<R> d = disp_pt(P, qp, qj, xi, yi, zg, S.x, S.y, S.z, j);
            const R r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
            R r, rinv;
            rdist(r2, r, rinv);
            R wk = kw(K, r);
            R hj = (R)S.h[j];
            R volj = sph_volume(P, hj, hd);
            R vw = volj * wk;
            trho += W.rho_new[j] / W.DEMpor[j] * wk * volj;
            tp += vw * W.p_new[j];
            tuz += vw * S.uz[j];
            tux += vw * S.ux[j];
            tuy += vw * S.uy[j];
            tt += vw * S.temp[j];
            flt += vw;
        }
        nq = 0;
    };
    auto pos = [&](int j) { return ldr(W.rec.pos + j); };
    for_rows_warp_pre<PosRec<R>>(P, ic, jc, kc, rows, cu, sm, lane, pos, [&](int j, const PosRec<R>& qj) {
        bool in = false;
        if (j >= 0) {
            Disp<R> d;
            R r2;
            in = tag_ptype(qj.w) == 1 && tag_btype(qj.w) == 0 &&
                 test_pair(P, qp, qj, xi, yi, zg, S.x, S.y, S.z, j, Rr, 1e-20, bd, d, r2);
        }
        if (in) qu[nq++][lane] = j;
        if (__any_sync(0xffffffffu, nq == OB_Q)) flush();
    });
    flush();
    trho = warp_sum(trho); tp = warp_sum(tp); tux = warp_sum(tux); tuy = warp_sum(tuy);
    tuz = warp_sum(tuz); tt = warp_sum(tt); flt = warp_sum(flt);
    if (lane != 0 || P.open_bc != 1) return;
    R pori = W.DEMpor[i];
    R vol0 = sph_volume(P, th, hd);
    R rho_old = W.rho_new[i];
    R pn, rn, ux, uy, uz, tn;
    if (bt == 1) {
        pn = tp / flt;
        rn = pori * (R)P.rho_gas;
        uz = (R)ob.inlet_uz * (R)2 - tuz / flt;
        ux = (R)0 - tux / flt;
        uy = (R)0 - tuy / flt;
        tn = (R)(ob.inlet_temp - P.t_ref);   // stored T - t_ref
    } else {
        pn = (R)0;
        rn = pori * (trho / flt);
        uz = tuz / flt;
        ux = tux / flt;
        uy = tuy / flt;
        tn = tt / flt;
    }
    R mn = rho_old * vol0;
    W.p_new[i] = pn;
    W.rho_new[i] = rn;
    W.m_new[i] = mn;
    S.ux[i] = ux; S.uy[i] = uy; S.uz[i] = uz;
    S.temp[i] = tn;
    // the XSPH pass reads buffer particles through the records
    *comp<R>(W.rec.f1, i, 0) = mn;
    *comp<R>(W.rec.f1, i, 1) = rn;
    if (P.c2_passes) pv_set_vol(W.rec.pb, i, pv_code<R>(mn / rn, ldr(W.rec.pos + i).w, S.ptype[i] == 1 || S.ptype[i] == 3));
    W.rec.ut[i] = mk4<R>(ux, uy, uz, tn);
}

// ---------------------------------------------------------------------------
// KERNEL_xsph3D_sph + KERNEL_xsph3D_calc_sph (functions_TIME.cuh:1735-1997).
// Writes the smoothed velocity/temperature of every particle (or a copy)
// into u_tmp/temp_tmp; the next reorder reads them.
// ---------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 6 : 1) k_xsph(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i];
    V4<R> ui = rec.ut[i];
    R uxi = ui.x, uyi = ui.y, uzi = ui.z, ti = ui.w;
    if (it != 1 || pt > 1000 || pt == 0 || pt == 9) {
        W.u_tmpx[i] = uxi; W.u_tmpy[i] = uyi; W.u_tmpz[i] = uzi; W.temp_tmp[i] = ti;
        return;
    }
    R th = (R)S.h[i];
    const C2Sum<R> K = c2_sum<R>(P, th);
    const PvRec<R> qi = ldr(rec.pb + i);
    const bool slow_i = pv_vol(qi) != pv_vol(qi);
    R c = (R)P.c_xsph;
    int cnt = min(W.ncnt[i], P.nb_cap);
    // the kernel's normalisation leaves the ratios below
    R tx = 0, ty = 0, tz = 0, tt = 0, flt = 0;
    const int* __restrict__ nb = W.nbr;
    nb_sum<NbP4<R>, PairV<R>>(
        cnt, nb, n, i,
        [&](int j) {
            NbP4<R> t;
            t.q = ldr(rec.pb + j);
            t.b = ldr(rec.ut + j);
            return t;
        },
        [&](const NbP4<R>& t, PairV<R>& g) { return pv_prep<R, true>(P, qi, slow_i, t.q, g); },
        [&](int j, NbP4<R>& t, PairV<R>& g) {
            int tag;
            if (!pv_fix(S, rec.pos, W.m_new, W.rho_new, slow_i, t.q, i, j, g, tag)) return;
            if (tag_ptype(tag) != 1 && tag_ptype(tag) != 3) {   // no neighbour of this sum
                g.vs = 0;
                t.b = ui;
            }
        },
        [&](int, const NbP4<R>& t, const PairV<R>& g) {
            const R v = g.vs;
            const bool in = v != (R)0;   // a wall's fields stay out of the sums
            const R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz;
            const R r = r2 * rsq_floor(r2);
            const R m = v * c2_w(K, r);
            tx += m * (in ? t.b.x - uxi : (R)0);
            ty += m * (in ? t.b.y - uyi : (R)0);
            tz += m * (in ? t.b.z - uzi : (R)0);
            tt += m * (in ? t.b.w - ti : (R)0);
            flt += m;
        });
    R on = (R)(pt > 0);
    const R iflt = c * rcp(flt);
    W.u_tmpx[i] = (uxi + tx * iflt) * on;
    W.u_tmpy[i] = (uyi + ty * iflt) * on;
    W.u_tmpz[i] = (uzi + tz * iflt) * on;
    W.temp_tmp[i] = (ti + (R)0.01 * tt * iflt) * on;
}

// ---------------------------------------------------------------------------
// The neighbour passes for any kernel and switch set (the passes above their
// own Wendland C2 forms).
// ---------------------------------------------------------------------------
// the planes xx, xy, xz, yy, yz, zz of the symmetric 3 x 3 matrix C
template <typename R>
__device__ __forceinline__ void cm_store(R* Cm, int n, int i, const R* C) {
    Cm[i] = C[0];
    Cm[(size_t)n + i] = C[1];
    Cm[(size_t)2 * n + i] = C[2];
    Cm[(size_t)3 * n + i] = C[4];
    Cm[(size_t)4 * n + i] = C[5];
    Cm[(size_t)5 * n + i] = C[8];
}
template <typename R, int KT, int L>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 8 : 1) k_passA_any(DevParams P, SphState<R> S, SphWork<R> W, DemState<double> D,
                                               DemWork<double> DW, const int4* __restrict__ drows) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i];
    R mo = S.m[i], ro = S.rho[i];
    if (it > 2) {
        W.m_new[i] = mo;
        W.rho_new[i] = ro;
        rec.f1[i] = mk4<R>(mo, ro, S.temp[i], W.DEMpor[i]);
        return;
    }
    R dprev = S.dDEMpor[i];
    if (grp.lane == 0) W.dDEMpor_prev[i] = dprev;
    double xi = S.x[i], yi = S.y[i], zi = S.z[i], hi = S.h[i];
    R th = (R)hi;
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    PosRec<R> qi = ldr(rec.pos + i);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R txx = 0, tyy = 0, tzz = 0, txy = 0, tyz = 0, tzx = 0, sflt = 0;
    const int* __restrict__ nb = W.nbr;
    const bool kgc = (P.kgc == 1);
    struct T {
        R p, w, cx, cy, cz, dx, dy, dz;
        int f;
    };
    auto load = [&](int j) {
                NbQ2<R> t;
                t.q = ldr(rec.pos + j);
                t.a = ldr(rec.mr0 + j);
                return t;
            };
    auto terms = [&](int j, const NbQ2<R>& t, T& o) {
        int ptj = tag_ptype(t.q.w);
        if (ptj > 1000) return false;
        Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
        R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
        rdist(r2, r, rinv);
        R irj = rcp(t.a.y);
        o.f = 0;
        if (ptj == 1) {
            o.f |= 1;
            o.p = t.a.x * irj;
            o.w = kw(K, r);
        }
        if (kgc && r2 > (R)0) {
            R dw = kdw(K, r);
            R c = -t.a.x * dw * irj * rinv;
            o.f |= 2;
            o.cx = c * g.dx;
            o.cy = c * g.dy;
            o.cz = c * g.dz;
            o.dx = g.dx;
            o.dy = g.dy;
            o.dz = g.dz;
        }
        return true;
    };
    auto add = [&](const T& o) {
        if (o.f & 1) sflt += o.p * o.w;
        if (o.f & 2) {
            txx += o.cx * o.dx;
            txy += o.cy * o.dx;
            tyy += o.cy * o.dy;
            tzx += o.cx * o.dz;
            tyz += o.cy * o.dz;
            tzz += o.cz * o.dz;
        }
    };
    if constexpr (L == 1)
        nb_walk<4, NbQ2<R>>(cnt, nb, n, i, load, [&](int j, const NbQ2<R>& t) {
            T o;
            if (terms(j, t, o)) add(o);
        });
    else
        ordered_walk<L, NbQ2<R>, T>(grp, cnt, [&](int k) { return __ldg(nb + nb_at(k, n, i)); }, load, terms, add);
    if (kgc && P.dim == 2) {
        // a bed in a plane y = const: the x-z block of the moment matrix
        const R det = txx * tzz - tzx * tzx;
        R C[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        if (fabs(det) > (R)1e-4) {
            const R rr = (R)1 / det;
            C[0] = tzz * rr;
            C[2] = -tzx * rr;
            C[6] = -tzx * rr;
            C[8] = txx * rr;
        }
        cm_store(W.Cm, n, i, C);
    } else if (kgc) {
        R det = txx * (tyy * tzz - tyz * tyz);
        det -= txy * (txy * tzz - tyz * tzx);
        det += tzx * (txy * tyz - tyy * tzx);
        R C[9];
        if (fabs(det) > (R)1e-4) {
            R rr = (R)1 / det;
            C[0] = (tyy * tzz - tyz * tyz) * rr;
            C[1] = (tzx * tyz - txy * tzz) * rr;
            C[2] = (txy * tyz - tzx * tyy) * rr;
            C[3] = (tzx * tyz - txy * tzz) * rr;
            C[4] = (txx * tzz - tzx * tzx) * rr;
            C[5] = (tzx * txy - txx * tyz) * rr;
            C[6] = (txy * tyz - tzx * tyy) * rr;
            C[7] = (tzx * txy - txx * tyz) * rr;
            C[8] = (txx * tyy - txy * txy) * rr;
        } else {
            C[0] = 1; C[1] = 0; C[2] = 0; C[3] = 0; C[4] = 1; C[5] = 0; C[6] = 0; C[7] = 0; C[8] = 1;
        }
        cm_store(W.Cm, n, i, C);
    }
    R por = 0, dfx = 0, dfy = 0, dfz = 0;
    if (P.nd > 0) {
        sph_dem_porosity<R, L>(P, W, D, DW, drows, grp, xi, yi, zi, hi, K, por, dfx, dfy, dfz);
    }
    if (grp.lane) return;
    R isf = rcp(sflt + (R)1e-20);
    R pori = (R)1 - por * isf;
    W.DEMpor[i] = pori;
    S.dDEMpor[i] = (dfx + dfy + dfz) * isf;
    // prep_sph
    R hd = (R)P.h_over_dx;
    R v = sph_volume(P, th, hd);
    R mref;
    if (pt == 9) mref = (R)P.rho_liquid * v * pori;
    else if (pt == -3 || pt == 0 || pt == 3 || pt == 1) mref = (R)P.rho_gas * v * pori;
    else mref = (R)P.rho_liquid * v * pori;
    if (pt == 9 && zi < 0.05) mref = (R)P.rho_gas * v * pori;
    R rref = (P.dim == 2) ? mref / ((th / hd) * (th / hd)) : mref / v;
    W.rho_ref[i] = rref;
    R mn = mo, rn = ro;
    if (P.rho_type == 1) {
        rn = mref / v;
        mn = mref;
    }
    W.rho_new[i] = rn;
    W.m_new[i] = mn;
    rec.f1[i] = mk4<R>(mn, rn, S.temp[i], pori);
}

template <typename R, bool FORCES, int KT, int L>
__global__ void __launch_bounds__(128) k_passB_any(DevParams P, SphState<R> S, SphWork<R> W, const DevFlags* F) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    // Shepard filter every freq_filt*decouple_stride steps (functions_PREP2.cuh:2120)
    const int filt = (F->step_count % P.filt_period) == 0;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    if (grp.lane == 0) {
        W.ftx[i] = 0; W.fty[i] = 0; W.ftz[i] = 0; W.ftot[i] = 0;
        W.pgfx[i] = 0; W.pgfy[i] = 0; W.pgfz[i] = 0;
        W.dtemp[i] = 0;
    }
    if (it > 2 || pt > 1000) return;
    bool adv = !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (!filt && !adv) return;
    R th = (R)S.h[i];
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    PosRec<R> qi = ldr(rec.pos + i);
    V4<R> upi = rec.up[i];
    V4<R> fi = rec.f1[i];
    R uxi = upi.x, uyi = upi.y, uzi = upi.z, pi = upi.w;
    R rhoi = fi.y, tempi = fi.z, pori = fi.w, mi = fi.x;
    R irhoi = rcp(rhoi);
    const bool kgc = (P.kgc == 1);
    Cm9<R> Cm = cm_load(W.Cm, n, i, kgc);
    R vis = (R)P.mu_gas, vis_h = (vis * vis) / (vis + vis);
    R kc = (R)P.k_sph;
    R eli = (P.sph_lagrangian != 0) ? (R)1 : (R)0;
    // per-particle factors of the pair terms
    R cp_i = -pori * irhoi * (rhoi / pori);      // rho_i/eps_i * (-eps_i / rho_i)
    R cv_i = vis_h * (R)4 * pori * irhoi;
    R visi = vis;
    if (FORCES && P.sps) visi += W.vist[i];   // viscosity + P3.vis_t (functions_PPE2.cuh:1323)
    R ch_i = (R)4 * pori * kc * kc * irhoi / (kc + kc);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R flt = 0, tx = 0, ty = 0, tz = 0, px = 0, py = 0, pz = 0, Rc = 0, ex = 0, ey = 0, ez = 0, et = 0;
    const int* __restrict__ nb = W.nbr;
    if constexpr (L > 1) {
        static_assert(!FORCES, "several lanes: the default forces, without artificial viscosity");
        struct T {
            R p, w, s, gx, gy, gz, cv, dux, duy, duz, ex, ey, ez, mr, et, rc, rr;
            int f;   // 1 filter, 2 forces
        };
        auto load = [&](int j) {
            NbQ44<R> t;
            t.q = ldr(rec.pos + j);
            t.a = ldr(rec.f1 + j);
            t.b = ldr(rec.up + j);
            return t;
        };
        auto terms = [&](int j, const NbQ44<R>& t, T& o) {
            const V4<R>& fj = t.a;
            const V4<R>& uj = t.b;
            Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
            R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
            rdist(r2, r, rinv);
            R mj = fj.x, irj = rcp(fj.y);
            o.f = 0;
            if (filt) {
                o.f |= 1;
                o.p = mj * irj;
                o.w = kw(K, r);
            }
            if (!adv || tag_ptype(t.q.w) >= 1000) return o.f != 0;
            o.f |= 2;
            R dw = kdw(K, r);
            R gx = dw * g.dx * rinv, gy = dw * g.dy * rinv, gz = dw * g.dz * rinv;
            cm_apply(Cm, kgc, gx, gy, gz);
            R tj = fj.z;
            o.gx = gx;
            o.gy = gy;
            o.gz = gz;
            o.s = cp_i * mj * (pi + uj.w) * irj;
            o.cv = (g.dx * gx + g.dy * gy + g.dz * gz) * cv_i * mj * irj * rinv * rinv;
            o.dux = uxi - uj.x;
            o.duy = uyi - uj.y;
            o.duz = uzi - uj.z;
            o.mr = mj * irj * ((R)1 - eli);
            R ug = uxi * gx + uyi * gy + uzi * gz;
            o.ex = (uj.x - uxi) * ug;
            o.ey = (uj.y - uyi) * ug;
            o.ez = (uj.z - uzi) * ug;
            o.et = (tj - tempi) * ug;
            o.rc = ch_i * mj * (tempi - tj) * dw * irj;
            o.rr = rcp(r + (R)1e-10);
            return true;
        };
        auto add = [&](const T& o) {
            if (o.f & 1) flt += o.p * o.w;
            if (!(o.f & 2)) return;
            if (P.fp != 0) {
                px += o.s * o.gx;
                py += o.s * o.gy;
                pz += o.s * o.gz;
            }
            if (P.fv != 0) {
                tx += o.cv * o.dux;
                ty += o.cv * o.duy;
                tz += o.cv * o.duz;
            }
            if (eli < (R)1) {
                ex += o.ex * o.mr;
                ey += o.ey * o.mr;
                ez += o.ez * o.mr;
                if (P.con != 0) et += o.et * o.mr;
            }
            if (P.con != 0) Rc += o.rc * o.rr;
        };
        ordered_walk<L, NbQ44<R>, T>(grp, cnt, [&](int k) { return __ldg(nb + nb_at(k, n, i)); }, load, terms, add);
    } else {
    nb_walk<4, NbQ44<R>>(
        cnt, nb, n, i,
        [&](int j) {
            NbQ44<R> t;
            t.q = ldr(rec.pos + j);
            t.a = ldr(rec.f1 + j);
            t.b = ldr(rec.up + j);
            return t;
        },
        [&](int j, const NbQ44<R>& t) {
            const V4<R>& fj = t.a;
            const V4<R>& uj = t.b;
            Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
            R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
            rdist(r2, r, rinv);
            R mj = fj.x, irj = rcp(fj.y);
            if (filt) flt += mj * irj * kw(K, r);
            if (!adv || tag_ptype(t.q.w) >= 1000) return;
            R dw = kdw(K, r);
            R gx = dw * g.dx * rinv, gy = dw * g.dy * rinv, gz = dw * g.dz * rinv;
            cm_apply(Cm, kgc, gx, gy, gz);
            R tj = fj.z;
            if ((P.fp != 0)) {
                R s = cp_i * mj * (pi + uj.w) * irj;
                px += s * gx;
                py += s * gy;
                pz += s * gz;
            }
            if ((P.fv != 0)) {
                R cv = cv_i;
                if (FORCES && P.sps) {
                    // harmonic mean of the two particles' viscosity + vis_t
                    const R visj = vis + W.vist[j];
                    cv = visi * visj / (visi + visj) * (R)4 * pori * irhoi;
                }
                R Cv = (g.dx * gx + g.dy * gy + g.dz * gz) * cv * mj * irj * rinv * rinv;
                tx += Cv * (uxi - uj.x);
                ty += Cv * (uyi - uj.y);
                tz += Cv * (uzi - uj.z);
            }
            if ((P.fva != 0)) {
                R uij = (uxi - uj.x) * g.dx + (uyi - uj.y) * g.dy + (uzi - uj.z) * g.dz;
                if (uij < (R)0) {
                    R hij = (th + th) * (R)0.5;
                    R phi = hij * uij / (r * r + (R)0.01 * hij * hij);
                    R Pij = mi * phi * ((R)-0.1 * (R)P.soundspeed + (R)0.02 * phi) / (rhoi + fj.y) * (R)0.5;
                    tx += -Pij * gx;
                    ty += -Pij * gy;
                    tz += -Pij * gz;
                }
            }
            if (FORCES) {
                const int ptj = tag_ptype(t.q.w);
                if (P.iface) {
                    // interface sharpness force (functions_PPE2.cuh:1450-1464): raw
                    // kernel slope; the neighbour's pressure only across a fluid-fluid
                    // interface (wall 0 and moving 9 excluded)
                    const bool flag = (pt != 0) && (pt != 9) && (ptj != 0) && (ptj != 9) && (pt != ptj);
                    const R mri = mi * irhoi, mrj = mj * irj;
                    R Ci = fabs(pi) * mri * mri + fabs(uj.w) * mrj * mrj * (R)flag;
                    Ci *= ((R)0.08 / mi) * dw * rinv;
                    tx += Ci * -g.dx;
                    ty += Ci * -g.dy;
                    tz += Ci * -g.dz;
                }
                if (P.fb && pt == 1 && ptj != 1) {
                    // repulsive force of non-fluid neighbours (functions_PPE2.cuh:1465-1472)
                    const R rr = r + (R)1e-10;
                    const R fb = (R)P.c_repulsive / rr / rr * kw(K, r) * ((R)2 * mj / (mi + mj));
                    tx += fb * g.dx;
                    ty += fb * g.dy;
                    tz += fb * g.dz;
                }
                if (P.ipf && pt == 1 && ptj == 1) {
                    // inter-particle surface tension (functions_PPE2.cuh:1490-1542): of the
                    // pair strengths of Parameters.cuh:134-148 only fluid-fluid (s_ff1 =
                    // 1.1e-6) is non-zero and every A is zero, so
                    // Cs = -s_ff1 w_ipf / (m_i (r + 1e-10)) with the cosine kernel
                    // w_ipf = -cos(3 pi / 4 r / h) for r < 2h (functions_INTERACTION.cuh:1-33)
                    const R tR = r * rcp(th);
                    const R wipf = tR < (R)2 ? -cos((R)(3.0 * 3.141592653 / 4.0) * tR) : (R)0;
                    const R Cs = -((R)1.1e-6 * (wipf / (mi * (r + (R)1e-10))));
                    tx += Cs * g.dx;
                    ty += Cs * g.dy;
                    tz += Cs * g.dz;
                }
            }
            if (eli < (R)1) {
                R mr = mj * irj * ((R)1 - eli);
                R ug = uxi * gx + uyi * gy + uzi * gz;
                ex += (uj.x - uxi) * ug * mr;
                ey += (uj.y - uyi) * ug * mr;
                ez += (uj.z - uzi) * ug * mr;
                if ((P.con != 0)) et += (tj - tempi) * ug * mr;
            }
            if ((P.con != 0)) Rc += ch_i * mj * (tempi - tj) * dw * irj * rcp(r + (R)1e-10);
        });
    }
    if (grp.lane) return;
    if (filt) S.flt_s[i] = flt;
    if (!adv) return;
    if (P.fg) tz += -(R)P.g_sph;
    W.ftx[i] = tx - ex;
    W.fty[i] = ty - ey;
    W.ftz[i] = tz - ez;
    W.ftot[i] = sqrt(tx * tx + ty * ty + tz * tz);
    W.pgfx[i] = px;
    W.pgfy[i] = py;
    W.pgfz[i] = pz;
    if ((P.con != 0)) W.dtemp[i] = Rc / (R)P.cp_sph * (R)(pt != -1) - et;
}

template <typename R, int KT, int L>
__global__ void __launch_bounds__(128) k_ppe_any(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    V4<R> upi = rec.up[i];
    bool solve = it <= 2 && !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (!solve) {
        W.p_new[i] = upi.w;
        return;
    }
    R th = (R)S.h[i];
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    PosRec<R> qi = ldr(rec.pos + i);
    V4<R> fi = rec.f1[i];
    R uxi = upi.x, uyi = upi.y, uzi = upi.z, rhoi = fi.y, pori = fi.w;
    R irhoi = rcp(rhoi), prhoi = pori * rhoi;
    R pux = pori * uxi, puy = pori * uyi, puz = pori * uzi;
    const bool kgc = (P.kgc == 1);
    Cm9<R> Cm = cm_load(W.Cm, n, i, kgc);
    int cnt = min(W.ncnt[i], P.nb_cap);
    R bx = 0, by = 0, bz = 0, A = 0, AP = 0;
    const int* __restrict__ nb = W.nbr;
    struct T {
        R vx, vy, vz, gx, gy, gz, a, c, p;
    };
    auto load = [&](int j) {
                NbQ44<R> t;
                t.q = ldr(rec.pos + j);
                t.a = ldr(rec.f1 + j);
                t.b = ldr(rec.up + j);
                return t;
            };
    auto terms = [&](int j, const NbQ44<R>& t, T& o) {
        int tj = t.q.w;
        if (tag_ptype(tj) >= 1000 || tag_itype(tj) == 4) return false;
        const V4<R>& fj = t.a;
        const V4<R>& uj = t.b;
        Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
        R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
        rdist(r2, r, rinv);
        R mj = fj.x, rhoj = fj.y, porj = fj.w, irj = rcp(rhoj);
        R dw = kdw(K, r);
        R gx = dw * g.dx * rinv, gy = dw * g.dy * rinv, gz = dw * g.dz * rinv;
        cm_apply(Cm, kgc, gx, gy, gz);
        R mr = mj * irj;
        o.vx = mr * (pux - porj * uj.x);
        o.vy = mr * (puy - porj * uj.y);
        o.vz = mr * (puz - porj * uj.z);
        o.gx = gx;
        o.gy = gy;
        o.gz = gz;
        o.c = -(g.dx * gx + g.dy * gy + g.dz * gz) * rinv * rinv;
        o.a = mj * ((prhoi + porj * rhoj) * irj * irhoi);
        o.p = uj.w;
        return true;
    };
    auto add = [&](const T& o) {
        bx += o.vx * o.gx;
        by += o.vy * o.gy;
        bz += o.vz * o.gz;
        const R a = o.a * o.c;
        A += a;
        AP += a * o.p;
    };
    if constexpr (L == 1)
        nb_walk<4, NbQ44<R>>(cnt, nb, n, i, load, [&](int j, const NbQ44<R>& t) {
            T o;
            if (terms(j, t, o)) add(o);
        });
    else
        ordered_walk<L, NbQ44<R>, T>(grp, cnt, [&](int k) { return __ldg(nb + nb_at(k, n, i)); }, load, terms, add);
    if (grp.lane) return;
    R b = (R)P.rho_gas * (bx + by + bz + (R)2 * S.dDEMpor[i] - W.dDEMpor_prev[i]) / (R)P.sdt;
    W.p_new[i] = (b + AP) / A;
}

template <typename R, int KT, int L>
__global__ void __launch_bounds__(128) k_passC_any(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i], bt = S.btype[i];
    if (grp.lane == 0) W.fpx[i] = 0, W.fpy[i] = 0, W.fpz[i] = 0;
    if (it > 2) {
        rec.ut[i] = mk4<R>(S.ux[i], S.uy[i], S.uz[i], S.temp[i]);
        return;
    }
    R fx = 0, fy = 0, fz = 0;
    bool pf = !(P.open_bc > 0 && bt > 0) && pt < 1000 && pt > 0;
    if (pf && (P.fp != 0)) {
        R th = (R)S.h[i];
        Knl<R, KT> K = knl_make<R, KT>(P, th);
        PosRec<R> qi = ldr(rec.pos + i);
        R pi = W.p_new[i], rhoi = W.rho_new[i], pori = rec.f1[i].w;
        R cpi = -pori * rcp(rhoi);
        const bool kgc = (P.kgc == 1);
        Cm9<R> Cm = cm_load(W.Cm, n, i, kgc);
        int cnt = min(W.ncnt[i], P.nb_cap);
        const int* __restrict__ nb = W.nbr;
        const R* __restrict__ pn = W.p_new;
        struct T {
            R c, gx, gy, gz;
        };
        auto load = [&](int j) {
                        NbQ2S<R> t;
                        t.q = ldr(rec.pos + j);
                        t.a = ldr(reinterpret_cast<const V2<R>*>(rec.f1 + j));
                        t.s = __ldg(pn + j);
                        return t;
                    };
        auto terms = [&](int j, const NbQ2S<R>& t, T& o) {
            if (tag_ptype(t.q.w) >= 1000) return false;
            Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
            R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
            rdist(r2, r, rinv);
            R dw = kdw(K, r);
            o.gx = dw * g.dx * rinv;
            o.gy = dw * g.dy * rinv;
            o.gz = dw * g.dz * rinv;
            cm_apply(Cm, kgc, o.gx, o.gy, o.gz);
            o.c = cpi * t.a.x * (pi + t.s) * rcp(t.a.y);
            return true;
        };
        auto add = [&](const T& o) {
            fx += o.c * o.gx;
            fy += o.c * o.gy;
            fz += o.c * o.gz;
        };
        if constexpr (L == 1)
            nb_walk<4, NbQ2S<R>>(cnt, nb, n, i, load, [&](int j, const NbQ2S<R>& t) {
                T o;
                if (terms(j, t, o)) add(o);
            });
        else
            ordered_walk<L, NbQ2S<R>, T>(grp, cnt, [&](int k) { return __ldg(nb + nb_at(k, n, i)); }, load, terms, add);
        if (grp.lane == 0) W.fpx[i] = fx, W.fpy[i] = fy, W.fpz[i] = fz;
    }
    if (grp.lane) return;
    if (pt == 9) {
        rec.ut[i] = mk4<R>(S.ux[i], S.uy[i], S.uz[i], S.temp[i]);
        return;
    }
    R ux0, uy0, uz0, ax, ay, az;
    if (pt > 0) {
        ux0 = S.ux[i]; uy0 = S.uy[i]; uz0 = S.uz[i];
        R b = (R)(bt == 0);
        ax = fx * b; ay = fy * b; az = fz * b;
    } else {
        ux0 = W.ux0[i]; uy0 = W.uy0[i]; uz0 = W.uz0[i];
        ax = ay = az = (R)0;
    }
    R dt = (R)P.sdt;
    R uxc = ux0 + ax * dt, uyc = uy0 + ay * dt, uzc = uz0 + az * dt;
    R lim = (R)P.u_limit;
    if ((uxc * uxc + uyc * uyc + uzc * uzc) >= lim * lim) {
        uxc = ux0; uyc = uy0; uzc = uz0;
    }
    if (!P.xsph && (P.sph_lagrangian != 0) && pt > 0) {
        S.x[i] += ((double)W.ux0[i] + (double)uxc) / 2.0 * P.sdt;
        S.y[i] += ((double)W.uy0[i] + (double)uyc) / 2.0 * P.sdt;
        S.z[i] += ((double)W.uz0[i] + (double)uzc) / 2.0 * P.sdt;
    }
    S.ux[i] = uxc; S.uy[i] = uyc; S.uz[i] = uzc;
    R tn = S.temp[i];
    if ((P.con != 0) && pt > 0) {
        tn = W.temp0[i] + W.dtemp[i] * dt * (R)(pt != -1);
        S.temp[i] = tn;
    }
    rec.ut[i] = mk4<R>(uxc, uyc, uzc, tn);
}

template <typename R, int KT, int L>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 6 : 1) k_xsph_any(DevParams P, SphState<R> S, SphWork<R> W) {
    grid_dep_wait();
    const LaneGroup<L> grp;
    const int i = grp.i;
    int n = P.ns;
    if (i >= n) return;
    const SphRec<R> rec = W.rec;
    int it = S.itype[i], pt = S.ptype[i];
    V4<R> ui = rec.ut[i];
    R uxi = ui.x, uyi = ui.y, uzi = ui.z, ti = ui.w;
    if (it != 1 || pt > 1000 || pt == 0 || pt == 9) {
        W.u_tmpx[i] = uxi; W.u_tmpy[i] = uyi; W.u_tmpz[i] = uzi; W.temp_tmp[i] = ti;
        return;
    }
    R th = (R)S.h[i];
    Knl<R, KT> K = knl_make<R, KT>(P, th);
    PosRec<R> qi = ldr(rec.pos + i);
    R c = (R)P.c_xsph;
    int cnt = min(W.ncnt[i], P.nb_cap);
    R tx = 0, ty = 0, tz = 0, tt = 0, flt = 0;
    const int* __restrict__ nb = W.nbr;
    struct T {
        R p, w, ux, uy, uz, t;
    };
    auto load = [&](int j) {
                NbQ24<R> t;
                t.q = ldr(rec.pos + j);
                t.a = ldr(reinterpret_cast<const V2<R>*>(rec.f1 + j));
                t.b = ldr(rec.ut + j);
                return t;
            };
    auto terms = [&](int j, const NbQ24<R>& t, T& o) {
        int ptj = tag_ptype(t.q.w);
        if (ptj != 1 && ptj != 3) return false;
        Disp<R> g = disp(P, qi, t.q, S.x, S.y, S.z, i, j);
        R r2 = g.dx * g.dx + g.dy * g.dy + g.dz * g.dz, r, rinv;
        rdist(r2, r, rinv);
        R w = kw(K, r);
        o.p = t.a.x * rcp(t.a.y);
        o.w = w;
        o.ux = t.b.x - uxi;
        o.uy = t.b.y - uyi;
        o.uz = t.b.z - uzi;
        o.t = t.b.w - ti;
        return true;
    };
    auto add = [&](const T& o) {
        R m = o.p * o.w;
        R cm = c * m;
        tx += cm * o.ux;
        ty += cm * o.uy;
        tz += cm * o.uz;
        tt += (R)0.01 * cm * o.t;
        flt += m;
    };
    if constexpr (L == 1)
        nb_walk<4, NbQ24<R>>(cnt, nb, n, i, load, [&](int j, const NbQ24<R>& t) {
            T o;
            if (terms(j, t, o)) add(o);
        });
    else
        ordered_walk<L, NbQ24<R>, T>(grp, cnt, [&](int k) { return __ldg(nb + nb_at(k, n, i)); }, load, terms, add);
    if (grp.lane) return;
    R on = (R)(pt > 0);
    R iflt = rcp(flt);
    W.u_tmpx[i] = (uxi + tx * iflt) * on;
    W.u_tmpy[i] = (uyi + ty * iflt) * on;
    W.u_tmpz[i] = (uzi + tz * iflt) * on;
    W.temp_tmp[i] = (ti + tt * iflt) * on;
}

// end of a step: the host loop's count++ (ISPH_Calc_seperate.cuh:925)
__global__ void k_tick(DevFlags* F) {
    grid_dep_wait(); F->step_count += 1; }

// ---------------------------------------------------------------------------
// printed maxima (kernel_copy_max_*, functions_OUTPUT.cuh:19-65 + cub max)
// out[0..2] = rho, |u|, ftotal over p_type!=0 && i_type<2 (zeroed by the
// caller).  Grid-stride blocks; block maxima are combined with an integer
// atomicMax on the bit patterns, which orders non-negative doubles.
// ---------------------------------------------------------------------------
template <typename R, typename RR = R>
__global__ void __launch_bounds__(256) k_stats(int n, const RR* __restrict__ rho, const R* __restrict__ ux,
                                               const R* __restrict__ uy, const R* __restrict__ uz,
                                               const R* __restrict__ ft, const int* __restrict__ ptype,
                                               const int* __restrict__ itype, double* out, DevFlags* F) {
    __shared__ double sm[3][256];
    double a = 0, b = 0, c = 0;
    int bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double uzi = uz ? (double)uz[i] : 0.0;   // 2-D sets pass no uz
        double u = sqrt((double)ux[i] * ux[i] + (double)uy[i] * uy[i] + uzi * uzi);
        if (!isfinite(u) || !isfinite((double)rho[i])) bad = 1;
        if (ptype[i] == 0 || itype[i] >= 2) continue;
        a = fmax(a, (double)rho[i]);
        b = fmax(b, u);
        c = fmax(c, ft ? (double)ft[i] : 0.0);
    }
    sm[0][threadIdx.x] = a; sm[1][threadIdx.x] = b; sm[2][threadIdx.x] = c;
    if (bad) atomicOr(&F->nan, 1);
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int q = 0; q < 3; q++) sm[q][threadIdx.x] = fmax(sm[q][threadIdx.x], sm[q][threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; q++)
            atomicMax(reinterpret_cast<unsigned long long*>(out + q), (unsigned long long)__double_as_longlong(sm[q][0]));
}

}  // namespace sphdem
