// records.cuh -- packed per-particle records read by the neighbour passes.
//
// A neighbour pass reads a handful of fields of every neighbour j.  Read
// from separate SoA arrays that is one scattered load (and one 32-byte
// sector) per field and neighbour; the passes were bound by the latency of
// those loads.  The records below put what a pass reads of j into one or
// two aligned vectors, so a neighbour costs 2-4 vector loads:
//
//   PosRec  position + type tag      written by the cell gather (NNPS)
//     FP32 build: int4 {qx, qy, qz, tag}; q = round((x - o) / s) with the
//       origin o at the centre of the cell-grid box and s = extent / 2^30
//       per axis.  Differences of two fixed-point positions are exact
//       integers; one int->float conversion and a multiply give the
//       displacement with an absolute error below s (3.7e-10 m on a 0.4 m
//       axis), against 6e-8 relative for rounding a double difference.
//       Positions farther than one extent from the centre set the OOR tag
//       bit; pairs with that bit take their displacement from the double
//       positions.
//     FP64 build: {double x, y, z; int tag}: the exact double positions.
//   tag = p_type << 16 | buffer_type << 5 | OOR << 4 | i_type
//   MR0  {m, rho}                      start of step (cell gather)
//   F1   {m_new, rho_new, temp, DEMpor} pass A; walls' rho_new is patched by
//                                      the Neumann wall pass
//   UP   {ux, uy, uz, pres}            cell gather; u* by the SPH predictor,
//                                      wall pressure by the first Neumann pass
//   UT   {ux, uy, uz, temp}            corrector (pass C), patched by the
//                                      open-boundary pass for buffer particles
// Wendland C2 (the configurations' kernel), read by its own passes:
//   PA   position + V0 = m / rho       start of step (cell gather), read by pass A
//   PB   position + V = m' / rho'      pass A; V of walls patched by the Neumann
//                                      pass, of buffers by the open-boundary pass
//   PU   {eps u*, p}                   SPH predictor, read by the pressure equation;
//                                      wall pressure by the first Neumann pass
//   RP   eps rho'                      pass A; walls patched by the Neumann pass
// A pair of the neighbour sums needs of j only its displacement, its volume
// m / rho and one more vector, so PA and PB carry the volume in the fourth
// word of the position record and the passes load 16 to 36 bytes per pair
// (24 to 48 with {m, rho, ...} beside the tagged position; the passes were
// bound by L1 wavefronts and issue slots).  The sign of the volume tells the
// types that the Shepard sums take (PA: p_type 1; PB: 1 or 3) from the
// others, and a NaN volume marks a particle that a pass cannot take from the
// record alone (outside the fixed-point range, p_type >= 1000, or a volume that
// is not >= 0): pv_slow reads that pair from the tagged records and the double
// positions.  Parked slots (i_type 3) are in no list; pass A leaves theirs unset.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "device_common.cuh"

namespace sphdem {

struct __align__(32) Dbl4 {
    double x, y, z, w;
};
struct __align__(32) QPos64 {
    double x, y, z;
    int w, pad;
};

template <typename R>
struct Vec;
template <>
struct Vec<float> {
    typedef float4 v4;
    typedef float2 v2;
    typedef int4 pos;
    typedef int4 pv;
};
template <>
struct Vec<double> {
    typedef Dbl4 v4;
    typedef double2 v2;
    typedef QPos64 pos;
    typedef Dbl4 pv;
};

template <typename R>
using V4 = typename Vec<R>::v4;
template <typename R>
using V2 = typename Vec<R>::v2;
template <typename R>
using PosRec = typename Vec<R>::pos;
template <typename R>
using PvRec = typename Vec<R>::pv;   // position + volume

// ---- tag -----------------------------------------------------------------
constexpr int TAG_OOR = 1 << 4;
__host__ __device__ __forceinline__ int make_tag(int ptype, int btype, int itype, int oor) {
    return (int)((unsigned)ptype << 16) | ((btype & 7) << 5) | (oor ? TAG_OOR : 0) | (itype & 15);
}
__device__ __forceinline__ int tag_ptype(int t) { return t >> 16; }
__device__ __forceinline__ int tag_btype(int t) { return (t >> 5) & 7; }
__device__ __forceinline__ int tag_itype(int t) { return t & 15; }

// ---- vector loads / stores (read-only path for the neighbour loads) ------
__device__ __forceinline__ float4 ldr(const float4* p) { return __ldg(p); }
__device__ __forceinline__ float2 ldr(const float2* p) { return __ldg(p); }
__device__ __forceinline__ int4 ldr(const int4* p) { return __ldg(p); }
__device__ __forceinline__ double2 ldr(const double2* p) { return __ldg(p); }
__device__ __forceinline__ Dbl4 ldr(const Dbl4* p) {   // one 32-byte load
    Dbl4 v;
    asm volatile("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ double ldr(const double* p) { return __ldg(p); }
__device__ __forceinline__ float ldr(const float* p) { return __ldg(p); }
__device__ __forceinline__ QPos64 ldr(const QPos64* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    double2 a = __ldg(q), b = __ldg(q + 1);
    QPos64 r;
    r.x = a.x; r.y = a.y; r.z = b.x;
    r.w = __double_as_longlong(b.y) & 0xffffffff;
    r.pad = 0;
    return r;
}
// plain (coherent) loads for records written earlier in the same kernel
__device__ __forceinline__ float4 ldc(const float4* p) { return *p; }
__device__ __forceinline__ Dbl4 ldc(const Dbl4* p) { return *p; }

template <typename R>
__device__ __forceinline__ V4<R> mk4(R a, R b, R c, R d);
template <>
__device__ __forceinline__ float4 mk4<float>(float a, float b, float c, float d) { return make_float4(a, b, c, d); }
template <>
__device__ __forceinline__ Dbl4 mk4<double>(double a, double b, double c, double d) { return Dbl4{a, b, c, d}; }
template <typename R>
__device__ __forceinline__ V2<R> mk2(R a, R b);
template <>
__device__ __forceinline__ float2 mk2<float>(float a, float b) { return make_float2(a, b); }
template <>
__device__ __forceinline__ double2 mk2<double>(double a, double b) { return make_double2(a, b); }

// component pointers for single-field patches (walls, buffers)
template <typename R>
__device__ __forceinline__ R* comp(V4<R>* p, int i, int c) { return reinterpret_cast<R*>(p + i) + c; }

// ---- position records ------------------------------------------------------
__device__ __forceinline__ int quantize(double v, double o, double inv, int& oor) {
    double t = __dmul_rn(__dsub_rn(v, o), inv);
    if (!(fabs(t) < 1073741823.0)) {   // |t| < 2^30 - 1; NaN lands here too
        oor = 1;
        return 0;
    }
    return __double2int_rn(t);
}

template <typename R>
__device__ __forceinline__ PosRec<R> make_pos(const DevParams& P, double x, double y, double z, int ptype, int btype,
                                              int itype);
template <>
__device__ __forceinline__ int4 make_pos<float>(const DevParams& P, double x, double y, double z, int ptype, int btype,
                                                int itype) {
    int oor = 0;
    int qx = quantize(x, P.q_org[0], P.q_inv[0], oor);
    int qy = quantize(y, P.q_org[1], P.q_inv[1], oor);
    int qz = quantize(z, P.q_org[2], P.q_inv[2], oor);
    return make_int4(qx, qy, qz, make_tag(ptype, btype, itype, oor));
}
template <>
__device__ __forceinline__ QPos64 make_pos<double>(const DevParams& P, double x, double y, double z, int ptype,
                                                   int btype, int itype) {
    QPos64 q;
    q.x = x; q.y = y; q.z = z;
    q.w = make_tag(ptype, btype, itype, 0);
    q.pad = 0;
    return q;
}
__device__ __forceinline__ void store_pos(int4* p, int i, const int4& v) { p[i] = v; }
__device__ __forceinline__ void store_pos(QPos64* p, int i, const QPos64& v) {
    double2* q = reinterpret_cast<double2*>(p + i);
    q[0] = make_double2(v.x, v.y);
    q[1] = make_double2(v.z, __longlong_as_double((long long)(unsigned)v.w));
}

// displacement x_i - x_j in field precision
template <typename R>
struct Disp {
    R dx, dy, dz;
};
__device__ __forceinline__ Disp<float> disp(const DevParams& P, const int4& a, const int4& b, const double* X,
                                            const double* Y, const double* Z, int i, int j) {
    Disp<float> d;
    if (((a.w | b.w) & TAG_OOR) == 0) {
        d.dx = (float)(a.x - b.x) * P.q_step[0];
        d.dy = (float)(a.y - b.y) * P.q_step[1];
        d.dz = (float)(a.z - b.z) * P.q_step[2];
    } else {
        d.dx = (float)(X[i] - X[j]);
        d.dy = (float)(Y[i] - Y[j]);
        d.dz = (float)(Z[i] - Z[j]);
    }
    return d;
}
__device__ __forceinline__ Disp<double> disp(const DevParams&, const QPos64& a, const QPos64& b, const double*,
                                             const double*, const double*, int, int) {
    return Disp<double>{a.x - b.x, a.y - b.y, a.z - b.z};
}
// displacement from a point given in double (mirror points, DEM centres)
__device__ __forceinline__ Disp<float> disp_pt(const DevParams& P, const int4& qp, const int4& b, double px, double py,
                                               double pz, const double* X, const double* Y, const double* Z, int j) {
    if (((qp.w | b.w) & TAG_OOR) == 0)
        return Disp<float>{(float)(qp.x - b.x) * P.q_step[0], (float)(qp.y - b.y) * P.q_step[1],
                           (float)(qp.z - b.z) * P.q_step[2]};
    return Disp<float>{(float)(px - X[j]), (float)(py - Y[j]), (float)(pz - Z[j])};
}
__device__ __forceinline__ Disp<double> disp_pt(const DevParams&, const QPos64&, const QPos64& b, double px, double py,
                                                double pz, const double*, const double*, const double*, int) {
    return Disp<double>{px - b.x, py - b.y, pz - b.z};
}

// ---- exact pair predicate with a fixed-point prefilter -----------------
// in == (sqrt(dx^2+dy^2+dz^2) + add < Rr) evaluated in FP64 exactly as the
// reference writes it (no contraction).  The FP32 build first compares the
// squared fixed-point displacement with Rr^2 (1 -/+ band); its error is
// below 2.5e-6 relative plus 3.5 steps/Rr, and band = 2e-6 + 8 steps/Rr
// covers both, so only pairs inside the band take the FP64 evaluation.
// d and r2 come back in field precision for the caller's sums.
struct Band {
    float lo, hi;
};
// FP64 build: a squared distance (rounded by less than 1e-15 of itself) that
// decides the predicate without the square root
__device__ __forceinline__ bool far64(double r2, double Rr) { return r2 > Rr * Rr * (1.0 + 4e-15); }
__device__ __forceinline__ Band make_band(const DevParams& P, double Rr) {
    double b = 2e-6 + P.q_abs / Rr;
    double r2 = Rr * Rr;
    return Band{(float)(r2 * (1.0 - b)), (float)(r2 * (1.0 + b))};
}
__device__ __forceinline__ bool test_pair(const DevParams& P, const int4& a, const int4& b, double ax, double ay,
                                          double az, const double* X, const double* Y, const double* Z, int j,
                                          double Rr, double add, Band bd, Disp<float>& d, float& r2) {
    if (((a.w | b.w) & TAG_OOR) == 0) {
        d.dx = (float)(a.x - b.x) * P.q_step[0];
        d.dy = (float)(a.y - b.y) * P.q_step[1];
        d.dz = (float)(a.z - b.z) * P.q_step[2];
        r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
        if (r2 < bd.lo) return true;
        if (r2 > bd.hi) return false;
    } else {
        d.dx = (float)(ax - X[j]);
        d.dy = (float)(ay - Y[j]);
        d.dz = (float)(az - Z[j]);
        r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
    }
    return __dadd_rn(pair_dist(ax, ay, az, X[j], Y[j], Z[j]), add) < Rr;
}
// test_pair for the two forms of the predicate at once: in0 with add = 0,
// in20 with add = 1e-20 (in20 implies in0); one prefilter, one FP64 distance
__device__ __forceinline__ void test_pair2(const DevParams& P, const int4& a, const int4& b, double ax, double ay,
                                           double az, const double* X, const double* Y, const double* Z, int j,
                                           double Rr, Band bd, Disp<float>& d, float& r2, bool& in0, bool& in20) {
    if (((a.w | b.w) & TAG_OOR) == 0) {
        d.dx = (float)(a.x - b.x) * P.q_step[0];
        d.dy = (float)(a.y - b.y) * P.q_step[1];
        d.dz = (float)(a.z - b.z) * P.q_step[2];
        r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
        if (r2 < bd.lo) { in0 = in20 = true; return; }
        if (r2 > bd.hi) { in0 = in20 = false; return; }
    } else {
        d.dx = (float)(ax - X[j]);
        d.dy = (float)(ay - Y[j]);
        d.dz = (float)(az - Z[j]);
        r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
    }
    const double r = pair_dist(ax, ay, az, X[j], Y[j], Z[j]);
    in0 = __dadd_rn(r, 0.0) < Rr;
    in20 = __dadd_rn(r, 1e-20) < Rr;
}
__device__ __forceinline__ void test_pair2(const DevParams&, const QPos64&, const QPos64& b, double ax, double ay,
                                           double az, const double*, const double*, const double*, int, double Rr,
                                           Band, Disp<double>& d, double& r2, bool& in0, bool& in20) {
    d.dx = ax - b.x;
    d.dy = ay - b.y;
    d.dz = az - b.z;
    r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
    if (far64(r2, Rr)) { in0 = in20 = false; return; }
    const double r = pair_dist(ax, ay, az, b.x, b.y, b.z);
    in0 = __dadd_rn(r, 0.0) < Rr;
    in20 = __dadd_rn(r, 1e-20) < Rr;
}
__device__ __forceinline__ bool test_pair(const DevParams&, const QPos64&, const QPos64& b, double ax, double ay,
                                          double az, const double*, const double*, const double*, int, double Rr,
                                          double add, Band, Disp<double>& d, double& r2) {
    d.dx = ax - b.x;
    d.dy = ay - b.y;
    d.dz = az - b.z;
    r2 = d.dx * d.dx + d.dy * d.dy + d.dz * d.dz;
    if (far64(r2, Rr)) return false;
    if (r2 < Rr * Rr * (1.0 - 4e-15) && add < 1e-17 * Rr) return true;
    return __dadd_rn(pair_dist(ax, ay, az, b.x, b.y, b.z), add) < Rr;
}

// ---- pair distance, reciprocal ----------------------------------------------
// r = |d| + 1e-20 and 1/r as the reference forms them
// (sqrt(dx^2+dy^2+dz^2) + 1e-20).  FP32: rsqrt (2 ulp) instead of an IEEE
// sqrt and divide; the self pair (d = 0) gives r = 1e-20, 1/r = 1e20.
__device__ __forceinline__ void rdist(float r2, float& r, float& rinv) {
    if (r2 > 0.f) {
        float s = rsqrtf(r2);
        r = r2 * s;
        rinv = s;
    } else {
        r = 1e-20f;
        rinv = 1e20f;
    }
}
__device__ __forceinline__ void rdist(double r2, double& r, double& rinv) {
    r = sqrt(r2) + 1e-20;
    rinv = 1.0 / r;
}
__device__ __forceinline__ float rcp(float a) { return __fdividef(1.0f, a); }
__device__ __forceinline__ double rcp(double a) { return 1.0 / a; }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double fdiv(double a, double b) { return a / b; }

// ---- smoothing kernel with per-particle constants -----------------------
// W and dW/dr of functions_KNL.cuh:2-144 with 1/h precomputed.
// KT is the kernel type when the kernel instantiation fixes it (3: Wendland
// C2, 5: Wendland C6; the loops then carry no type test), -1 when it is read
// from kt.
template <typename R, int KT = -1>
struct Knl {
    static_assert(KT == -1 || KT == 3 || KT == 5, "kernel types fixed at compile time: Wendland C2 and C6");
    int kt;
    R tA, ih, th;   // normalisation, 1/h, h
};
template <typename R, int KT = -1>
__device__ __forceinline__ Knl<R, KT> knl_make(const DevParams& P, R th) {
    Knl<R, KT> k;
    k.kt = P.kernel_type;
    k.tA = knl_tmpA<R>(P.kernel_type, P.dim, th);
    k.ih = rcp(th);
    k.th = th;
    return k;
}
// The other kernel types (Gaussian, cubic/quintic splines, Wendland C4) are
// called out of line: inlined into every neighbour loop, their exp/pow
// code held registers and kept the loops from being scheduled well even
// when the Wendland branches run.
template <typename R>
__device__ __noinline__ R knl_w_call(int kt, R tA, R tH, R rr) {
    return knl_w<R>(kt, tA, tH, rr);
}
template <typename R>
__device__ __noinline__ R knl_dw_call(int kt, R tA, R tH, R rr) {
    return knl_dw<R>(kt, tA, tH, rr);
}
template <typename R, int KT>
__device__ __forceinline__ R kw(const Knl<R, KT>& k, R rr) {
    if (KT == 3 || (KT == -1 && k.kt == 3)) {
        R q = rr * k.ih * (R)0.5;
        if (!(q < (R)1)) return (R)0;
        R a = (R)1 - q, a2 = a * a;
        return k.tA * a2 * a2 * ((R)1 + (R)4 * q);
    }
    if constexpr (KT != 3) {
        if (KT == 5 || k.kt == 5) {
            R q = rr * k.ih * (R)0.5;
            if (!(q < (R)1)) return (R)0;
            R a = (R)1 - q, a2 = a * a, a4 = a2 * a2;
            return k.tA * a4 * a4 * ((R)1 + (R)8 * q + (R)25 * q * q + (R)32 * q * q * q);
        }
        if constexpr (KT == -1) return knl_w_call<R>(k.kt, k.tA, k.th, rr);
    }
    return (R)0;
}
template <typename R, int KT>
__device__ __forceinline__ R kdw(const Knl<R, KT>& k, R rr) {
    if (KT == 3 || (KT == -1 && k.kt == 3)) {
        R q = rr * k.ih * (R)0.5;
        if (!(q < (R)1)) return (R)0;
        R a = (R)1 - q;
        return ((R)0.5 * k.ih) * k.tA * ((R)-20 * q * a * a * a);
    }
    if constexpr (KT != 3) {
        if (KT == 5 || k.kt == 5) {
            R q = rr * k.ih * (R)0.5;
            if (!(q < (R)1)) return (R)0;
            R a = (R)1 - q, a2 = a * a, a4 = a2 * a2;
            return ((R)0.5 * k.ih) * k.tA * ((R)-22 * q * a4 * a2 * a * ((R)16 * q * q + (R)7 * q + (R)1));
        }
        if constexpr (KT == -1) return knl_dw_call<R>(k.kt, k.tA, k.th, rr);
    }
    return (R)0;
}

// ---- gradient correction with the matrix held in registers --------------
template <typename R>
struct Cm9 {
    R c[9];
};
template <typename R>
__device__ __forceinline__ Cm9<R> cm_load(const R* __restrict__ Cm, int n, int i, int on) {
    // six stored planes (xx, xy, xz, yy, yz, zz) of the symmetric matrix
    constexpr int plane[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    Cm9<R> m;
#pragma unroll
    for (int q = 0; q < 9; q++) m.c[q] = on ? Cm[(size_t)plane[q] * n + i] : (R)((q % 4) == 0);
    return m;
}
template <typename R>
__device__ __forceinline__ void cm_apply(const Cm9<R>& m, int on, R& ax, R& ay, R& az) {
    if (!on) return;
    R a = ax, b = ay, c = az;
    ax = m.c[0] * a + m.c[1] * b + m.c[2] * c;
    ay = m.c[3] * a + m.c[4] * b + m.c[5] * c;
    az = m.c[6] * a + m.c[7] * b + m.c[8] * c;
}

// neighbour record bundles loaded by the list passes
template <typename R>
struct NbQ2 {
    PosRec<R> q;
    V2<R> a;
};
template <typename R>
struct NbQ2S {
    PosRec<R> q;
    V2<R> a;
    R s;
};
template <typename R>
struct NbQ44 {
    PosRec<R> q;
    V4<R> a, b;
};
template <typename R>
struct NbQ24 {
    PosRec<R> q;
    V2<R> a;
    V4<R> b;
};

// ---- the SPH neighbour list ---------------------------------------------
// Blocks of 8 entries per particle: entry k of particle i at
// ((k / 8) n + i) 8 + k % 8.  A particle's 8 consecutive entries fill one
// 32-byte sector: the list build's stores of one particle land in the same
// sector (written back whole from L2) and a walk loads B entries in one
// vector load, while the particles of a warp (consecutive i) still read
// consecutive sectors.
__host__ __device__ __forceinline__ size_t nb_at(int k, int n, int i) {
    return ((size_t)(k >> 3) * n + i) * 8 + (k & 7);
}

// ---- pair sums over position + volume records --------------------------------
// the volume word: +V for the types the Shepard sum takes, -V for the
// others, NaN for a particle of the slow path
template <typename R>
__device__ __forceinline__ R pv_code(R v, int tag, bool shepard) {
    if (!(v >= (R)0) || (tag & TAG_OOR) || tag_ptype(tag) >= 1000)
        return sizeof(R) == 4 ? (R)__int_as_float(0x7fffffff) : (R)__longlong_as_double(0x7fffffffffffffffll);
    return shepard ? v : -v;
}
__device__ __forceinline__ int4 pv_make(const int4& q, float v) { return make_int4(q.x, q.y, q.z, __float_as_int(v)); }
__device__ __forceinline__ Dbl4 pv_make(const QPos64& q, double v) { return Dbl4{q.x, q.y, q.z, v}; }
__device__ __forceinline__ float pv_vol(const int4& q) { return __int_as_float(q.w); }
__device__ __forceinline__ double pv_vol(const Dbl4& q) { return q.w; }
__device__ __forceinline__ void pv_set_vol(int4* p, int i, float v) { reinterpret_cast<float*>(p + i)[3] = v; }
__device__ __forceinline__ void pv_set_vol(Dbl4* p, int i, double v) { p[i].w = v; }
__device__ __forceinline__ Disp<float> pv_disp(const DevParams& P, const int4& a, const int4& b) {
    return Disp<float>{(float)(a.x - b.x) * P.q_step[0], (float)(a.y - b.y) * P.q_step[1],
                       (float)(a.z - b.z) * P.q_step[2]};
}
__device__ __forceinline__ Disp<double> pv_disp(const DevParams&, const Dbl4& a, const Dbl4& b) {
    return Disp<double>{a.x - b.x, a.y - b.y, a.z - b.z};
}
// displacement from the double positions and the plain volume of j; kept
// out of line, the loops hold registers for the common path only
template <typename R>
__device__ __noinline__ V4<R> pv_slow(const double* X, const double* Y, const double* Z, const R* m, const R* rho,
                                      int i, int j) {
    return mk4<R>((R)(X[i] - X[j]), (R)(Y[i] - Y[j]), (R)(Z[i] - Z[j]), m[j] / rho[j]);
}
// 1/|d| and |d| with |d|^2 floored (the self pair: d = 0, every term of it
// carries a component of d or a difference that is 0)
__device__ __forceinline__ float rsq_floor(float r2) {
    float s;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(fmaxf(r2, 1e-30f)));
    return s;
}
__device__ __forceinline__ double rsq_floor(double r2) { return rsqrt(fmax(r2, 1e-60)); }

// Wendland C2 without its constant factors, which leave the sums:
// dW/dr / r = gn (1-q)^3 with gn = -5 tA / h^2 and W = tA (1-q)^4 (1 + 4q),
// q = r / 2h: a pair needs no division by r.
template <typename R>
struct C2Sum {
    R hq, gn, wn;   // 1 / 2h, the factors of dW/dr / r and of W
};
template <typename R>
__device__ __forceinline__ C2Sum<R> c2_sum(const DevParams& P, R th) {
    const R ih = (R)1 / th, tA = knl_tmpA<R>(3, P.dim, th);
    return C2Sum<R>{(R)0.5 * ih, (R)-5 * ih * ih * tA, tA};
}
template <typename R>
__device__ __forceinline__ R c2_g(const C2Sum<R>& s, R r) {
    R a = (R)1 - r * s.hq;
    a = a > (R)0 ? a : (R)0;
    return a * a * a;
}
template <typename R>
__device__ __forceinline__ R c2_w(const C2Sum<R>& s, R r) {
    const R q = r * s.hq;
    R a = (R)1 - q;
    a = a > (R)0 ? a : (R)0;
    const R a2 = a * a;
    return a2 * a2 * ((R)1 + (R)4 * q);
}

// the gradient correction is the inverse of a symmetric moment matrix: six
// planes xx, xy, xz, yy, yz, zz (the identity when it is off)
template <typename R>
struct Cm6 {
    R xx, xy, xz, yy, yz, zz;
};
template <typename R>
__device__ __forceinline__ Cm6<R> cm6_load(const R* __restrict__ Cm, int n, int i, bool on) {
    if (!on) return Cm6<R>{1, 0, 0, 1, 0, 1};
    return Cm6<R>{Cm[i], Cm[(size_t)n + i], Cm[(size_t)2 * n + i], Cm[(size_t)3 * n + i], Cm[(size_t)4 * n + i],
                  Cm[(size_t)5 * n + i]};
}
template <typename R>
__device__ __forceinline__ Disp<R> cm6_mul(const Cm6<R>& c, R x, R y, R z) {
    return Disp<R>{c.xx * x + c.xy * y + c.xz * z, c.xy * x + c.yy * y + c.yz * z, c.xz * x + c.yz * y + c.zz * z};
}

// neighbour record bundles of the position + volume passes
template <typename R>
struct NbP {
    PvRec<R> q;
};
template <typename R>
struct NbPS {
    PvRec<R> q;
    R s;
};
template <typename R>
struct NbP4 {
    PvRec<R> q;
    V4<R> b;
};
template <typename R>
struct NbP4S {
    PvRec<R> q;
    V4<R> b;
    R s;
};
// ---- batched neighbour-list walk -------------------------------------------
// The list passes are bound by the latency of the dependent loads (list
// entry -> neighbour records) and by L1 wavefronts.  The entries of a batch
// of 4 come in one 16-byte load, requested two batches ahead, so their
// latency (the list streams from L2 or HBM) is hidden behind the arithmetic
// of the batches before.  The records of a batch are loaded before any of
// its arithmetic; prep turns each into its pair (displacement, volume), fix
// replaces those that a record does not give (rare; a branch per batch), and
// comp runs on the four pairs without branches between them.  The sums run
// in list order.  The last batch is padded with the particle itself at zero
// volume, which adds nothing.
__device__ __forceinline__ int4 nb_ld4(const int* p) {
    int4 v;
    asm volatile("ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
template <typename T, typename PV, typename L, typename P, typename X, typename C>
__device__ __forceinline__ void nb_sum(int cnt, const int* __restrict__ nb, int n, int i, L load, P prep, X fix,
                                       C comp) {
    if (cnt <= 0) return;
    const int* p = nb + (size_t)i * 8;   // entry k of particle i: nb_at(k, n, i)
    const size_t step = (size_t)n * 8;
    int4 e0 = nb_ld4(p), e1 = make_int4(i, i, i, i);
    if (cnt > 4) e1 = nb_ld4(p + 4);
    auto batch = [&](const int4& e, int m) {
        int j[4] = {e.x, e.y, e.z, e.w};
        T r[4];
        PV g[4];
        bool bad = false;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (m < 4 && u >= m) j[u] = i;
            r[u] = load(j[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) bad |= prep(r[u], g[u]);
        if (bad) {
#pragma unroll
            for (int u = 0; u < 4; u++) fix(j[u], r[u], g[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (m < 4 && u >= m) g[u].v = g[u].vs = 0;
            comp(j[u], r[u], g[u]);
        }
    };
    int k = 0;
#pragma unroll 1
    for (; k + 4 <= cnt; k += 4) {
        // entries k+8 .. k+11 lie one block of 8 further
        int4 e2 = e1;
        if (k + 8 < cnt) e2 = nb_ld4(p + (size_t)((k >> 3) + 1) * step + (k & 4));
        batch(e0, 4);
        e0 = e1;
        e1 = e2;
    }
    if (k < cnt) batch(e0, cnt - k);
}

// the same list in batches of 4 for the passes that keep per-pair control
// flow; entries requested one batch ahead
template <int B, typename T, typename L, typename C>
__device__ __forceinline__ void nb_walk(int cnt, const int* __restrict__ nb, int n, int i, L load, C comp) {
    static_assert(B == 4, "list walks load 4 entries at a time");
    if (cnt <= 0) return;
    int k = 0;
    int4 v = nb_ld4(nb + nb_at(0, n, i));
    for (; k + 4 <= cnt; k += 4) {
        const int j[4] = {v.x, v.y, v.z, v.w};
        if (k + 4 < cnt) v = nb_ld4(nb + nb_at(k + 4, n, i));
        T r[4];
#pragma unroll
        for (int u = 0; u < 4; u++) r[u] = load(j[u]);
#pragma unroll
        for (int u = 0; u < 4; u++) comp(j[u], r[u]);
    }
    for (; k < cnt; k++) {
        const T r = load(v.x);
        comp(v.x, r);
        v.x = v.y;
        v.y = v.z;
    }
}

// ---- several lanes per particle, sums in list order -------------------------
// A set of a few thousand particles leaves a scheduler less than a warp, and a
// pass then lasts one thread's walk.  L lanes share a particle: each forms the
// terms of one entry (the operands of the sums' FMAs), then all add them in
// list order, so every lane holds the bits that one thread's walk gives.
template <int L>
struct LaneGroup {
    int i, lane;
    unsigned mask, base;
    __device__ __forceinline__ LaneGroup() {
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        i = t / L;
        lane = t % L;
        base = (threadIdx.x & 31) & ~(L - 1);
        mask = (L == 32 ? 0xffffffffu : (1u << L) - 1u) << base;
    }
};
template <int L, typename T>
__device__ __forceinline__ T shfl_terms(unsigned mask, const T& t, int l) {
    static_assert(sizeof(T) % 4 == 0, "terms are 32- or 64-bit values");
    constexpr int N = sizeof(T) / 4;
    T o;
    const int* a = reinterpret_cast<const int*>(&t);
    int* b = reinterpret_cast<int*>(&o);
#pragma unroll
    for (int q = 0; q < N; q++) b[q] = __shfl_sync(mask, a[q], l, L);
    return o;
}
// entry(k): list entry k; load(j): its record; terms(j, r, t): false when the
// pair adds nothing; add(t)
template <int L, typename Rec, typename T, typename E, typename LD, typename TM, typename AD>
__device__ __forceinline__ void ordered_walk(const LaneGroup<L>& g, int cnt, E entry, LD load, TM terms, AD add) {
    int j = g.lane < cnt ? entry(g.lane) : 0;
    for (int k0 = 0; k0 < cnt; k0 += L) {
        const int k = k0 + g.lane, jc = j;
        T t{};
        bool ok = false;
        if (k < cnt) {
            const Rec r = load(jc);
            if (k + L < cnt) j = entry(k + L);
            ok = terms(jc, r, t);
        }
        const unsigned m = (__ballot_sync(g.mask, ok) & g.mask) >> g.base;
#pragma unroll
        for (int l = 0; l < L; l++)
            if ((m >> l) & 1u) add(shfl_terms<L, T>(g.mask, t, l));
    }
}

}  // namespace sphdem
