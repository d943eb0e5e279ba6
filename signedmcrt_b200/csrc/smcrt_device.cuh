// smcrt_device.cuh -- device building blocks of the B200 photon-packet transport.
//
// Everything here is templated on the transport precision R (float or double);
// boundary events (normal + Fresnel + reflect/refract) always run in double.
// Reference formulas are cited by file:line of the signedMCRT sources.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "../../include/smcrt.h"

namespace smcrt {

// Scenes up to kMaxRegions regions and kMaxPrims primitives travel in the
// launch's parameter block (constant bank: warp-broadcast operands); larger
// scenes, up to kMaxRegionsDev regions, live in device memory (SceneG).
constexpr int kMaxPrims = 32;
constexpr int kMaxRegions = 16;
constexpr int kMaxRegionsDev = 255;
constexpr int kMaxPrimsDev = 4096;
constexpr int kMaxDetectors = 16;
// Detector bins privatized per CTA as 32-bit counts in shared memory (16 KiB);
// larger bin sets (camera images) add straight into the global FP64 bins.
constexpr int kMaxSharedBins = 4096;
constexpr int kMaxTallyCopies = 16;
constexpr int kMaxAdjGroups = 5;  // parameter groups of one adjoint launch (3 parameters each)
constexpr double kPI = 3.14159265358979323846264338327950288;

// Device status flags (smcrt_stats.device_status).
enum : int { STATUS_STEP_CAP = 1, STATUS_ERROR_STATE = 2, STATUS_STREAM_EXHAUSTED = 4, STATUS_BAD_INDEX = 8, STATUS_ABORTED = 16 };

// ---------------------------------------------------------------------------
template <class R>
struct V3 {
    R x, y, z;
};
template <class R> __host__ __device__ __forceinline__ V3<R> operator+(V3<R> a, V3<R> b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class R> __host__ __device__ __forceinline__ V3<R> operator-(V3<R> a, V3<R> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class R> __host__ __device__ __forceinline__ V3<R> operator*(V3<R> a, R s) { return {a.x * s, a.y * s, a.z * s}; }
template <class R> __host__ __device__ __forceinline__ V3<R> operator*(R s, V3<R> a) { return {s * a.x, s * a.y, s * a.z}; }
template <class R> __device__ __forceinline__ R dot3(V3<R> a, V3<R> b) { return (a.x * b.x) + (a.y * b.y) + (a.z * b.z); }
template <class R> __device__ __forceinline__ R len3(V3<R> a) { return sqrt(a.x * a.x + a.y * a.y + a.z * a.z); }
// Larger and smaller of x and a number c; a NaN x gives c, as fmax and fmin do.  In
// FP64 a compare and a select: fmax and fmin on doubles, which also look for a NaN
// c, are several instructions more.
__device__ __forceinline__ float max_r(float x, float c) { return fmaxf(x, c); }
__device__ __forceinline__ float min_r(float x, float c) { return fminf(x, c); }
__device__ __forceinline__ double max_r(double x, double c) { return x > c ? x : c; }
__device__ __forceinline__ double min_r(double x, double c) { return x < c ? x : c; }
template <class R> __device__ __forceinline__ R clampr(R x, R lo, R hi) { return fmin(fmax(x, lo), hi); }
template <class R> __device__ __forceinline__ R fsign(R a, R b) { return copysign(fabs(a), b); }  // Fortran sign(a,b)
__device__ __forceinline__ void sincos_r(float x, float* s, float* c) { sincosf(x, s, c); }
__device__ __forceinline__ void sincos_r(double x, double* s, double* c) { sincos(x, s, c); }
__device__ __forceinline__ float cospi_r(float x) { return cospif(x); }
__device__ __forceinline__ double cospi_r(double x) { return cospi(x); }

// ---------------------------------------------------------------------------
// Scene tables (kernel-parameter resident: constant bank, warp-broadcast reads).
template <class R>
struct DPrim {
    R m[12];  // row-vector affine, m[3*i+j] = M[i][j]
    R q[8];
    int kind;
    int nmods;   // modifiers, innermost first
    int mod[2];
    R mp[2][3];
};
//
// Most regions are one box, sphere or capsule without modifiers whose transform
// only translates; `shape` names them (RegionShape), so that their value costs
// three adds instead of the affine map's nine multiply-adds and no walk through
// the primitive, modifier and fold switches.  With a rotation part of exactly 1
// and 0 the affine map's products are exact and its sums add zeros, so both forms
// give the same bits (the sign of a zero aside, which no distance depends on).
// The sweeps are bound by instruction issue, so this is worth as much as it saves:
// with the sweep's outputs cut to those a step uses, sphere_water 103.3 -> 88.7 ms
// (4e6 packets), layered_vessels 117.0 -> 83.2 ms (2e6), the FP64 render of 256^3
// voxels 795 -> 521 us.
enum RegionShape : int { SHAPE_GENERIC = 0, SHAPE_BOX, SHAPE_SPHERE, SHAPE_CAPSULE };
template <class R>
struct DRegion {
    int first, n, op, shape;
    R t[3], q[7];  // a plain shape's translation and parameters
    R k, kappa, albedo, hgg, g2, nidx;
    R mus, mua;  // for the adjoint's scatter/absorption terms
};

// Optical properties of one batch instance, per region (the per-region fields of
// DRegion; the geometry is shared by all instances of a batch).
template <class R>
struct InstOptics {
    R kappa[kMaxRegions], albedo[kMaxRegions], hgg[kMaxRegions], g2[kMaxRegions], nidx[kMaxRegions];
    double nidx64[kMaxRegions];
};

template <class R>
struct SceneT {
    int nregions, nprims;
    int has_mods, pad;  // some primitive carries modifiers
    DPrim<R> prim[kMaxPrims];
    DRegion<R> region[kMaxRegions];
};

// A scene in device memory (the same tables behind pointers, read through the
// L1 cache with warp-uniform addresses), with a bounding sphere per region:
// bound[4 r .. 4 r + 3] = world centre and radius, radius < 0 when the region
// has none (see sweep_regions).  cull_margin covers the rounding of the test.
template <class R>
struct SceneG {
    int nregions, nprims;
    int has_mods, pad;
    const DPrim<R>* prim;
    const DRegion<R>* region;
    const R* bound;
    R cull_margin;
};

// The sums of products below say which product is fused with which add (mad), and
// leave the compiler no other pair to contract.  A region's value is formed in several
// places of a kernel (sweeps over all regions and over the kept ones, FP32 and
// FP64, crossings), each an inlined copy of this code: a copy contracted in another way
// would round in another way, and histories would depend on which sweep took a step.
// SMCRT_FMAD 0 (the units built with --fmad=false): separate roundings, as the CPU
// restatement.
#ifndef SMCRT_FMAD
#define SMCRT_FMAD 1
#endif
__device__ __forceinline__ float mad(float a, float b, float c) { return SMCRT_FMAD ? __fmaf_rn(a, b, c) : a * b + c; }
__device__ __forceinline__ double mad(double a, double b, double c) { return SMCRT_FMAD ? __fma_rn(a, b, c) : a * b + c; }
// a + b of products formed before, each rounded
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
// a b + c d + e f, and its case of squares
template <class R>
__device__ __forceinline__ R mad3(R a, R b, R c, R d, R e, R f) {
    return mad(e, f, mad(a, b, c * d));
}
template <class R>
__device__ __forceinline__ R dot_m(V3<R> a, V3<R> b) {
    return mad3(a.x, b.x, a.y, b.y, a.z, b.z);
}
template <class R>
__device__ __forceinline__ R len_m(V3<R> a) {
    return sqrt(dot_m(a, a));
}

// pos .dot. transform, src/vector_class.f90:292-304
template <class R>
__device__ __forceinline__ V3<R> xform(const R* m, V3<R> a) {
    V3<R> d;
    d.x = mad3(m[0], a.x, m[3], a.y, m[6], a.z) + m[9];
    d.y = mad3(m[1], a.x, m[4], a.y, m[7], a.z) + m[10];
    d.z = mad3(m[2], a.x, m[5], a.y, m[8], a.z) + m[11];
    return d;
}

// The capsule at a point in its own coordinates (src/sdfs/sdfs.f90:628-648).
template <class R>
__device__ __forceinline__ R capsule_at(const R* q, V3<R> p, R r) {
    V3<R> a{q[0], q[1], q[2]}, b{q[3], q[4], q[5]};
    V3<R> pa = p - a, ba = b - a;
    R h = clampr(dot_m(pa, ba) / dot_m(ba, ba), (R)0, (R)1);
    return len_m(V3<R>{mad(-ba.x, h, pa.x), mad(-ba.y, h, pa.y), mad(-ba.z, h, pa.z)}) - r;
}

// Primitive SDFs, src/sdfs/sdfs.f90:494-735
template <class R>
__device__ __forceinline__ R eval_prim_base(const DPrim<R>& pr, V3<R> pos) {
    const V3<R> p = xform(pr.m, pos);
    const R* q = pr.q;
    const R zero = 0, one = 1, half = (R)0.5;
    switch (pr.kind) {
        case SMCRT_SPHERE:
            return len_m(p) - q[0];
        case SMCRT_BOX: {
            R dx = fabs(p.x) - q[0], dy = fabs(p.y) - q[1], dz = fabs(p.z) - q[2];
            R mx = fmax(dx, zero), my = fmax(dy, zero), mz = fmax(dz, zero);
            return len_m(V3<R>{mx, my, mz}) + fmin(fmax(dx, fmax(dy, dz)), zero);
        }
        case SMCRT_TORUS: {
            R tx = sqrt(mad(p.z, p.z, p.x * p.x)) - q[0];
            return sqrt(mad(p.y, p.y, tx * tx)) - q[1];
        }
        case SMCRT_CYLINDER: {
            V3<R> a{q[0], q[1], q[2]}, b{q[3], q[4], q[5]};
            V3<R> ba = b - a, pa = p - a;
            R baba = dot_m(ba, ba), paba = dot_m(pa, ba);
            V3<R> c{mad(pa.x, baba, -(ba.x * paba)), mad(pa.y, baba, -(ba.y * paba)), mad(pa.z, baba, -(ba.z * paba))};
            R x = mad(-q[6], baba, len_m(c));
            R y = mad(-baba, half, fabs(mad(-baba, half, paba)));
            R x2 = x * x, y2 = (y * y) * baba, d;
            if (fmax(x, y) < zero) {
                d = -fmin(x2, y2);
            } else {
                if (x > zero && y > zero) d = add(x2, y2);
                else if (x > zero) d = x2;
                else if (y > zero) d = y2;
                else d = zero;
            }
            return fsign(sqrt(fabs(d)) / baba, d);
        }
        case SMCRT_TRIPRISM: {
            return fmax(fabs(p.z) - q[1], mad(-q[0], half, fmax(mad(fabs(p.x), (R)0.866025, p.y * half), -p.y)));
        }
        case SMCRT_SEGMENT:
        case SMCRT_CAPSULE:
            return capsule_at(q, p, (pr.kind == SMCRT_SEGMENT) ? (R)0.1 : q[6]);
        case SMCRT_CONE: {
            V3<R> a{q[0], q[1], q[2]}, b{q[3], q[4], q[5]};
            R ra = q[6], rb = q[7];
            R rba = rb - ra;
            R baba = dot_m(b - a, b - a);
            R papa = dot_m(p - a, p - a);
            R paba = dot_m(p - a, b - a) / baba;
            R x = sqrt(fmax(mad(-(baba * paba), paba, papa), zero));
            R cax = (paba < half) ? fmax(zero, x - ra) : fmax(zero, x - rb);
            R cay = fabs(paba - half) - half;
            R k = mad(rba, rba, baba);
            R f = clampr(mad(rba, x - ra, paba * baba) / k, zero, one);
            R cbx = mad(-f, rba, x - ra);
            R cby = paba - f;
            R s = (cbx < zero && cay < zero) ? -one : one;
            return s * sqrt(fmin(mad(cax, cax, baba * cay * cay), mad(cbx, cbx, baba * cby * cby)));
        }
        case SMCRT_EGG: {
            V3<R> pin{fabs(p.x), p.y, p.z};
            R r = q[0] - q[1];
            R hin = q[2] + r;
            R l = mad(hin, hin, -(r * r)) / ((R)2 * r);
            if (pin.y <= zero) return len_m(pin) - q[0];
            if ((pin.y - hin) * l > pin.x * hin)
                return len_m(V3<R>{pin.x, pin.y - hin, pin.z}) - ((q[0] + l) - sqrt(mad(hin, hin, l * l)));
            return len_m(V3<R>{pin.y, pin.x + l, pin.z}) - (q[0] + l);
        }
        case SMCRT_PLANE:
            return mad3(p.x, q[0], p.y, q[1], p.z, q[2]);
    }
    return zero;
}

// Modifiers (src/sdfs/sdfModifiers.f90:273-375): the point the wrapped SDF is
// evaluated at, and the value the modifier returns from the wrapped SDF's value.
template <class R>
__device__ __forceinline__ V3<R> mod_point(int kind, const R* q, V3<R> p) {
    const R zero = 0;
    switch (kind) {
        case SMCRT_MOD_REVOLUTION:  // (|(x, z)| - o, y, 0)
            return V3<R>{sqrt(mad(p.x, p.x, p.z * p.z)) - q[0], p.y, zero};
        case SMCRT_MOD_ELONGATE:  // max(|p| - size, 0)
            return V3<R>{fmax(fabs(p.x) - q[0], zero), fmax(fabs(p.y) - q[1], zero), fmax(fabs(p.z) - q[2], zero)};
        case SMCRT_MOD_TWIST: {  // rotation by k z about z
            R s, c;
            sincos_r(q[0] * p.z, &s, &c);
            return V3<R>{mad(c, p.x, -(s * p.y)), mad(s, p.x, c * p.y), p.z};
        }
        case SMCRT_MOD_BEND: {  // rotation by k x about z
            R s, c;
            sincos_r(q[0] * p.x, &s, &c);
            return V3<R>{mad(c, p.x, -(s * p.y)), mad(s, p.x, c * p.y), p.z};
        }
        default:  // onion, extrude: the wrapped SDF sees the point itself
            return p;
    }
}
template <class R>
__device__ __forceinline__ R mod_value(int kind, const R* q, R d, V3<R> p) {
    const R zero = 0;
    switch (kind) {
        case SMCRT_MOD_ONION:
            return fabs(d) - q[0];
        case SMCRT_MOD_EXTRUDE: {  // w = (d, |z| - h, 0)
            const R wy = fabs(p.z) - q[0];
            const R mx = fmax(d, zero), my = fmax(wy, zero);
            return fmin(fmax(d, wy), zero) + sqrt(mad(mx, mx, my * my));
        }
        case SMCRT_MOD_ELONGATE: {
            const R qx = fabs(p.x) - q[0], qy = fabs(p.y) - q[1], qz = fabs(p.z) - q[2];
            return d + fmin(fmax(qx, fmax(qy, qz)), zero);
        }
        default:
            return d;
    }
}

// A primitive with its modifiers: points map outermost modifier first, values
// innermost first, as the nested evaluate calls of the reference do.  MODS =
// false compiles the primitive alone, for scenes without modifiers.
template <class R, bool MODS = true>
__device__ __forceinline__ R eval_prim(const DPrim<R>& pr, V3<R> pos) {
    if (!MODS || pr.nmods == 0) return eval_prim_base(pr, pos);
    const V3<R> p1 = pr.nmods == 2 ? mod_point(pr.mod[1], pr.mp[1], pos) : pos;
    const V3<R> p2 = mod_point(pr.mod[0], pr.mp[0], p1);
    R d = mod_value(pr.mod[0], pr.mp[0], eval_prim_base(pr, p2), p1);
    if (pr.nmods == 2) d = mod_value(pr.mod[1], pr.mp[1], d, pos);
    return d;
}

// A region of a plain shape (RegionShape).
template <class R>
__device__ __forceinline__ R eval_shape(const DRegion<R>& g, V3<R> pos) {
    const V3<R> p{pos.x + g.t[0], pos.y + g.t[1], pos.z + g.t[2]};
    const R* q = g.q;
    if (g.shape == SHAPE_BOX) {
        const R dx = fabs(p.x) - q[0], dy = fabs(p.y) - q[1], dz = fabs(p.z) - q[2];
        const R m = max_r(dx, max_r(dy, dz));
        if (m <= (R)0) return m;  // inside: the outer length is 0
        const R mx = max_r(dx, (R)0), my = max_r(dy, (R)0), mz = max_r(dz, (R)0);
        return len_m(V3<R>{mx, my, mz});
    }
    if (g.shape == SHAPE_SPHERE) return len_m(p) - q[0];
    return capsule_at(q, p, q[6]);
}

// eval_model (src/sdfs/sdf_base.f90:145-160), CSG ops src/sdfs/sdfModifiers.f90:412-475:
// any region.  S: SceneT (parameter block) or SceneG (device memory).
template <class R, bool MODS, class S>
__device__ __forceinline__ R eval_model(const S& sc, int r, V3<R> pos) {
    const DRegion<R>& g = sc.region[r];
    R d = eval_prim<R, MODS>(sc.prim[g.first], pos);
    for (int i = 1; i < g.n; ++i) {
        R d2 = eval_prim<R, MODS>(sc.prim[g.first + i], pos);
        switch (g.op) {
            case SMCRT_OP_UNION: d = fmin(d, d2); break;
            case SMCRT_OP_SMOOTH_UNION: {
                R h = fmax(g.k - fabs(d - d2), (R)0) / g.k;
                d = mad(-(h * h * h * g.k), (R)1 / (R)6, fmin(d, d2));
                break;
            }
            case SMCRT_OP_SUBTRACTION: d = fmax(-d, d2); break;
            case SMCRT_OP_INTERSECTION: d = fmax(d, d2); break;
        }
    }
    return d;
}


template <class R, bool MODS = true, class S = SceneT<R>>
__device__ __forceinline__ R eval_region(const S& sc, int r, V3<R> pos) {
    const DRegion<R>& g = sc.region[r];
    if (g.shape != SHAPE_GENERIC) return eval_shape(g, pos);
    return eval_model<R, MODS, S>(sc, r, pos);
}

// calcNormal, src/sdfs/sdf_base.f90:165-189 (always double)
template <bool MODS = true, class S = SceneT<double>>
__device__ __forceinline__ V3<double> calc_normal(const S& sc, int r, V3<double> p, double h) {
    // the four directions (1,-1,-1), (-1,-1,1), (-1,1,-1), (1,1,1), in one loop: one
    // copy of the region's code
    V3<double> n{0, 0, 0};
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const V3<double> e{i == 0 || i == 3 ? 1.0 : -1.0, i >= 2 ? 1.0 : -1.0, i & 1 ? 1.0 : -1.0};
        const V3<double> v = e * eval_region<double, MODS, S>(sc, r, p + e * h);
        n = i == 0 ? v : n + v;
    }
    double t = len3(n);
    return V3<double>{n.x / t, n.y / t, n.z / t};
}

// fresnel / reflect / refract, src/surfaces.f90:42-120
template <class R>
__device__ __forceinline__ R fresnel(V3<R> I, V3<R> N, R n1, R n2) {
    R costt = fabs(dot3(I, N));
    R sintt = sqrt((R)1 - costt * costt);
    R sint2 = n1 / n2 * sintt;
    if (sint2 > (R)1) return (R)1;
    if (costt == (R)1) return (R)0;
    R cost2 = sqrt((R)1 - sint2 * sint2);
    R f1 = fabs((n1 * costt - n2 * cost2) / (n1 * costt + n2 * cost2));
    R f2 = fabs((n1 * cost2 - n2 * costt) / (n1 * cost2 + n2 * costt));
    return (R)0.5 * (f1 * f1 + f2 * f2);
}
template <class R>
__device__ __forceinline__ V3<R> reflect(V3<R> I, V3<R> N) {
    return I - (R)2 * dot3(N, I) * N;
}
template <class R>
__device__ __forceinline__ V3<R> refract(V3<R> I, V3<R> N, R eta) {
    V3<R> Nt = N;
    R c1 = dot3(Nt, I);
    if (c1 < (R)0) c1 = -c1;
    else Nt = (R)(-1) * N;
    R c2 = sqrt((R)1 - (eta * eta) * ((R)1 - c1 * c1));
    return eta * I + (eta * c1 - c2) * Nt;
}

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11).
__host__ __device__ __forceinline__ void philox4x32_10(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                                       uint32_t c3, uint32_t out[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
#ifdef __CUDA_ARCH__
        uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
#else
        uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
        uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0, hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
#endif
        uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    out[0] = c0;
    out[1] = c1;
    out[2] = c2;
    out[3] = c3;
}

template <class R> struct U01;
template <> struct U01<float> {
    static constexpr int kWords = 1;
    __device__ __forceinline__ static float from(uint32_t a, uint32_t) { return (float)(a >> 9) * 0x1p-23f + 0x1p-24f; }
};
template <> struct U01<double> {
    static constexpr int kWords = 2;
    __device__ __forceinline__ static double from(uint32_t a, uint32_t b) {
        uint64_t m = ((uint64_t)a << 20) | (uint64_t)(b >> 12);
        return (double)m * 0x1p-52 + 0x1p-53;
    }
};

// One Philox block (out of line unless SMCRT_PHILOX_INLINE: one copy of the 10
// rounds per kernel, at the cost of a call per four draws).
#ifdef SMCRT_PHILOX_INLINE
static __device__ __forceinline__ uint4 philox_block(
#else
static __device__ __noinline__ uint4 philox_block(
#endif
    uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1, uint32_t c2,
                                                 uint32_t c3) {
    uint32_t o[4];
    philox4x32_10(k0, k1, c0, c1, c2, c3, o);
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Per-packet uniform stream: counter RNG keyed (seed, instance, packet id); in
// replay builds (INJ) an injected uniform stream instead.  The key words live in
// the caller's constant bank (seed, instance) and are passed at each refill.  A
// stream is its position alone: between passes no words are kept, and the block
// that holds the position is made again at the next draw.
template <class R, bool INJ = false>
struct Stream {
    uint32_t p0, p1;
    uint32_t pos;  // Philox words consumed (INJ: uniforms consumed)
    uint32_t b0, b1, b2, b3;  // unconsumed words of the current block, consumed from b0
    int left;
    const double* inj;
    int ninj;
    int flags;
    unsigned long long seed;
    uint32_t inst;

    __device__ __forceinline__ void init(uint64_t seed_, uint32_t instance, uint64_t pid, const double* injected,
                                         int n) {
        seed = seed_;
        inst = instance;
        p0 = (uint32_t)pid;
        p1 = (uint32_t)(pid >> 32);
        pos = 0;
        left = 0;
        inj = injected;
        ninj = n;
        flags = 0;
    }
    __device__ __forceinline__ int ndraws() const { return INJ ? (int)pos : (int)(pos / U01<R>::kWords); }
    __device__ __forceinline__ R next() {
        if (INJ) {
            if ((int)pos >= ninj) {
                flags |= STATUS_STREAM_EXHAUSTED;
                ++pos;
                return (R)0.5;
            }
            return (R)inj[pos++];
        }
        if (left < U01<R>::kWords) {
            const uint4 o = philox_block((uint32_t)seed, (uint32_t)(seed >> 32), pos >> 2, inst, p0, p1);
            const bool two = pos & 2u, one = pos & 1u;
            b0 = two ? o.z : o.x;
            b1 = two ? o.w : o.y;
            b2 = o.z;
            b3 = o.w;
            if (U01<R>::kWords == 1 && one) {
                b0 = b1;
                b1 = b2;
                b2 = b3;
            }
            left = 4 - (int)(pos & 3u);
        }
        R u;
        if (U01<R>::kWords == 1) {
            u = U01<R>::from(b0, 0u);
            b0 = b1;
            b1 = b2;
            b2 = b3;
        } else {
            u = U01<R>::from(b0, b1);
            b0 = b2;
            b1 = b3;
        }
        left -= U01<R>::kWords;
        pos += U01<R>::kWords;
        return u;
    }
};

// Five FP32 draws of a Philox stream at once: those of one interaction (albedo,
// bias, angle, azimuth or roulette, next optical depth).  Two blocks cover them
// wherever the position lies, so the lanes of a warp make both together; drawing
// one by one, each draw refills some of the lanes, and the warp pays for up to
// five blocks.  The words are the stream's; done() moves its position past those taken.
struct Draw5 {
    uint32_t r[5];
    uint32_t used;
    __device__ __forceinline__ void fill(const Stream<float, false>& s) {
        uint32_t a[8];
        const uint32_t k0 = (uint32_t)s.seed, k1 = (uint32_t)(s.seed >> 32), c = s.pos >> 2;
        philox4x32_10(k0, k1, c, s.inst, s.p0, s.p1, a);
        philox4x32_10(k0, k1, c + 1u, s.inst, s.p0, s.p1, a + 4);
        if (s.pos & 2u) {
#pragma unroll
            for (int i = 0; i < 6; ++i) a[i] = a[i + 2];
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) r[i] = s.pos & 1u ? a[i + 1] : a[i];
        used = 0;
    }
    __device__ __forceinline__ float next() {
        const float u = U01<float>::from(r[0], 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = r[i + 1];
        ++used;
        return u;
    }
    __device__ __forceinline__ void done(Stream<float, false>& s) {
        s.pos += used;
        s.left = 0;
    }
};

// scatter, src/photon.f90:713-779 (the bias test with p = 0 consumes one draw
// when g != 0).  FP64 uses the reference's formulas; FP32 evaluates the same
// angles in forms free of the 1 - cos^2 cancellations: 1 -+ cos(theta) come
// factored out of the HG inverse CDF, and sin/cos(phi) from sincospi, so the
// FP32 direction is accurate to a few ulps even for near-forward scatters.
__device__ __forceinline__ void hg_angles(float hgg, float g2, float u, float& cost, float& sint) {
    float omc, opc;  // 1 - cos(theta), 1 + cos(theta)
    if (hgg == 0.0f) {
        omc = 2.0f * (1.0f - u);
        opc = 2.0f * u;
    } else {
        const float den = 1.0f - hgg + 2.0f * hgg * u;
        const float temp = (1.0f - g2) / den;
        omc = (1.0f - hgg) * (1.0f - u) * (temp + (1.0f - hgg)) / den;
        opc = (1.0f + hgg) * u * (1.0f + hgg + temp) / den;
    }
    cost = (omc < opc) ? 1.0f - omc : opc - 1.0f;
    sint = sqrtf(omc * opc);
}
__device__ __forceinline__ void hg_angles(double hgg, double g2, double u, double& cost, double& sint) {
    if (hgg == 0.0) {
        cost = 2.0 * u - 1.0;
    } else {
        const double temp = (1.0 - g2) / (1.0 - hgg + 2.0 * hgg * u);
        cost = (1.0 + g2 - temp * temp) / (2.0 * hgg);
    }
    sint = sqrt(1.0 - cost * cost);
}
__device__ __forceinline__ void phi_angles(float u, float& cosp, float& sinp) { sincospif(2.0f * u, &sinp, &cosp); }
__device__ __forceinline__ void phi_angles(double u, double& cosp, double& sinp) {
    cosp = cospi(2.0 * u);
    const double s = sqrt(1.0 - cosp * cosp);
    sinp = (u < 0.5) ? s : -s;  // phi = 2 pi u < pi  <=>  u < 1/2
}

// mu_out: the sampled cos(theta) (the HG variate, before the vertical-case sign
// rule), for the adjoint's d log p_HG / dg.
template <class R, class Rng>
__device__ __forceinline__ V3<R> hg_scatter(V3<R> d, R hgg, R g2, Rng& rng, R* mu_out = nullptr) {
    const R one = 1;
    R cost, sint;
    if (hgg == (R)0) {
        hg_angles(hgg, g2, rng.next(), cost, sint);
    } else {
        (void)rng.next();
        hg_angles(hgg, g2, rng.next(), cost, sint);
    }
    if (mu_out) *mu_out = cost;
    R cosp, sinp;
    phi_angles(rng.next(), cosp, sinp);
    bool vertical = (one - fabs(d.z) <= (R)1e-12);
    R temp = 0;
    if (!vertical) {
        temp = (sizeof(R) == 4) ? sqrt(d.x * d.x + d.y * d.y) : sqrt(one - d.z * d.z);
        if (temp == (R)0) vertical = true;
    }
    V3<R> o;
    if (vertical) {
        o.x = sint * cosp;
        o.y = sint * sinp;
        o.z = fsign(cost, d.z);
    } else {
        o.x = sint * (d.x * d.z * cosp - d.y * sinp) / temp + d.x * cost;
        o.y = sint * (d.y * d.z * cosp + d.x * sinp) / temp + d.y * cost;
        o.z = -one * sint * cosp * temp + d.z * cost;
    }
    return o;
}

// ---------------------------------------------------------------------------
// Grid and detectors.
template <class R>
struct GridT {
    int nx, ny, nz, pad;
    R xmax, ymax, zmax;
    R inset;            // 2^-31 of the largest half size: crawls end this far before a voxel face
    R vx, vy, vz;       // voxel sizes 2*max/n
    R sx, sy, sz;       // n/(2*max) as written: n * p / (2 * max)
    double xmax_d, ymax_d, zmax_d;  // exact half sizes (grid-exit test on FP64 positions)
    double sx_d, sy_d, sz_d;        // n / (2 max) in FP64 (FP32 transport's cell index of an FP64 position)
    double vx_d, vy_d, vz_d;        // voxel sizes 2 max / n in FP64 (the walk's face positions)
};

struct DetT {
    int kind, layer, nb, pad;  // nb = bins per axis (nbins + 1)
    long long off;
    double pos[3], dir[3];
    double r1, r2, bw, bwy;
    double e1[3], e2[3], n[3], width, height;
};

template <class R>
struct SourceT {
    int kind, annulus_type;
    R pos[3], dir[3], p1[3], p2[3], p3[3];
    R radius, radius_hi, sin_beta, cos_beta, zstart;
    R rot[9];  // circular source rotation (rotationAlign), row-major M[i][j]
    int circ_swap;
};

// Launch parameters (one __grid_constant__ block in the constant bank).
template <class R>
struct Params {
    SceneT<R> sc;
    SceneT<double> sc64;  // boundary events
    // scenes beyond the parameter block (the BIG kernel instantiation): device tables
    SceneG<R> gsc;
    SceneG<double> gsc64;
    GridT<R> grid;
    SourceT<R> src;
    DetT det[kMaxDetectors];
    int ndet;
    int kernel;
    int end_early;
    int max_steps;
    R eps;
    R near_band;  // FP32 transport: sweeps closer than this to a surface are taken in FP64
    // nearest-region cache: allowed (every region 1-Lipschitz) and the rounding
    // margin of its test (FP32 transport: the FP32 sweeps' margin for both sweeps)
    int cache_ok;
    float cache_margin;  // rounded up
    // sort group of each action, one nibble per action (the round's list order)
    unsigned long long group_order;
    // shared-memory fluence privatisation (FP32 plain launches): a sub-box of
    // voxels (0-based origin, extents; priv_n cells, 0 = off) whose segments each
    // CTA sums in shared memory as 64-bit fixed point and adds to the grid once
    int priv_n;
    int priv_o[3], priv_d[3];
    double normal_h;
    unsigned long long seed;
    unsigned long long budget_ns;  // per-launch device time budget (0 = none)
    unsigned int instance;
    long long first;
    long long count;
    int sbins;    // detector bins counted in shared memory (0: global atomics)
    int tcopies;                     // fluence-grid copies the CTAs spread their adds over
    unsigned tmask;                  // tcopies - 1 (tcopies is a power of two)
    long long ncell;
    double* jtab[kMaxTallyCopies];   // the grid of each copy; jtab[0] is the output grid
    // batch launches: instance i has packets [bprefix[i], bprefix[i+1]) of the
    // launch, seed bseed[i], optics bopt[i], tally jtab[0] + i * ncell and
    // detector bins + i * nbins; per-instance packets/draws/scatters in bstats
    const InstOptics<R>* bopt;
    const long long* bprefix;
    const unsigned long long* bseed;
    unsigned long long* bstats;  // [ninst][3]
    int ninst;
    long long nbins;
    // adjoint launches: d loss / d (per-packet fluence) per voxel, d loss / d
    // (per-packet detector counts) per bin, the parameter group of each region
    // (255: none) and the output sums [3][ngroups] (d/d mua, d/d mus, d/d g)
    const float* adj_w;
    const double* adj_gbins;
    double* adj_out;
    int adj_ngroups;
    unsigned char adj_group[kMaxRegions];
    // second-moment runs (the VAR instantiation): each packet slot's voxel-score
    // table (kVarSlotBytes each: (voxel, score) pairs, the used list and its
    // count; slot-major over the persistent grid's CTAs) and the per-voxel sum of
    // squared per-packet scores
    unsigned char* var_tab;
    double* jmean2;
};

}  // namespace smcrt
