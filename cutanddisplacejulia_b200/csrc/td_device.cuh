// Device-side triangular dislocation (TD) evaluation for one (observation,
// triangle) pair: full-space strain / displacement, the half-space free-surface
// correction and the image dislocation.
//
// Semantics follow the reference's per-point arithmetic in src/TD.jl:
//   frame + TDCS coordinates       CalculateLocalTriCoords! :712-732, GlobalToTDECoords :870-908
//   interior angles, side vectors  CalcTDVectsAndAngles :962-1008
//   points on a side               trimodefinder :1010-1079
//   full-space strain / disp       TDstrainFS :1499-1620, TDdispFS :735-867 (the reference sums
//                                  three angular dislocations; here the same closed loop is
//                                  summed as three straight segments, see seg_integrals)
//   free-surface correction        AngSetupStrainFSC :1867-2081, AngSetupDispFSC :1258-1409
//   image dislocation              ComputeStrainInfluences :670-708, ComputeDispInfluences :631-668
// The free-surface rows come from fsc_rows.cuh (generated by gen/gen_fsc.py).
//
// Data layout: everything that depends only on the triangle (frames, angles,
// per-dislocation constants of every closed-form term, slip rotations) is
// computed once per triangle by td_setup_kernel into a TriDev record; the pair
// kernels stage records in shared memory (one, or eight of the small ones, at a
// time) and every thread of the block (one observation point each) reads each as
// a broadcast.
#pragma once
#include <cfloat>
#include <cstddef>
#include <cstdint>

#include <math.h>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define CAD_HD __host__ __device__ __forceinline__
#else
#define CAD_HD inline
#endif

namespace cad {

#ifndef __CUDACC__
// plain C++ build of the device code (used only to test it on a CPU)
inline double rsqrt(double x) { return 1.0 / sqrt(x); }
inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
#endif

// math functions in the pair bodies' arithmetic type
CAD_HD double cad_rsqrt(double x) { return rsqrt(x); }
CAD_HD float cad_rsqrt(float x) { return rsqrtf(x); }
CAD_HD double cad_log(double x) { return log(x); }
CAD_HD float cad_log(float x) { return logf(x); }

// Accumulators of the free-surface correction, end B minus end A (fsc_end and
// fsc_disp_end fill them; fsc_rows.cuh combines them).
template <typename R>
struct FscAcc {
    R h0, h1r, h1i, Mr, Mi, Sr, Si, Yr, Yi;   // powers of zeta over r
    R g1r, g1i, Or, Oi, w2r, w2i, Nr, Ni;     // powers of eta over r
    R t1, t2, tq, At1, At2, Atq;              // (y1, y2, q) / r^3, and times the end's depth a
    R s11, s12, s1q, s22, s2q;                // a x second derivatives of 1 / r
    R u, v, c3;                               // image segment: 1 / (r w), its I term, 1 / r^3
};
template <typename R>
struct FscDispAcc {
    R F, phi, chi, Br, Bi, B3r, B3i, B4r, B4i;
    R O1r, O1i, O2r, O2i, zg1r, zg1i;
    R ah0, zh0, azt1, azt2, aztq;
};

}  // namespace cad

#include "fsc_rows.cuh"

namespace cad {

// ------------------------------------------------------------------ records
// Every field of a record has the record's type T, so a record is a plain
// array of T: the FP32 copy used for far-field pairs is an element-wise
// conversion of the FP64 record (flags are stored as 0 / 1 values).
template <typename T>
struct FrameT {          // a TD (real or image) in its own coordinate system
    T P2[3];
    T P2lo[3];           // FP32 records: P2 - (double)(float)P2 (0 in FP64 records)
    T Vn[3], Vs[3], Vd[3];
    T p1y, p1z, p3y, p3z;           // TDCS (y, z) of P1 and P3; P2 is the origin
    T t23y, t32x, t31y, t13x, base; // on-a-side test constants
    T sy[3], sz[3];                 // unit vectors (TDCS y, z) of the sides P1-P2, P2-P3, P3-P1
    T flat;                         // 1: all vertex z exactly 0
};

template <typename T>
struct FscSideT {        // one TD side PA -> PB of the free-surface correction
    T skip;              // 1: the side has no correction (beta test); 2: it carries no slip (build_side_burgers)
    T ea, eb;            // horizontal direction of the side: ADCS y1 = ea X + eb Y, y2 = eb X - ea Y, y3 = -Z
    T PA[3];
    T PAlo[3];           // as P2lo
    T y1B, y2B;          // PB in ADCS
    T aA, aB;            // depths of the ends
    T s, c, nu;          // sine and cosine of the inclination beta, Poisson's ratio
    T cM, B1;            // -(1 - 2 nu) cot(beta) / 2, (1 - 2 nu) cot(beta)
    T ct2, tn2;          // cot and tan of beta / 2
    T K4;                // 1 / (4 pi (1 - nu))
    T cs[3][3];          // ADCS slip of each unit mode m (Dn, Dss, Dds), component g, times K4
    FscRows<T> ks;
    FscDispRows<T> kd;
};

template <typename T>
struct TriDevT {
    T Dss, Dds, Dn;
    T K8;                // 1 / (8 pi (1 - nu))
    FrameT<T> real;
    FrameT<T> image;
    FscSideT<T> side[3];
};

using Frame = FrameT<double>;
using FscSide = FscSideT<double>;
using TriDev = TriDevT<double>;
static_assert(sizeof(TriDevT<float>) * 2 == sizeof(TriDevT<double>), "records are plain arrays of their type");

// Number of values of a record needed by a full-space-only kernel / in all.
constexpr int kTriWordsFS = (int)(offsetof(TriDev, image) / sizeof(double));
constexpr int kTriWordsHS = (int)(sizeof(TriDev) / sizeof(double));
constexpr int kTriWordsImg = (int)(offsetof(TriDev, side) / sizeof(double));   // real + image frames
constexpr int kSideWords = (int)(sizeof(FscSide) / sizeof(double));

// ------------------------------------------------------------------ helpers
template <typename R>
CAD_HD R qnan()
{
#ifdef __CUDA_ARCH__
    return (R)__longlong_as_double(0x7ff8000000000000LL);
#else
    return (R)__builtin_nan("");
#endif
}

// Unfused arithmetic for the quantities that feed exact comparisons (TDCS
// coordinates, barycentric configuration test, side test), so that those
// decisions match an unfused FP64 evaluation bit for bit.
CAD_HD double mul_rn(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    double r = a * b;
#if !defined(__CUDACC__) && defined(__GNUC__) && defined(__x86_64__)
    asm("" : "+x"(r));   // plain C++ test build: keep the product out of any fused multiply-add
#endif
    return r;
#endif
}
CAD_HD double add_rn(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
CAD_HD double sub_rn(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dsub_rn(a, b);
#else
    return a - b;
#endif
}
CAD_HD float mul_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    float r = a * b;
#if !defined(__CUDACC__) && defined(__GNUC__) && defined(__x86_64__)
    asm("" : "+x"(r));
#endif
    return r;
#endif
}
CAD_HD float add_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fadd_rn(a, b);
#else
    return a + b;
#endif
}
CAD_HD float sub_rn(float a, float b)
{
#ifdef __CUDA_ARCH__
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}
template <typename R>
CAD_HD R dot3_rn(R a0, R a1, R a2, R b0, R b1, R b2)
{
    return add_rn(add_rn(mul_rn(a0, b0), mul_rn(a1, b1)), mul_rn(a2, b2));
}
CAD_HD double cad_atan2(double y, double x) { return atan2(y, x); }
CAD_HD float cad_atan2(float y, float x) { return atan2f(y, x); }

// Observation point minus a record origin, in R.  FP64 records subtract
// unfused; FP32 records subtract their origin's two float parts in FP64 and
// round the difference once.
template <typename R>
CAD_HD void rel_origin(const R* o, const R* olo, double X, double Y, double Z, R& dX, R& dY, R& dZ)
{
    if constexpr (sizeof(R) == sizeof(double)) {
        dX = sub_rn(X, (double)o[0]);
        dY = sub_rn(Y, (double)o[1]);
        dZ = sub_rn(Z, (double)o[2]);
    } else {
        dX = (R)((X - (double)o[0]) - (double)olo[0]);
        dY = (R)((Y - (double)o[1]) - (double)olo[1]);
        dZ = (R)((Z - (double)o[2]) - (double)olo[2]);
    }
}

// Symmetric tensor t (xx,yy,zz,xy,xz,yz) -> A-rotated, A column-major 3x3
// (TensorTransformation3D! form).
template <typename R>
CAD_HD void tensor_rot(R t[6], const R* A)
{
    const R two = R(2.0);
    const R Txx = t[0], Tyy = t[1], Tzz = t[2], Txy = t[3], Txz = t[4], Tyz = t[5];
    t[0] = A[0] * A[0] * Txx + two * A[0] * A[3] * Txy + two * A[0] * A[6] * Txz + two * A[3] * A[6] * Tyz +
           A[3] * A[3] * Tyy + A[6] * A[6] * Tzz;
    t[1] = A[1] * A[1] * Txx + two * A[1] * A[4] * Txy + two * A[1] * A[7] * Txz + two * A[4] * A[7] * Tyz +
           A[4] * A[4] * Tyy + A[7] * A[7] * Tzz;
    t[2] = A[2] * A[2] * Txx + two * A[2] * A[5] * Txy + two * A[2] * A[8] * Txz + two * A[5] * A[8] * Tyz +
           A[5] * A[5] * Tyy + A[8] * A[8] * Tzz;
    t[3] = A[0] * A[1] * Txx + (A[0] * A[4] + A[1] * A[3]) * Txy + (A[0] * A[7] + A[1] * A[6]) * Txz +
           (A[3] * A[7] + A[4] * A[6]) * Tyz + A[3] * A[4] * Tyy + A[6] * A[7] * Tzz;
    t[4] = A[0] * A[2] * Txx + (A[0] * A[5] + A[2] * A[3]) * Txy + (A[0] * A[8] + A[2] * A[6]) * Txz +
           (A[3] * A[8] + A[5] * A[6]) * Tyz + A[3] * A[5] * Tyy + A[6] * A[8] * Tzz;
    t[5] = A[1] * A[2] * Txx + (A[2] * A[4] + A[1] * A[5]) * Txy + (A[2] * A[7] + A[1] * A[8]) * Txz +
           (A[5] * A[7] + A[4] * A[8]) * Tyz + A[4] * A[5] * Tyy + A[7] * A[8] * Tzz;
}

// Observation point -> TDCS of frame f.
template <typename R>
CAD_HD void to_tdcs(const FrameT<R>& f, double X, double Y, double Z, R& x, R& y, R& z)
{
    R dX, dY, dZ;
    rel_origin(f.P2, f.P2lo, X, Y, Z, dX, dY, dZ);
    x = dot3_rn(f.Vn[0], f.Vn[1], f.Vn[2], dX, dY, dZ);
    y = dot3_rn(f.Vs[0], f.Vs[1], f.Vs[2], dX, dY, dZ);
    z = dot3_rn(f.Vd[0], f.Vd[1], f.Vd[2], dX, dY, dZ);
}

// Whether the point (TDCS) lies on a side of the triangle, in its plane: the
// reference's trimodefinder returning 0.  Its other two values select which
// way the angular dislocations run; segments need no such choice.
template <typename R>
CAD_HD bool on_side(const FrameT<R>& f, R x, R y, R z)
{
    if (x != 0.0) return false;
    const R dy = sub_rn(y, f.p3y), dz = sub_rn(z, f.p3z);
    const R a = add_rn(mul_rn(f.t23y, dy), mul_rn(f.t32x, dz)) / f.base;
    const R b = add_rn(mul_rn(f.t31y, dy), mul_rn(f.t13x, dz)) / f.base;
    const R c = sub_rn(sub_rn(R(1.0), a), b);
    if (a <= 0.0 && b > c && c > a) return false;
    if (b <= 0.0 && c > a && a > b) return false;
    if (c <= 0.0 && a > b && b > c) return false;
    return (a == 0.0 && b >= 0.0 && c >= 0.0) || (a >= 0.0 && b == 0.0 && c >= 0.0) ||
           (a >= 0.0 && b >= 0.0 && c == 0.0);
}

// ------------------------------------------------- full-space dislocation
// The field of a triangular dislocation depends on its boundary alone (the
// displacement also on the solid angle the triangle subtends), so it is the
// sum over the three sides of the line integrals of a straight dislocation
// segment (de Wit 1960; Hirth and Lothe, Theory of Dislocations, ch. 4).
// With d the offset of the point from the side's line, s the coordinate along
// it and R the distance, a side contributes
//   V = int ds / R    K = int ds / R^3    T = int s ds / R^3
//   I = 3 int ds / R^5                    Q = -3 int s ds / R^5
// One segment costs about a third of the angular dislocation it replaces, and
// the vertex distances serve two sides each.
template <typename R>
struct SegInt {
    R K, I, T, Q, V;
};

template <typename R>
CAD_HD constexpr R tiny_square()   // its reciprocal's square does not overflow
{
    return sizeof(R) == sizeof(double) ? R(1e-140) : R(1e-18);
}

// Integrals of one side from its end distances (R, 1 / R) and the coordinates
// sA, sB of the ends along it, rho2 = |d|^2.  The side is taken in the
// direction in which the nearer end has the smaller coordinate, so R + s of
// the farther end cannot cancel; the nearer end's is rho2 / (R - s) when its
// coordinate is negative.
template <bool LOG, typename R>
CAD_HD SegInt<R> seg_integrals(R RA, R iA, R RB, R iB, R sA, R sB, R rho2)
{
    const bool fwd = sA + sB >= R(0.0);
    const R a = fwd ? sA : -sB, b = fwd ? sB : -sA;
    const R Ra = fwd ? RA : RB, Rb = fwd ? RB : RA;
    const R ia = fwd ? iA : iB, ib = fwd ? iB : iA;
    const bool out = a >= R(0.0);
    // (a point exactly on the side keeps finite integrals: whether its pair is
    // NaN is on_side's decision, triangle by triangle)
    // (FP32 takes the place of 0 alone: offsets below 1e-9 are the size of a mesh in
    // very small units, whose field overflows rather than be wrong)
    const R least = sizeof(R) == sizeof(double) ? tiny_square<R>() : R(0.0);
    const R den = out ? Ra + a : (rho2 > least ? rho2 : tiny_square<R>()), num = out ? R(1.0) : Ra - a;
    const R wb = Rb + b;
    const R inv = R(1.0) / (den * wb);
    const R iwa = inv * wb * num, iwb = inv * den;   // 1 / (R + s) at both ends
    const R ua = ia * iwa, ub = ib * iwb;
    SegInt<R> g;
    g.K = ua - ub;
    g.I = ua * ua * (R(2.0) * Ra + a) * ia - ub * ub * (R(2.0) * Rb + b) * ib;
    g.T = iA - iB;
    g.Q = iA * iA * iA - iB * iB * iB;
    g.V = LOG ? cad_log(wb * iwa) : R(0.0);
    return g;
}

constexpr double kInv4Pi = 0.079577471545947667884;   // 1 / (4 pi)

// Strain of a segment for a unit Burgers vector along each of its own axes
// (n, m = t x n, t the side's direction): the point is offset (x, e) along
// (n, m).  First letter: the Burgers vector's axis.  k1 = 1 / (4 pi) and K8 =
// 1 / (8 pi (1 - nu)), or both times a common factor.
template <typename R>
struct SegStrain {
    R nnn, nmm, ntt, nnm, nmt, nnt;
    R mnn, mmm, mtt, mnm, mmt, mnt;
    R tnt, tmt;
};
template <typename R>
CAD_HD SegStrain<R> seg_strain(const SegInt<R>& g, R x, R e, R k1, R K8)
{
    const R x2 = x * x, e2 = e * e, ka = k1 - R(2.0) * K8;
    const R Hnn = x2 * g.I - g.K, Hmm = e2 * g.I - g.K, Htt = -(Hnn + Hmm);
    const R hT = R(0.5) * ka * g.T, kK = K8 * g.K, k1K = k1 * g.K, kaK = ka * g.K, kI = K8 * g.I, kQ = K8 * g.Q;
    SegStrain<R> s;
    s.nnn = e * (k1K + K8 * Hnn);
    s.nmm = e * (kaK + K8 * Hmm);
    s.ntt = K8 * e * Htt;
    s.nnm = x * (e2 * kI - kK);
    s.nmt = -hT - e2 * kQ;
    s.nnt = -e * x * kQ;
    s.mmm = -x * (k1K + K8 * Hmm);
    s.mnn = -x * (kaK + K8 * Hnn);
    s.mtt = -K8 * x * Htt;
    s.mnm = e * (kK - x2 * kI);
    s.mnt = hT + x2 * kQ;
    s.mmt = e * x * kQ;
    s.tnt = R(0.5) * e * k1K;
    s.tmt = R(-0.5) * x * k1K;
    return s;
}

// -Omega / (4 pi): the solid-angle part of the displacement (x the TDCS offset
// from the plane, dy, dz from the three vertices, Rv the vertex distances).
template <typename R>
CAD_HD R solid_angle_term(R x, const R dy[3], const R dz[3], const R Rv[3])
{
    const R x2 = x * x;
    const R one = -x * ((dy[1] - dy[0]) * (dz[2] - dz[0]) - (dz[1] - dz[0]) * (dy[2] - dy[0]));
    const R ab = x2 + dy[0] * dy[1] + dz[0] * dz[1];
    const R ac = x2 + dy[0] * dy[2] + dz[0] * dz[2];
    const R bc = x2 + dy[1] * dy[2] + dz[1] * dz[2];
    const R two = Rv[0] * Rv[1] * Rv[2] + ab * Rv[2] + ac * Rv[1] + bc * Rv[0];
    return R(-2.0) * R(kInv4Pi) * cad_atan2(one, two);
}

// Strain of unit slip n, strike, dip (TDCS xx, yy, zz, xy, xz, yz) and the
// displacement (its solid-angle part included) of frame f at TDCS (x, y, z).
// K8 = 1 / (8 pi (1 - nu)).  In the segment's own axes (n = TD normal,
// m = t x n in the plane, t along the side) the offset is (x, e, 0), the
// Hessian of V is H (diagonal entries x^2 I - K, e^2 I - K), and a unit
// Burgers vector b gives
//   strain -1/(4 pi) sym(b w) K + (1/(4 pi) - 2 K8) sym((b x t) grad V) - K8 (b.w) H
//   displacement 1/(4 pi) (b x t) V - K8 ((b x t) V + (b.w) grad V)
// with w = (-e, x, 0) and grad V = (-x K, -e K, T).
template <bool STRAIN, bool DISP, typename R>
CAD_HD void td_unit(const FrameT<R>& f, R x, R y, R z, R K8, R E[3][6], R U[3][3])
{
    const R k1 = R(kInv4Pi);
    const R dy[3] = {y - f.p1y, y, y - f.p3y}, dz[3] = {z - f.p1z, z, z - f.p3z};
    const R x2 = x * x;
    R Rv[3], iR[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const R q = x2 + dy[v] * dy[v] + dz[v] * dz[v];
        iR[v] = cad_rsqrt(q);
        Rv[v] = q * iR[v];
    }
    if (STRAIN) {
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int k = 0; k < 6; ++k) E[m][k] = R(0.0);
    }
    if (DISP) {
        const R Fi = solid_angle_term(x, dy, dz, Rv);
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
            for (int c = 0; c < 3; ++c) U[m][c] = m == c ? Fi : R(0.0);
    }
#pragma unroll
    for (int sd = 0; sd < 3; ++sd) {
        const int A = sd, B = sd == 2 ? 0 : sd + 1;
        const R ty = f.sy[sd], tz = f.sz[sd];
        const R sA = -(dy[A] * ty + dz[A] * tz), sB = -(dy[B] * ty + dz[B] * tz);
        const R e = dy[A] * tz - dz[A] * ty;
        const R e2 = e * e;
        const SegInt<R> g = seg_integrals<DISP>(Rv[A], iR[A], Rv[B], iR[B], sA, sB, x2 + e2);
        if (STRAIN) {
            const SegStrain<R> q = seg_strain(g, x, e, k1, K8);
            const R yy = ty * ty, zz = tz * tz, yz = ty * tz, dd = zz - yy;
            E[0][0] += q.nnn;
            E[0][1] += q.nmm * zz + q.ntt * yy + R(2.0) * q.nmt * yz;
            E[0][2] += q.nmm * yy + q.ntt * zz - R(2.0) * q.nmt * yz;
            E[0][3] += q.nnm * tz + q.nnt * ty;
            E[0][4] += q.nnt * tz - q.nnm * ty;
            E[0][5] += (q.ntt - q.nmm) * yz + q.nmt * dd;
            // b = m and b = t in TDCS, then unit strike = (tz m + ty t), unit dip = (-ty m + tz t)
            const R r1 = q.mmm * zz + q.mtt * yy + R(2.0) * q.mmt * yz;
            const R r2 = q.mmm * yy + q.mtt * zz - R(2.0) * q.mmt * yz;
            const R r3 = q.mnm * tz + q.mnt * ty, r4 = q.mnt * tz - q.mnm * ty;
            const R r5 = (q.mtt - q.mmm) * yz + q.mmt * dd;
            const R q1 = R(2.0) * q.tmt * yz, q3 = q.tnt * ty, q4 = q.tnt * tz, q5 = q.tmt * dd;
            E[1][0] += tz * q.mnn;
            E[1][1] += tz * r1 + ty * q1;
            E[1][2] += tz * r2 - ty * q1;
            E[1][3] += tz * r3 + ty * q3;
            E[1][4] += tz * r4 + ty * q4;
            E[1][5] += tz * r5 + ty * q5;
            E[2][0] += -ty * q.mnn;
            E[2][1] += tz * q1 - ty * r1;
            E[2][2] += -tz * q1 - ty * r2;
            E[2][3] += tz * q3 - ty * r3;
            E[2][4] += tz * q4 - ty * r4;
            E[2][5] += tz * q5 - ty * r5;
        }
        if (DISP) {
            const R cV = k1 - K8;
            // b = n: -cV V m + K8 e grad V;  b = m: cV V n - K8 x grad V;  b = t: none
            const R xK = x * g.K, eK = e * g.K;
            const R vm = -cV * g.V - K8 * e * eK, vt = K8 * e * g.T;
            const R um = -K8 * x * g.T, un = cV * g.V + K8 * x * xK, uw = K8 * x * eK;
            U[0][0] -= K8 * e * xK;
            U[0][1] += vm * tz + vt * ty;
            U[0][2] += vt * tz - vm * ty;
            const R a1 = uw * tz + um * ty, a2 = um * tz - uw * ty;
            U[1][0] += tz * un;
            U[1][1] += tz * a1;
            U[1][2] += tz * a2;
            U[2][0] -= ty * un;
            U[2][1] -= ty * a1;
            U[2][2] -= ty * a2;
        }
    }
}

// Strain (6) and displacement (3) at a point of frame f carrying the slip
// (Dn, Dss, Dds) = b, added into E and U (EFCS): td_unit with the Burgers vector
// contracted side by side, for sums over modes (6 strains instead of 18, one
// rotation instead of three).
template <bool STRAIN, bool DISP, typename R>
CAD_HD void td_net(const FrameT<R>& f, double X, double Y, double Z, R bn, R bs, R bd, R K8, R E[6], R U[3])
{
    R x, y, z;
    to_tdcs(f, X, Y, Z, x, y, z);
    const bool nan = on_side(f, x, y, z);
    const R k1 = R(kInv4Pi);
    const R dy[3] = {y - f.p1y, y, y - f.p3y}, dz[3] = {z - f.p1z, z, z - f.p3z};
    const R x2 = x * x;
    R Rv[3], iR[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const R q = x2 + dy[v] * dy[v] + dz[v] * dz[v];
        iR[v] = cad_rsqrt(q);
        Rv[v] = q * iR[v];
    }
    R T[6] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)}, V[3] = {R(0.0), R(0.0), R(0.0)};
    if (DISP) {
        const R Fi = solid_angle_term(x, dy, dz, Rv);
        V[0] = bn * Fi;
        V[1] = bs * Fi;
        V[2] = bd * Fi;
    }
#pragma unroll
    for (int sd = 0; sd < 3; ++sd) {
        const int A = sd, B = sd == 2 ? 0 : sd + 1;
        const R ty = f.sy[sd], tz = f.sz[sd];
        const R sA = -(dy[A] * ty + dz[A] * tz), sB = -(dy[B] * ty + dz[B] * tz);
        const R e = dy[A] * tz - dz[A] * ty;
        const SegInt<R> g = seg_integrals<DISP>(Rv[A], iR[A], Rv[B], iR[B], sA, sB, x2 + e * e);
        const R bm = tz * bs - ty * bd, bt = ty * bs + tz * bd;
        if (STRAIN) {
            const SegStrain<R> q = seg_strain(g, x, e, k1, K8);
            const R mm = bn * q.nmm + bm * q.mmm, tt = bn * q.ntt + bm * q.mtt;
            const R nm = bn * q.nnm + bm * q.mnm, nt = bn * q.nnt + bm * q.mnt + bt * q.tnt;
            const R mt = bn * q.nmt + bm * q.mmt + bt * q.tmt;
            const R yy = ty * ty, zz = tz * tz, yz = ty * tz;
            T[0] += bn * q.nnn + bm * q.mnn;
            T[1] += mm * zz + tt * yy + R(2.0) * mt * yz;
            T[2] += mm * yy + tt * zz - R(2.0) * mt * yz;
            T[3] += nm * tz + nt * ty;
            T[4] += nt * tz - nm * ty;
            T[5] += (tt - mm) * yz + mt * (zz - yy);
        }
        if (DISP) {
            const R cV = (k1 - K8) * g.V, w = K8 * (bn * e - bm * x);   // w grad V, and the V terms
            const R um = -w * e * g.K - bn * cV, ut = w * g.T;
            V[0] += bm * cV - w * x * g.K;
            V[1] += um * tz + ut * ty;
            V[2] += ut * tz - um * ty;
        }
    }
    if (STRAIN) {
        const R Rot[9] = {f.Vn[0], f.Vn[1], f.Vn[2], f.Vs[0], f.Vs[1], f.Vs[2], f.Vd[0], f.Vd[1], f.Vd[2]};
        tensor_rot(T, Rot);
#pragma unroll
        for (int k = 0; k < 6; ++k) E[k] += nan ? qnan<R>() : T[k];
    }
    if (DISP) {
#pragma unroll
        for (int c = 0; c < 3; ++c) U[c] += nan ? qnan<R>() : f.Vn[c] * V[0] + f.Vs[c] * V[1] + f.Vd[c] * V[2];
    }
}

// Adds the strain (EFCS) of frame f's slip modes into E.  A flat (z = 0) image
// triangle keeps the reference's detached xz / yz components: there the
// accumulated value is carried into the image TDCS, its xz and yz negated,
// and those two returned as they stood in the TDCS (src/TD.jl:1518-1525,
// :1610-1617).
template <bool IMAGE, typename R>
CAD_HD void add_strain(const FrameT<R>& f, bool nan, const R slip[3], R T[3][6], R E[3][6])
{
    const R Rot[9] = {f.Vn[0], f.Vn[1], f.Vn[2], f.Vs[0], f.Vs[1], f.Vs[2], f.Vd[0], f.Vd[1], f.Vd[2]};
    if (IMAGE && f.flat != R(0)) {
        const R RotInv[9] = {f.Vn[0], f.Vs[0], f.Vd[0], f.Vn[1], f.Vs[1], f.Vd[1], f.Vn[2], f.Vs[2], f.Vd[2]};
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            tensor_rot(E[m], RotInv);
            const R kx = E[m][4], ky = E[m][5];
            E[m][4] = -kx;
            E[m][5] = -ky;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                if (slip[m] != R(0.0)) E[m][k] += slip[m] * T[m][k];
                if (nan) E[m][k] = qnan<R>();
            }
            tensor_rot(E[m], Rot);
            E[m][4] = kx;
            E[m][5] = ky;
        }
        return;
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        tensor_rot(T[m], Rot);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            if (slip[m] != R(0.0)) E[m][k] += slip[m] * T[m][k];
            if (nan) E[m][k] = qnan<R>();
        }
    }
}

// The same for the displacement (flat image: the detached z component).
template <bool IMAGE, typename R>
CAD_HD void add_disp(const FrameT<R>& f, bool nan, const R slip[3], R T[3][3], R U[3][3])
{
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        R keep = R(0.0);
        const bool flat = IMAGE && f.flat != R(0);
        if (flat) {
            const R a = U[m][0], b = U[m][1], c = U[m][2];
            U[m][0] = f.Vn[0] * a + f.Vn[1] * b + f.Vn[2] * c;
            U[m][1] = f.Vs[0] * a + f.Vs[1] * b + f.Vs[2] * c;
            keep = f.Vd[0] * a + f.Vd[1] * b + f.Vd[2] * c;
            U[m][2] = -keep;
#pragma unroll
            for (int c2 = 0; c2 < 3; ++c2)
                if (slip[m] != R(0.0)) U[m][c2] += slip[m] * T[m][c2];
            const R p = U[m][0], q = U[m][1], r = U[m][2];
#pragma unroll
            for (int c2 = 0; c2 < 3; ++c2) U[m][c2] = f.Vn[c2] * p + f.Vs[c2] * q + f.Vd[c2] * r;
        } else if (slip[m] != R(0.0)) {
#pragma unroll
            for (int c2 = 0; c2 < 3; ++c2)
                U[m][c2] += slip[m] * (f.Vn[c2] * T[m][0] + f.Vs[c2] * T[m][1] + f.Vd[c2] * T[m][2]);
        }
        if (nan) U[m][0] = U[m][1] = U[m][2] = qnan<R>();
        if (flat) U[m][2] = keep;
    }
}

template <bool IMAGE, bool STRAIN, bool DISP, typename R>
CAD_HD void td_fs(const FrameT<R>& f, double X, double Y, double Z, R Dss, R Dds, R Dn, R K8, R E[3][6], R U[3][3])
{
    R x, y, z;
    to_tdcs(f, X, Y, Z, x, y, z);
    const bool nan = on_side(f, x, y, z);
    const R slip[3] = {Dn, Dss, Dds};
    R T[3][6], V[3][3];
    td_unit<STRAIN, DISP>(f, x, y, z, K8, T, V);
    if (STRAIN) add_strain<IMAGE>(f, nan, slip, T, E);
    if (DISP) add_disp<IMAGE>(f, nan, slip, V, U);
}

template <bool IMAGE, typename R>
CAD_HD void strain_fs(const FrameT<R>& f, double X, double Y, double Z, R Dss, R Dds, R Dn, R K8, R E[3][6])
{
    td_fs<IMAGE, true, false>(f, X, Y, Z, Dss, Dds, Dn, K8, E, (R(*)[3]) nullptr);
}

template <bool IMAGE, typename R>
CAD_HD void disp_fs(const FrameT<R>& f, double X, double Y, double Z, R Dss, R Dds, R Dn, R K8, R U[3][3])
{
    td_fs<IMAGE, false, true>(f, X, Y, Z, Dss, Dds, Dn, K8, (R(*)[6]) nullptr, U);
}

// --------------------------------------------------- free-surface correction
// out-of-line code that stays out of the callers' register allocation
#ifdef __CUDACC__
#define CAD_OUTLINE static __host__ __device__ __noinline__
#else
#define CAD_OUTLINE static inline
#endif

// Observation point -> horizontal ADCS coordinates of a side, relative to PA,
// and its depth.
template <typename R>
CAD_HD void to_adcs(const FscSideT<R>& s, double X, double Y, double Z, R& y1, R& y2, R& z)
{
    R dX, dY, dZ;
    rel_origin(s.PA, s.PAlo, X, Y, Z, dX, dY, dZ);
    y1 = s.ea * dX + s.eb * dY;
    y2 = s.eb * dX - s.ea * dY;
    z = (R)(-Z);
}

// What the strain's and the displacement's functions of one end share: r, 1 / r,
// 1 / (r + q), 1 / (r + f z3).
template <typename R>
struct FscEnd {
    R r, ir, ip, iw;
};

// Adds sg x the values of one end of a side (depth a, point at (y1, y2) from
// it and at depth z) to the accumulators.  f = +-1 takes the inclined leg's
// functions along +z3 or -z3 (both ends alike); w = r + f z3 is rho^2 / (r - f
// z3) where f z3 < 0, so it never cancels.
template <bool FIRST, typename R>
CAD_HD void fsc_end(const FscSideT<R>& k, R y1, R y2, R a, R z, R f, R z1, R z3, FscAcc<R>& v, FscEnd<R>& end)
{
    const R sg = FIRST ? R(-1.0) : R(1.0);
    const R q = z + a;
    const R r2 = y1 * y1 + y2 * y2 + q * q;
    const R ir = cad_rsqrt(r2), r = r2 * ir, ir2 = ir * ir, ir3 = ir2 * ir;
    const R zf = f * z3, p = r + q;
    const bool out = zf >= R(0.0);
    const R den = out ? r + zf : z1 * z1 + y2 * y2, num = out ? R(1.0) : r - zf;
    const R inv = R(1.0) / (p * den);
    const R ip = inv * den, iw = inv * p * num;
    end = FscEnd<R>{r, ir, ip, iw};
    const R N1 = R(1.0) - R(2.0) * k.nu, hN = R(0.5) * N1;
    const R c1r = y1 * ip, c1i = y2 * ip;                                    // zeta
    const R c2r = c1r * c1r - c1i * c1i, c2i = R(2.0) * c1r * c1i;
    const R c3r = c2r * c1r - c2i * c1i, c3i = c2r * c1i + c2i * c1r;
    const R n1r = z1 * iw, n1i = y2 * iw;                                    // f eta
    const R n2r = n1r * n1r - n1i * n1i, n2i = R(2.0) * n1r * n1i;
    const R n3r = n2r * n1r - n2i * n1i, n3i = n2r * n1i + n2i * n1r;
    const R kq = q * ir, kz = zf * ir, az = a * z;
    const R d2 = -(R(2.0) + kq) * ir2, d3 = -(R(3.0) + kq) * ir2;            // D h_m / zeta^m
    const R dd3 = (R(8.0) + kq * (R(9.0) + R(3.0) * kq)) * ir3;              // D^2 h_3 / zeta^3
    const R e2 = -(R(2.0) + kz) * ir2, e3 = (R(3.0) + kz) * ir2;
    const R ee3 = (R(8.0) + kz * (R(9.0) + R(3.0) * kz)) * ir3;
    const R m2 = sg * k.cM * (N1 * ir + (a + z) * d2);
    const R m3 = sg * (hN * k.nu * ir + R(0.5) * (k.nu * z - hN * a) * d3 - R(0.25) * az * dd3);
    const R ms = sg * (R(0.5) * (N1 * a - z) * d2 - hN * ir);
    const R my = sg * k.nu * z * d2;
    const R sir = sg * ir, sf = sg * f;
    v.h0 = (FIRST ? R(0.0) : v.h0) + sir;
    v.h1r = (FIRST ? R(0.0) : v.h1r) + sir * c1r;
    v.h1i = (FIRST ? R(0.0) : v.h1i) + sir * c1i;
    v.Mr = (FIRST ? R(0.0) : v.Mr) + m2 * c2r + m3 * c3r;
    v.Mi = (FIRST ? R(0.0) : v.Mi) + m2 * c2i + m3 * c3i;
    v.Sr = (FIRST ? R(0.0) : v.Sr) + ms * c2r;
    v.Si = (FIRST ? R(0.0) : v.Si) + ms * c2i;
    v.Yr = (FIRST ? R(0.0) : v.Yr) + my * c2r;
    v.Yi = (FIRST ? R(0.0) : v.Yi) + my * c2i;
    const R g1 = sf * ir, w2 = sf * e2;
    const R o2 = a * w2 - sg * k.c * ir, n3 = sg * R(0.25) * z * (f * a * ee3 + k.c * e3);
    v.g1r = (FIRST ? R(0.0) : v.g1r) + g1 * n1r;
    v.g1i = (FIRST ? R(0.0) : v.g1i) + g1 * n1i;
    v.Or = (FIRST ? R(0.0) : v.Or) + o2 * n2r;
    v.Oi = (FIRST ? R(0.0) : v.Oi) + o2 * n2i;
    v.w2r = (FIRST ? R(0.0) : v.w2r) + w2 * n2r;
    v.w2i = (FIRST ? R(0.0) : v.w2i) + w2 * n2i;
    v.Nr = (FIRST ? R(0.0) : v.Nr) + n3 * n3r;
    v.Ni = (FIRST ? R(0.0) : v.Ni) + n3 * n3i;
    const R s3 = sg * ir3, u1 = y1 * s3, u2 = y2 * s3, uq = q * s3, a3 = R(3.0) * a * ir2;
    v.t1 = (FIRST ? R(0.0) : v.t1) + u1;
    v.t2 = (FIRST ? R(0.0) : v.t2) + u2;
    v.tq = (FIRST ? R(0.0) : v.tq) + uq;
    v.At1 = (FIRST ? R(0.0) : v.At1) + a * u1;
    v.At2 = (FIRST ? R(0.0) : v.At2) + a * u2;
    v.Atq = (FIRST ? R(0.0) : v.Atq) + a * uq;
    v.s11 = (FIRST ? R(0.0) : v.s11) + (a3 * y1 * u1 - a * s3);
    v.s12 = (FIRST ? R(0.0) : v.s12) + a3 * y1 * u2;
    v.s1q = (FIRST ? R(0.0) : v.s1q) + a3 * y1 * uq;
    v.s22 = (FIRST ? R(0.0) : v.s22) + (a3 * y2 * u2 - a * s3);
    v.s2q = (FIRST ? R(0.0) : v.s2q) + a3 * y2 * uq;
    const R u = ir * iw;
    v.u = (FIRST ? R(0.0) : v.u) + sg * u;
    v.v = (FIRST ? R(0.0) : v.v) + sg * u * u * (R(2.0) + kz);
    v.c3 = (FIRST ? R(0.0) : v.c3) + s3;
}

// Adds a segment's strain to e[slip][component] (ADCS) for unit slips along the
// ADCS axes: the segment's axes are n = (c, 0, sg s), m = (0, 1, 0) and t =
// (-sg s, 0, c); g3 = -1 negates the vertical slip.
template <typename R>
CAD_HD void add_segment_adcs(const SegStrain<R>& q, R c, R ss, R g3, R e[3][6])   // ss = sg s
{
    const R cc = c * c, s2 = ss * ss, cs = c * ss, dd = cc - s2;
    const R a0 = cc * q.nnn + s2 * q.ntt - R(2.0) * cs * q.nnt, a2 = s2 * q.nnn + cc * q.ntt + R(2.0) * cs * q.nnt;
    const R a3 = c * q.nnm - ss * q.nmt, a4 = cs * (q.nnn - q.ntt) + dd * q.nnt, a5 = ss * q.nnm + c * q.nmt;
    const R b0 = R(2.0) * cs * q.tnt, b3 = ss * q.tmt, b4 = dd * q.tnt, b5 = c * q.tmt;   // -11, 33; -12; 13; 23
    e[0][0] += c * a0 + ss * b0;
    e[0][1] += c * q.nmm;
    e[0][2] += c * a2 - ss * b0;
    e[0][3] += c * a3 + ss * b3;
    e[0][4] += c * a4 - ss * b4;
    e[0][5] += c * a5 - ss * b5;
    e[1][0] += cc * q.mnn + s2 * q.mtt - R(2.0) * cs * q.mnt;
    e[1][1] += q.mmm;
    e[1][2] += s2 * q.mnn + cc * q.mtt + R(2.0) * cs * q.mnt;
    e[1][3] += c * q.mnm - ss * q.mmt;
    e[1][4] += cs * (q.mnn - q.mtt) + dd * q.mnt;
    e[1][5] += ss * q.mnm + c * q.mmt;
    const R gs = g3 * ss, gc = g3 * c;
    e[2][0] += gs * a0 - gc * b0;
    e[2][1] += gs * q.nmm;
    e[2][2] += gs * a2 + gc * b0;
    e[2][3] += gs * a3 - gc * b3;
    e[2][4] += gs * a4 + gc * b4;
    e[2][5] += gs * a5 + gc * b5;
}

// Strain of a side's correction in ADCS for a unit ADCS slip along each axis
// (divided by K4).  The functions of the two ends are differenced before any
// coefficient multiplies them: far from the side the ends nearly cancel.
// FULL: with the full-space fields of the side and of its mirror image added
// (the image segment runs along the same line as the correction's inclined
// leg and shares its functions; the image dislocation's Burgers vector is the
// mirrored one, reversed), so that the sum over a triangle's sides is its
// whole half-space strain.  A near-vertical side (skip) has no correction.
template <bool FULL, typename R>
CAD_HD void side_strain_adcs(const FscSideT<R>& s, double X, double Y, double Z, R e[3][6])
{
    R y1, y2, z;
    to_adcs(s, X, Y, Z, y1, y2, z);
    const R qA = z + s.aA, qB = z + s.aB;
    const R y1b = y1 - s.y1B, y2b = y2 - s.y2B;
    const R z3A = s.c * qA - s.s * y1, z3B = s.c * qB - s.s * y1b;
    const R f = z3A + z3B >= R(0.0) ? R(1.0) : R(-1.0);
    const R z1 = s.c * y1 + s.s * qA;
    FscAcc<R> v;
    FscEnd<R> eA, eB;
    fsc_end<true>(s, y1, y2, s.aA, z, f, z1, z3A, v, eA);
    fsc_end<false>(s, y1b, y2b, s.aB, z, f, s.c * y1b + s.s * qB, z3B, v, eB);
    if (FULL && s.skip != R(0)) {
#pragma unroll
        for (int k = 0; k < 18; ++k) e[k / 6][k % 6] = R(0.0);
    } else {
        fsc_rows(s.ks, v, z, e);
    }
    if (FULL) {
        const R k1 = R(1.0) - s.nu, K8 = R(0.5);   // 1 / (4 pi) and 1 / (8 pi (1 - nu)) over K4
        SegInt<R> g;
        g.K = -f * v.u;
        g.I = -f * v.v;
        g.T = v.h0;
        g.Q = v.c3;
        g.V = R(0.0);
        add_segment_adcs(seg_strain(g, z1, y2, k1, K8), s.c, s.s, R(-1.0), e);
        const R pA = z - s.aA, pB = z - s.aB;   // vertical offsets from the real ends
        const R x = s.c * y1 - s.s * pA;
        const R rA2 = fmax(y1 * y1 + y2 * y2 + pA * pA, tiny_square<R>());   // finite at a vertex too
        const R rB2 = fmax(y1b * y1b + y2b * y2b + pB * pB, tiny_square<R>());
        const R iA = cad_rsqrt(rA2), iB = cad_rsqrt(rB2);
        const SegInt<R> h = seg_integrals<false>(rA2 * iA, iA, rB2 * iB, iB, -(s.s * y1 + s.c * pA),
                                                 -(s.s * y1b + s.c * pB), x * x + y2 * y2);
        add_segment_adcs(seg_strain(h, x, y2, k1, K8), s.c, -s.s, R(1.0), e);
    }
}

// Tensor in ADCS -> EFCS (a rotation about the vertical axis).
template <typename R>
CAD_HD void adcs_to_efcs(R t[6], R a, R b)
{
    const R aa = a * a, bb = b * b, ab = a * b;
    const R t11 = t[0], t22 = t[1], t12 = t[3], t13 = t[4], t23 = t[5];
    t[0] = aa * t11 + bb * t22 + R(2.0) * ab * t12;
    t[1] = bb * t11 + aa * t22 - R(2.0) * ab * t12;
    t[3] = ab * (t11 - t22) + (bb - aa) * t12;
    t[4] = -(a * t13 + b * t23);
    t[5] = a * t23 - b * t13;
}

// One side's harmonic correction to the strain, added into E (EFCS).
template <typename R>
CAD_HD void fsc_strain(const FscSideT<R>& s, double X, double Y, double Z, R Dss, R Dds, R Dn, R E[3][6])
{
    R e[3][6];
    side_strain_adcs<false>(s, X, Y, Z, e);
    const R slip[3] = {Dn, Dss, Dds};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        R T[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) T[k] = s.cs[m][0] * e[0][k] + s.cs[m][1] * e[1][k] + s.cs[m][2] * e[2][k];
        adcs_to_efcs(T, s.ea, s.eb);
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] += T[k];
    }
}

// The same correction as a linear map of the side's Burgers vector: G[j] is
// the EFCS strain of a unit Burgers vector along EFCS axis j.  A side shared
// by two triangles is traversed in opposite directions, and the reversed
// side's map is the negative of this one (the two dislocation segments
// cancel), so one evaluation per mesh edge serves both triangles.
template <bool FULL, typename R>
CAD_HD void side_strain_map(const FscSideT<R>& s, double X, double Y, double Z, R G[3][6])
{
    R e[3][6];
    side_strain_adcs<FULL>(s, X, Y, Z, e);
    const R ca = s.K4 * s.ea, cb = s.K4 * s.eb;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        G[0][k] = ca * e[0][k] + cb * e[1][k];
        G[1][k] = cb * e[0][k] - ca * e[1][k];
        G[2][k] = -s.K4 * e[2][k];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) adcs_to_efcs(G[j], s.ea, s.eb);
}

// The whole half-space map of a side as tractions: W[j][r] = traction r
// (normal, strike, dip) on an element with axes n, ss, ds for a unit Burgers
// vector along EFCS axis j.  The element's axes are turned into ADCS, where
// each traction is one weighted sum of the six strains.
template <typename R>
CAD_HD void side_traction_map(const FscSideT<R>& s, double X, double Y, double Z, R lam, R G2, const R n[3],
                              const R ss[3], const R ds[3], R W[3][3])
{
    R e[3][6];
    side_strain_adcs<true>(s, X, Y, Z, e);
    const R g = s.K4 * G2, l = s.K4 * lam;
    const R n1 = s.ea * n[0] + s.eb * n[1], n2 = s.eb * n[0] - s.ea * n[1], n3 = -n[2];
    R t[3][3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const R* d = r == 0 ? n : r == 1 ? ss : ds;
        const R d1 = s.ea * d[0] + s.eb * d[1], d2 = s.eb * d[0] - s.ea * d[1], d3 = -d[2];
        const R li = r == 0 ? l * (n1 * n1 + n2 * n2 + n3 * n3) : R(0.0);
        const R p0 = g * n1 * d1 + li, p1 = g * n2 * d2 + li, p2 = g * n3 * d3 + li;
        const R p3 = g * (n1 * d2 + n2 * d1), p4 = g * (n1 * d3 + n3 * d1), p5 = g * (n2 * d3 + n3 * d2);
#pragma unroll
        for (int j = 0; j < 3; ++j)
            t[j][r] = p0 * e[j][0] + p1 * e[j][1] + p2 * e[j][2] + p3 * e[j][3] + p4 * e[j][4] + p5 * e[j][5];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        W[0][r] = s.ea * t[0][r] + s.eb * t[1][r];
        W[1][r] = s.eb * t[0][r] - s.ea * t[1][r];
        W[2][r] = -t[2][r];
    }
}

// E[m] += sign * (the map G applied to the EFCS Burgers vector of unit mode m
// of the triangle with frame `real`), for the modes with non-zero slip.
template <typename R>
CAD_HD void fsc_apply_map(const R (*G)[6], R sign, const FrameT<R>& real, R Dss, R Dds, R Dn, R E[3][6])
{
    const R slip[3] = {Dn, Dss, Dds};
    const R* axes[3] = {real.Vn, real.Vs, real.Vd};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        const R w0 = sign * axes[m][0] * slip[m], w1 = sign * axes[m][1] * slip[m], w2 = sign * axes[m][2] * slip[m];
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] += w0 * G[0][k] + w1 * G[1][k] + w2 * G[2][k];
    }
}

// Adds sg x one end's values to the displacement accumulators (h: the end's
// shared values, f their direction).  ff is that of the Burgers function, whose
// tangent's numerator and denominator are returned.
template <bool FIRST, typename R>
CAD_HD void fsc_disp_end(const FscSideT<R>& k, R y1, R y2, R a, R z, R f, R ff, const FscEnd<R>& h, FscDispAcc<R>& v,
                         R& fn, R& fd)
{
    const R sg = FIRST ? R(-1.0) : R(1.0);
    const R q = z + a;
    const R ir = h.ir, ir2 = ir * ir, ir3 = ir2 * ir;
    const R z1 = k.c * y1 + k.s * q, zf = f * (k.c * q - k.s * y1);
    const R p = h.r + q;
    fn = ff * y2;
    fd = ff > R(0.0) ? p * k.ct2 - y1 : y1 + p * k.tn2;
    const R ip = h.ip, iw = h.iw;
    const R N1 = R(1.0) - R(2.0) * k.nu, N2 = R(2.0) * (R(1.0) - k.nu);
    const R c1r = y1 * ip, c1i = y2 * ip;
    const R c2r = c1r * c1r - c1i * c1i, c2i = R(2.0) * c1r * c1i;
    const R n1r = z1 * iw, n1i = y2 * iw;
    const R n2r = n1r * n1r - n1i * n1i, n2i = R(2.0) * n1r * n1i;
    const R az = a * z, sir = sg * ir;
    const R b1 = sg * k.B1 * (N1 - (a + z) * ir);
    const R b2 = sg * (R(0.5) * (az * (R(2.0) + q * ir) * ir2 - N1 * (k.nu + a * ir)) + k.nu * z * ir);
    const R b3 = sg * (N1 + (N1 * a - z) * ir);
    const R b4 = sg * (R(2.0) * N2 * k.nu + (N2 * a + R(2.0) * k.nu * z) * ir);
    v.Br = (FIRST ? R(0.0) : v.Br) + b1 * c1r + b2 * c2r;
    v.Bi = (FIRST ? R(0.0) : v.Bi) + b1 * c1i + b2 * c2i;
    v.B3r = (FIRST ? R(0.0) : v.B3r) + b3 * c1r;
    v.B3i = (FIRST ? R(0.0) : v.B3i) + b3 * c1i;
    v.B4r = (FIRST ? R(0.0) : v.B4r) + b4 * c1r;
    v.B4i = (FIRST ? R(0.0) : v.B4i) + b4 * c1i;
    const R g1 = f * sir, o1 = sg * k.c + a * g1, o2 = -z * (a * f * sg * (R(2.0) + zf * ir) * ir2 + k.c * sir), zg = z * g1;
    v.O1r = (FIRST ? R(0.0) : v.O1r) + o1 * n1r;
    v.O1i = (FIRST ? R(0.0) : v.O1i) + o1 * n1i;
    v.O2r = (FIRST ? R(0.0) : v.O2r) + o2 * n2r;
    v.O2i = (FIRST ? R(0.0) : v.O2i) + o2 * n2i;
    v.zg1r = (FIRST ? R(0.0) : v.zg1r) + zg * n1r;
    v.zg1i = (FIRST ? R(0.0) : v.zg1i) + zg * n1i;
    const R t = sg * az * ir3;
    v.ah0 = (FIRST ? R(0.0) : v.ah0) + a * sir;
    v.zh0 = (FIRST ? R(0.0) : v.zh0) + z * sir;
    v.azt1 = (FIRST ? R(0.0) : v.azt1) + t * y1;
    v.azt2 = (FIRST ? R(0.0) : v.azt2) + t * y2;
    v.aztq = (FIRST ? R(0.0) : v.aztq) + t * q;
}

// Displacement of a side's correction in ADCS, d[3 component + slip], for a
// unit ADCS slip along each axis (without K4), from the ends' shared values eA,
// eB (direction f) and chi = int ds / R along the leg.  The Burgers function's
// own direction follows the side of the vertical plane through PA the point
// lies on, as the reference's choice between beta and beta - pi does: it then
// stays on one branch at both ends, and their difference is one arctangent.
template <typename R>
CAD_HD void fsc_disp_ends(const FscSideT<R>& s, R y1, R y2, R z, R f, const FscEnd<R>& eA, const FscEnd<R>& eB, R chi,
                          R d[9])
{
    const R ff = y1 >= R(0.0) ? R(-1.0) : R(1.0);
    FscDispAcc<R> v;
    R nA, dA, nB, dB;
    fsc_disp_end<true>(s, y1, y2, s.aA, z, f, ff, eA, v, nA, dA);
    fsc_disp_end<false>(s, y1 - s.y1B, y2 - s.y2B, s.aB, z, f, ff, eB, v, nB, dB);
    v.phi = cad_log(eA.ip * ((eB.r + z) + s.aB));
    v.chi = chi;
    v.F = R(2.0) * cad_atan2(nB * dA - nA * dB, dA * dB + nA * nB);
    fsc_disp_rows(s.kd, v, d);
}

template <typename R>
CAD_HD FscEnd<R> fsc_end_values(R y1, R y2, R q, R f, R z1, R z3)
{
    const R r2 = y1 * y1 + y2 * y2 + q * q;
    FscEnd<R> e;
    e.ir = cad_rsqrt(r2);
    e.r = r2 * e.ir;
    const R zf = f * z3, p = e.r + q;
    const bool out = zf >= R(0.0);
    const R den = out ? e.r + zf : z1 * z1 + y2 * y2, num = out ? R(1.0) : e.r - zf;
    const R inv = R(1.0) / (p * den);
    e.ip = inv * den;
    e.iw = inv * p * num;
    return e;
}

template <typename R>
CAD_HD void fsc_disp_adcs(const FscSideT<R>& s, double X, double Y, double Z, R d[9])
{
    R y1, y2, z;
    to_adcs(s, X, Y, Z, y1, y2, z);
    const R qA = z + s.aA, qB = z + s.aB;
    const R y1b = y1 - s.y1B, y2b = y2 - s.y2B;
    const R z3A = s.c * qA - s.s * y1, z3B = s.c * qB - s.s * y1b;
    const R f = z3A + z3B >= R(0.0) ? R(1.0) : R(-1.0);
    const FscEnd<R> eA = fsc_end_values(y1, y2, qA, f, s.c * y1 + s.s * qA, z3A);
    const FscEnd<R> eB = fsc_end_values(y1b, y2b, qB, f, s.c * y1b + s.s * qB, z3B);
    fsc_disp_ends(s, y1, y2, z, f, eA, eB, f * cad_log(eA.iw / eB.iw), d);
}

// Adds a segment's strain and displacement (its axes as in add_segment_adcs)
// for the Burgers vector (b0, b1, b2) along the ADCS axes to T and u.
template <bool DISP, typename R>
CAD_HD void add_segment_net(const SegInt<R>& g, R x, R e, R k1, R K8, R c, R ss, R b0, R b1, R b2, R T[6], R u[3])
{
    const SegStrain<R> q = seg_strain(g, x, e, k1, K8);
    const R bn = c * b0 + ss * b2, bm = b1, bt = c * b2 - ss * b0;
    const R nn = bn * q.nnn + bm * q.mnn, mm = bn * q.nmm + bm * q.mmm, tt = bn * q.ntt + bm * q.mtt;
    const R nm = bn * q.nnm + bm * q.mnm, nt = bn * q.nnt + bm * q.mnt + bt * q.tnt;
    const R mt = bn * q.nmt + bm * q.mmt + bt * q.tmt;
    const R cc = c * c, s2 = ss * ss, cs = c * ss;
    T[0] += cc * nn + s2 * tt - R(2.0) * cs * nt;
    T[1] += mm;
    T[2] += s2 * nn + cc * tt + R(2.0) * cs * nt;
    T[3] += c * nm - ss * mt;
    T[4] += cs * (nn - tt) + (cc - s2) * nt;
    T[5] += ss * nm + c * mt;
    if (DISP) {   // as in td_net
        const R cV = (k1 - K8) * g.V, w = K8 * (bn * e - bm * x);
        const R un = bm * cV - w * x * g.K, um = -w * e * g.K - bn * cV, ut = w * g.T;
        u[0] += c * un - ss * ut;
        u[1] += um;
        u[2] += ss * un + c * ut;
    }
}

// Strain and displacement (EFCS) at the point of side s carrying the slip of its
// mode 0: the correction and the real and image segments, without the solid
// angles; added into E and U.
template <bool DISP, typename R>
CAD_HD void side_sum_full(const FscSideT<R>& s, double X, double Y, double Z, R E[6], R U[3])
{
    R y1, y2, z;
    to_adcs(s, X, Y, Z, y1, y2, z);
    const R qA = z + s.aA, qB = z + s.aB;
    const R y1b = y1 - s.y1B, y2b = y2 - s.y2B;
    const R z3A = s.c * qA - s.s * y1, z3B = s.c * qB - s.s * y1b;
    const R f = z3A + z3B >= R(0.0) ? R(1.0) : R(-1.0);
    const R z1 = s.c * y1 + s.s * qA;
    const R b0 = s.cs[0][0], b1 = s.cs[0][1], b2 = s.cs[0][2];
    R T[6] = {R(0.0), R(0.0), R(0.0), R(0.0), R(0.0), R(0.0)}, u[3] = {R(0.0), R(0.0), R(0.0)};
    SegInt<R> g;
    FscEnd<R> eA, eB;
    {
        FscAcc<R> v;
        fsc_end<true>(s, y1, y2, s.aA, z, f, z1, z3A, v, eA);
        fsc_end<false>(s, y1b, y2b, s.aB, z, f, s.c * y1b + s.s * qB, z3B, v, eB);
        if (s.skip == R(0)) {
            R e[3][6];
            fsc_rows(s.ks, v, z, e);
#pragma unroll
            for (int k = 0; k < 6; ++k) T[k] = b0 * e[0][k] + b1 * e[1][k] + b2 * e[2][k];
        }
        g.K = -f * v.u;
        g.I = -f * v.v;
        g.T = v.h0;
        g.Q = v.c3;
    }
    g.V = DISP ? f * cad_log(eA.iw / eB.iw) : R(0.0);
    const R k1 = R(1.0) - s.nu, K8 = R(0.5);   // 1 / (4 pi) and 1 / (8 pi (1 - nu)) over K4
    add_segment_net<DISP>(g, z1, y2, k1, K8, s.c, s.s, b0, b1, -b2, T, u);
    {
        const R pA = z - s.aA, pB = z - s.aB;   // vertical offsets from the real ends
        const R x = s.c * y1 - s.s * pA;
        const R rA2 = fmax(y1 * y1 + y2 * y2 + pA * pA, tiny_square<R>());   // finite at a vertex too
        const R rB2 = fmax(y1b * y1b + y2b * y2b + pB * pB, tiny_square<R>());
        const R iA = cad_rsqrt(rA2), iB = cad_rsqrt(rB2);
        const SegInt<R> h = seg_integrals<DISP>(rA2 * iA, iA, rB2 * iB, iB, -(s.s * y1 + s.c * pA),
                                                -(s.s * y1b + s.c * pB), x * x + y2 * y2);
        add_segment_net<DISP>(h, x, y2, k1, K8, s.c, -s.s, b0, b1, b2, T, u);
    }
    if (DISP) {
        if (s.skip == R(0)) {
            R d[9];
            fsc_disp_ends(s, y1, y2, z, f, eA, eB, g.V, d);
#pragma unroll
            for (int i = 0; i < 3; ++i) u[i] += b0 * d[3 * i] + b1 * d[3 * i + 1] + b2 * d[3 * i + 2];
        }
        U[0] += s.ea * u[0] + s.eb * u[1];
        U[1] += s.eb * u[0] - s.ea * u[1];
        U[2] -= u[2];
    }
    adcs_to_efcs(T, s.ea, s.eb);
#pragma unroll
    for (int k = 0; k < 6; ++k) E[k] += T[k];
}

// One side's harmonic correction to the displacement, added into U (EFCS).
template <typename R>
CAD_HD void fsc_disp(const FscSideT<R>& s, double X, double Y, double Z, R Dss, R Dds, R Dn, R U[3][3])
{
    R d[9];
    fsc_disp_adcs(s, X, Y, Z, d);
    const R slip[3] = {Dn, Dss, Dds};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        R u[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) u[i] = s.cs[m][0] * d[3 * i] + s.cs[m][1] * d[3 * i + 1] + s.cs[m][2] * d[3 * i + 2];
        U[m][0] += s.ea * u[0] + s.eb * u[1];
        U[m][1] += s.eb * u[0] - s.ea * u[1];
        U[m][2] -= u[2];
    }
}

// The free-surface displacement of side s at (X, Y, Z) for a unit Burgers
// vector along EFCS axis j, without the factor 1 / (4 pi (1 - nu)).  As for
// the strain map, the reversed side's map is the negative of this one.
template <typename R>
CAD_HD void fsc_disp_map(const FscSideT<R>& s, double X, double Y, double Z, R Gu[3][3])
{
    R d[9];
    fsc_disp_adcs(s, X, Y, Z, d);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        R u[3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            u[i] = j == 0 ? s.ea * d[3 * i] + s.eb * d[3 * i + 1] : j == 1 ? s.eb * d[3 * i] - s.ea * d[3 * i + 1] : -d[3 * i + 2];
        Gu[j][0] = s.ea * u[0] + s.eb * u[1];
        Gu[j][1] = s.eb * u[0] - s.ea * u[1];
        Gu[j][2] = -u[2];
    }
}

// U[m] += sign * 2 K8 * (the map Gu applied to the EFCS Burgers vector of
// unit mode m of the triangle with frame `real`), for the modes with
// non-zero slip (2 K8 = 1 / (4 pi (1 - nu))).
template <typename R>
CAD_HD void fsc_apply_disp_map(const R Gu[3][3], R sign, const FrameT<R>& real, R Dss, R Dds, R Dn, R K8, R U[3][3])
{
    const R slip[3] = {Dn, Dss, Dds};
    const R* axes[3] = {real.Vn, real.Vs, real.Vd};
    const R f = sign * (K8 + K8);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        const R w0 = axes[m][0] * slip[m], w1 = axes[m][1] * slip[m], w2 = axes[m][2] * slip[m];
#pragma unroll
        for (int c = 0; c < 3; ++c) U[m][c] += f * (w0 * Gu[0][c] + w1 * Gu[1][c] + w2 * Gu[2][c]);
    }
}

// -------------------------------------------------------- triangle setup
// The per-triangle setup uses unfused arithmetic throughout: it is negligible
// work, and the half-space terms of the two ends of a side cancel far from the
// side, which amplifies any inconsistency between the side angle beta and the
// side vector (fused rounding of |S| alone is enough to show).
CAD_HD double sq_rn(double a) { return mul_rn(a, a); }
CAD_HD double norm3_rn(double a, double b, double c) { return sqrt(add_rn(add_rn(sq_rn(a), sq_rn(b)), sq_rn(c))); }
CAD_HD void cross3_rn(const double a[3], const double b[3], double c[3])
{
    c[0] = sub_rn(mul_rn(a[1], b[2]), mul_rn(a[2], b[1]));
    c[1] = sub_rn(mul_rn(a[2], b[0]), mul_rn(a[0], b[2]));
    c[2] = sub_rn(mul_rn(a[0], b[1]), mul_rn(a[1], b[0]));
}

CAD_HD void build_frame(const double P1[3], const double P2[3], const double P3[3], Frame& f)
{
    double a[3], b[3], Vn[3], Vs[3], Vd[3];
    for (int i = 0; i < 3; ++i) { a[i] = sub_rn(P2[i], P1[i]); b[i] = sub_rn(P3[i], P1[i]); }
    cross3_rn(a, b, Vn);
    const double nn = norm3_rn(Vn[0], Vn[1], Vn[2]);
    for (int i = 0; i < 3; ++i) Vn[i] = Vn[i] / nn;
    const double eZ[3] = {0.0, 0.0, 1.0};
    cross3_rn(eZ, Vn, Vs);
    if (Vs[0] == 0.0 && Vs[1] == 0.0 && Vs[2] == 0.0) {   // horizontal TD
        Vs[0] = mul_rn(0.0, Vn[2]);
        Vs[1] = mul_rn(1.0, Vn[2]);
        Vs[2] = mul_rn(0.0, Vn[2]);
    }
    const double ns = norm3_rn(Vs[0], Vs[1], Vs[2]);
    for (int i = 0; i < 3; ++i) Vs[i] = Vs[i] / ns;
    cross3_rn(Vn, Vs, Vd);
    for (int i = 0; i < 3; ++i) { f.P2[i] = P2[i]; f.Vn[i] = Vn[i]; f.Vs[i] = Vs[i]; f.Vd[i] = Vd[i]; }

    double p1[3], p3[3];
    {
        const double d1[3] = {sub_rn(P1[0], P2[0]), sub_rn(P1[1], P2[1]), sub_rn(P1[2], P2[2])};
        const double d3[3] = {sub_rn(P3[0], P2[0]), sub_rn(P3[1], P2[1]), sub_rn(P3[2], P2[2])};
        p1[0] = dot3_rn(Vn[0], Vn[1], Vn[2], d1[0], d1[1], d1[2]);
        p1[1] = dot3_rn(Vs[0], Vs[1], Vs[2], d1[0], d1[1], d1[2]);
        p1[2] = dot3_rn(Vd[0], Vd[1], Vd[2], d1[0], d1[1], d1[2]);
        p3[0] = dot3_rn(Vn[0], Vn[1], Vn[2], d3[0], d3[1], d3[2]);
        p3[1] = dot3_rn(Vs[0], Vs[1], Vs[2], d3[0], d3[1], d3[2]);
        p3[2] = dot3_rn(Vd[0], Vd[1], Vd[2], d3[0], d3[1], d3[2]);
    }
    f.p1y = p1[1]; f.p1z = p1[2]; f.p3y = p3[1]; f.p3z = p3[2];
    double e12[3], e13[3], e23[3];
    for (int i = 0; i < 3; ++i) { e12[i] = sub_rn(0.0, p1[i]); e13[i] = sub_rn(p3[i], p1[i]); e23[i] = sub_rn(p3[i], 0.0); }
    const double n12 = norm3_rn(e12[0], e12[1], e12[2]);
    const double n13 = norm3_rn(e13[0], e13[1], e13[2]);
    const double n23 = norm3_rn(e23[0], e23[1], e23[2]);
    for (int i = 0; i < 3; ++i) { e12[i] /= n12; e13[i] /= n13; e23[i] /= n23; }
    // on-a-side test constants (trimodefinder on the TDCS (y, z) plane)
    f.t23y = sub_rn(0.0, p3[2]);
    f.t32x = sub_rn(p3[1], 0.0);
    f.t13x = sub_rn(p1[1], p3[1]);
    const double t13y = sub_rn(p1[2], p3[2]);
    f.t31y = sub_rn(p3[2], p1[2]);
    f.base = add_rn(mul_rn(f.t23y, f.t13x), mul_rn(f.t32x, t13y));

    const double* side[3] = {e12, e23, e13};
    for (int v = 0; v < 3; ++v) {
        f.sy[v] = v == 2 ? -side[v][1] : side[v][1];
        f.sz[v] = v == 2 ? -side[v][2] : side[v][2];
    }
    f.flat = (P1[2] == 0.0 && P2[2] == 0.0 && P3[2] == 0.0) ? 1.0 : 0.0;
    for (int i = 0; i < 3; ++i) f.P2lo[i] = 0.0;
}

// The geometry of side PA -> PB (frame, beta test, row coefficients); its
// slip coefficients cs are left zero.
CAD_HD void build_side_geom(const double PA[3], const double PB[3], double nu, FscSide& s)
{
    for (int m = 0; m < 3; ++m)
        for (int g = 0; g < 3; ++g) s.cs[m][g] = 0.0;
    const double S[3] = {sub_rn(PB[0], PA[0]), sub_rn(PB[1], PA[1]), sub_rn(PB[2], PA[2])};
    const double Sv = norm3_rn(S[0], S[1], S[2]);
    const double beta = acos(-S[2] / Sv);
    s.skip = ((fabs(beta) < DBL_EPSILON) || (fabs(M_PI - beta) < DBL_EPSILON) || (fabs(1.0 / tan(beta)) > 5e3)) ? 1.0 : 0.0;
    for (int i = 0; i < 3; ++i) { s.PA[i] = PA[i]; s.PAlo[i] = 0.0; }
    const double n1 = norm3_rn(S[0], S[1], 0.0);
    s.ea = n1 > 0.0 ? S[0] / n1 : 1.0;
    s.eb = n1 > 0.0 ? S[1] / n1 : 0.0;
    s.y1B = add_rn(mul_rn(s.ea, S[0]), mul_rn(s.eb, S[1]));
    s.y2B = sub_rn(mul_rn(s.eb, S[0]), mul_rn(s.ea, S[1]));
    s.aA = -PA[2];
    s.aB = -PB[2];
    s.s = n1 / Sv;
    s.c = -S[2] / Sv;
    s.nu = nu;
    s.K4 = 1.0 / (4.0 * M_PI * sub_rn(1.0, nu));
    s.B1 = s.cM = 0.0;
    s.ct2 = s.tn2 = 1.0;
    if (s.skip != 0.0) return;
    const double N1 = sub_rn(1.0, mul_rn(2.0, nu));
    s.B1 = N1 * s.c / s.s;
    s.cM = -0.5 * s.B1;
    s.ct2 = (1.0 + s.c) / s.s;   // cot(beta / 2)
    s.tn2 = s.s / (1.0 + s.c);
    if (s.c < 0.0) {
        s.ct2 = s.s / (1.0 - s.c);
        s.tn2 = (1.0 - s.c) / s.s;
    }
    fsc_rows_setup(s.s, s.c, nu, s.ks);
    fsc_rows_setup(s.s, s.c, nu, s.kd);
}

// EFCS Burgers vector w -> the side's ADCS slip coefficients (times K4).
CAD_HD void side_slip(const FscSide& s, const double w[3], double cs[3])
{
    cs[0] = mul_rn(s.K4, add_rn(mul_rn(s.ea, w[0]), mul_rn(s.eb, w[1])));
    cs[1] = mul_rn(s.K4, sub_rn(mul_rn(s.eb, w[0]), mul_rn(s.ea, w[1])));
    cs[2] = -mul_rn(s.K4, w[2]);
}

CAD_HD void build_side(const double PA[3], const double PB[3], const Frame& real, double Dss, double Dds,
                       double Dn, double nu, FscSide& s)
{
    build_side_geom(PA, PB, nu, s);
    // unit-mode slip vectors: TDCS (n, s, d) -> EFCS -> ADCS
    const double slip[3] = {Dn, Dss, Dds};
    const double* axes[3] = {real.Vn, real.Vs, real.Vd};
    for (int m = 0; m < 3; ++m) {
        double w[3];
        for (int i = 0; i < 3; ++i) w[i] = mul_rn(axes[m][i], slip[m]);
        side_slip(s, w, s.cs[m]);
    }
}

// Side PA -> PB carrying the net Burgers vector B (EFCS) of every triangle side
// on that mesh edge, as unit mode 0 (evaluate with Dn = 1, Dss = Dds = 0).  The
// slip coefficients follow build_side's for w = B.  skip is 2 where B is zero:
// the side adds nothing whatever its geometry (it may have no length).
CAD_HD void build_side_burgers(const double PA[3], const double PB[3], const double B[3], double nu, FscSide& s)
{
    build_side_geom(PA, PB, nu, s);
    side_slip(s, B, s.cs[0]);
    if (B[0] == 0.0 && B[1] == 0.0 && B[2] == 0.0) s.skip = 2.0;
}

// ------------------------------------------- full-space sums over mesh edges
// A mesh edge PA -> PB with the net Burgers vector B of the triangle sides on
// it: unit direction t and length, and B in the products a point needs, with k1 = 1 / (4 pi),
// K8 = 1 / (8 pi (1 - nu)).
struct SegRec {
    double PA[3], t[3], len;
    double b1[3];   // -k1 / 2 B
    double bK[3];   // -K8 B
    double c1[3];   // (k1 - 2 K8) / 2 B x t
    double c2[3];   // (k1 - K8) B x t
    double slips;   // 0 where B is zero
};
constexpr int kSegWords = (int)(sizeof(SegRec) / sizeof(double));

CAD_HD void build_segment(const double PA[3], const double PB[3], const double B[3], double K8, SegRec& s)
{
    const bool none = B[0] == 0.0 && B[1] == 0.0 && B[2] == 0.0;   // (its sides may have no direction)
    const double S[3] = {PB[0] - PA[0], PB[1] - PA[1], PB[2] - PA[2]};
    const double len = norm3_rn(S[0], S[1], S[2]), ka = kInv4Pi - 2.0 * K8;
    for (int i = 0; i < 3; ++i) {
        s.PA[i] = PA[i];
        s.t[i] = none ? (i == 0 ? 1.0 : 0.0) : S[i] / len;
        s.b1[i] = -0.5 * kInv4Pi * B[i];
        s.bK[i] = -K8 * B[i];
    }
    s.len = none ? 0.0 : len;
    double c[3];
    cross3_rn(B, s.t, c);
    for (int i = 0; i < 3; ++i) {
        s.c1[i] = 0.5 * ka * c[i];
        s.c2[i] = (kInv4Pi - K8) * c[i];
    }
    s.slips = none ? 0.0 : 1.0;
}

// Strain of a segment at a point, added into E, and its displacement (but for
// the solid angles), added into U; EFCS throughout.  With r the point's offset
// from the segment's line and w = t x r,
//   grad V = T t - K r,  H = I r r + (3 K - I r.r) t t - K 1 - Q (r t + t r)
//   strain = -k1 K sym(B w) + (k1 - 2 K8) sym((B x t) grad V) - K8 (B.w) H
//   displacement = (k1 - K8) V B x t - K8 (B.w) grad V
template <bool STRAIN, bool DISP>
CAD_HD void segment_sum(const SegRec& s, double X, double Y, double Z, double E[6], double U[3])
{
    const double d[3] = {X - s.PA[0], Y - s.PA[1], Z - s.PA[2]};
    const double* t = s.t;
    const double at = d[0] * t[0] + d[1] * t[1] + d[2] * t[2];
    const double r[3] = {d[0] - at * t[0], d[1] - at * t[1], d[2] - at * t[2]};
    const double w[3] = {t[1] * r[2] - t[2] * r[1], t[2] * r[0] - t[0] * r[2], t[0] * r[1] - t[1] * r[0]};
    const double rho2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    const double sA = -at, sB = s.len - at;
    const double qA = fmax(rho2 + sA * sA, tiny_square<double>()), qB = fmax(rho2 + sB * sB, tiny_square<double>());
    const double iA = cad_rsqrt(qA), iB = cad_rsqrt(qB);
    const SegInt<double> g = seg_integrals<DISP>(qA * iA, iA, qB * iB, iB, sA, sB, rho2);
    const double be = s.bK[0] * w[0] + s.bK[1] * w[1] + s.bK[2] * w[2];
    const double gv[3] = {g.T * t[0] - g.K * r[0], g.T * t[1] - g.K * r[1], g.T * t[2] - g.K * r[2]};
    if (STRAIN) {
        const double bK = be * g.K, hI = 0.5 * be * g.I, hQ = be * g.Q, tt = 3.0 * bK - be * g.I * rho2;
        double a[3], b[3], kw[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = hI * r[i] - hQ * t[i];
            b[i] = tt * t[i];
            kw[i] = g.K * w[i];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
            E[i] += 2.0 * (s.b1[i] * kw[i] + s.c1[i] * gv[i] + r[i] * a[i]) + t[i] * b[i] - bK;
#pragma unroll
        for (int k = 3; k < 6; ++k) {
            const int i = k == 5 ? 1 : 0, j = k == 3 ? 1 : 2;
            E[k] += s.b1[i] * kw[j] + s.b1[j] * kw[i] + s.c1[i] * gv[j] + s.c1[j] * gv[i] + r[i] * a[j] + r[j] * a[i] +
                    t[i] * b[j];
        }
    }
    if (DISP)
#pragma unroll
        for (int c = 0; c < 3; ++c) U[c] += g.V * s.c2[c] + be * gv[c];
}

// ------------------------------------------------------------ pair drivers
// Whether the point lies on a side or a vertex of the triangle or of its
// mirror image, in its plane (the pair is NaN there).
CAD_HD bool on_side_or_vertex(const Frame& f, double X, double Y, double Z)
{
    double x, y, z;
    to_tdcs(f, X, Y, Z, x, y, z);
    if (x != 0.0) return false;
    return on_side(f, x, y, z) || (y == 0.0 && z == 0.0) || (y == f.p1y && z == f.p1z) || (y == f.p3y && z == f.p3z);
}
CAD_HD bool pair_on_side(const TriDev& t, double X, double Y, double Z)
{
    return on_side_or_vertex(t.real, X, Y, Z) || on_side_or_vertex(t.image, X, Y, Z);
}

template <bool HS, typename R>
CAD_HD void pair_strain(const TriDevT<R>& t, double X, double Y, double Z, R E[3][6])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] = R(0.0);
    strain_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
    if (HS) {
#pragma unroll 1
        for (int sd = 0; sd < 3; ++sd)
            if (t.side[sd].skip == R(0)) fsc_strain(t.side[sd], X, Y, Z, t.Dss, t.Dds, t.Dn, E);
        strain_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
    }
}

// Sum of the three sides' maps of this triangle at a point, signed by the
// sides' directions: entry (edge e, value q) at G[e * ge + q * gq]; code[sd] =
// +-(e + 1) for side sd traversed along / against edge e's direction, 0 for
// none.
template <int Q>
CAD_HD void sum_side_maps(const double* G, int64_t gq, int64_t ge, const int* code, double S[Q])
{
#pragma unroll
    for (int q = 0; q < Q; ++q) S[q] = 0.0;
#pragma unroll
    for (int sd = 0; sd < 3; ++sd) {
        const int c = code[sd];
        if (c == 0) continue;
        const double* g = G + ((int64_t)(c > 0 ? c : -c) - 1) * ge;
        const double sg = c > 0 ? 1.0 : -1.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) S[q] += sg * g[q * gq];
    }
}

// Half-space strain with the sides' corrections read from per-edge maps
// (side_strain_map<false>), real and image full-space terms evaluated here.
CAD_HD void pair_strain_edges(const TriDev& t, double X, double Y, double Z, const double* G, int64_t gq, int64_t ge,
                              const int* code, double E[3][6])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] = 0.0;
    strain_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
    double S[18];
    sum_side_maps<18>(G, gq, ge, code, S);
    fsc_apply_map((double(*)[6])S, 1.0, t.real, t.Dss, t.Dds, t.Dn, E);
    strain_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
}

// Half-space strain from maps that hold all of it (side_strain_map<true>).
CAD_HD void pair_strain_full(const TriDev& t, double X, double Y, double Z, const double* G, int64_t gq, int64_t ge,
                             const int* code, double E[3][6])
{
    double S[18];
    sum_side_maps<18>(G, gq, ge, code, S);
    const bool nan = pair_on_side(t, X, Y, Z);
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] = nan ? qnan<double>() : 0.0;
    fsc_apply_map((double(*)[6])S, 1.0, t.real, t.Dss, t.Dds, t.Dn, E);
}

// Half-space strain and displacement without the free-surface corrections
// (real and image full-space terms only): the shared-edge sums add the
// corrections once per mesh edge.
CAD_HD void pair_strain_fs_image(const TriDev& t, double X, double Y, double Z, double E[3][6])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] = 0.0;
    strain_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
    strain_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
}

CAD_HD void pair_disp_fs_image(const TriDev& t, double X, double Y, double Z, double U[3][3])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) U[m][c] = 0.0;
    disp_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
    disp_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
}

// Half-space displacement with the free-surface corrections of the triangle's
// sides read from per-edge maps (fsc_disp_map), addressed as in
// pair_strain_edges.
CAD_HD void pair_disp_edges(const TriDev& t, double X, double Y, double Z, const double* G, int64_t gq, int64_t ge,
                            const int* code, double U[3][3])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) U[m][c] = 0.0;
    disp_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
#pragma unroll 1
    for (int sd = 0; sd < 3; ++sd) {
        const int c = code[sd];
        if (c == 0) continue;
        const int64_t e = (int64_t)(c > 0 ? c : -c) - 1;
        double Gu[3][3];
#pragma unroll
        for (int q = 0; q < 9; ++q) Gu[q / 3][q % 3] = G[e * ge + q * gq];
        fsc_apply_disp_map(Gu, c > 0 ? 1.0 : -1.0, t.real, t.Dss, t.Dds, t.Dn, t.K8, U);
    }
    disp_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
}

template <bool HS, typename R>
CAD_HD void pair_disp(const TriDevT<R>& t, double X, double Y, double Z, R U[3][3])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int c = 0; c < 3; ++c) U[m][c] = R(0.0);
    disp_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
    if (HS) {
#pragma unroll 1
        for (int sd = 0; sd < 3; ++sd)
            if (t.side[sd].skip == R(0)) fsc_disp(t.side[sd], X, Y, Z, t.Dss, t.Dds, t.Dn, U);
        disp_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, U);
    }
}

// Sums over the modes of the real (HS: and image) full-space terms of a
// triangle, added into E and U.  A flat image keeps the reference's per-mode
// order (add_strain, add_disp).
template <bool STRAIN, bool DISP>
CAD_OUTLINE void pair_net_flat(const TriDev& t, double X, double Y, double Z, double E[6], double U[3])
{
    if (STRAIN) {
        double M[3][6];
        pair_strain_fs_image(t, X, Y, Z, M);
        for (int k = 0; k < 6; ++k) E[k] += (M[0][k] + M[1][k]) + M[2][k];
    }
    if (DISP) {
        double M[3][3];
        pair_disp_fs_image(t, X, Y, Z, M);
        for (int c = 0; c < 3; ++c) U[c] += (M[0][c] + M[1][c]) + M[2][c];
    }
}
template <bool HS, bool STRAIN, bool DISP>
CAD_HD void pair_net(const TriDev& t, double X, double Y, double Z, double E[6], double U[3])
{
    if (t.Dn == 0.0 && t.Dss == 0.0 && t.Dds == 0.0) {   // only the NaN of points on a side is left
        double x, y, z;
        to_tdcs(t.real, X, Y, Z, x, y, z);
        bool nan = on_side(t.real, x, y, z);
        if (HS) nan = nan || pair_on_side(t, X, Y, Z);
        if (nan) {
            if (STRAIN)
                for (int k = 0; k < 6; ++k) E[k] = qnan<double>();
            if (DISP)
                for (int c = 0; c < 3; ++c) U[c] = qnan<double>();
        }
        return;
    }
    if (HS && t.image.flat != 0.0) {
        pair_net_flat<STRAIN, DISP>(t, X, Y, Z, E, U);
        return;
    }
    td_net<STRAIN, DISP>(t.real, X, Y, Z, t.Dn, t.Dss, t.Dds, t.K8, E, U);
    if (HS) td_net<STRAIN, DISP>(t.image, X, Y, Z, t.Dn, t.Dss, t.Dds, t.K8, E, U);
}

// -Omega / (4 pi) x the slip of a frame's triangle (EFCS), added into U.
CAD_HD void add_angle(const Frame& f, double X, double Y, double Z, double Dss, double Dds, double Dn, double U[3])
{
    double x, y, z;
    to_tdcs(f, X, Y, Z, x, y, z);
    const double dy[3] = {y - f.p1y, y, y - f.p3y}, dz[3] = {z - f.p1z, z, z - f.p3z};
    double Rv[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        const double q = x * x + dy[v] * dy[v] + dz[v] * dz[v];
        Rv[v] = q * cad_rsqrt(q);
    }
    const double Fi = solid_angle_term(x, dy, dz, Rv);
    const double bn = Dn * Fi, bs = Dss * Fi, bd = Dds * Fi;
#pragma unroll
    for (int c = 0; c < 3; ++c) U[c] += f.Vn[c] * bn + f.Vs[c] * bs + f.Vd[c] * bd;
}

// What displacement sums over mesh edges leave to each triangle: the solid
// angles (HS: the mirror image's too), and NaN where the point lies on a side.
template <bool HS, bool STRAIN>
CAD_HD void pair_angle(const TriDev& t, double X, double Y, double Z, double E[6], double U[3])
{
    if (t.Dn != 0.0 || t.Dss != 0.0 || t.Dds != 0.0) {
        add_angle(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, U);
        if (HS) add_angle(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, U);
    }
    if (HS ? pair_on_side(t, X, Y, Z) : on_side_or_vertex(t.real, X, Y, Z)) {
        if (STRAIN)
            for (int k = 0; k < 6; ++k) E[k] = qnan<double>();
        for (int c = 0; c < 3; ++c) U[c] = qnan<double>();
    }
}

// sides = false leaves the half-space sides unset (their fields come from the
// mesh's edges).
CAD_HD void build_triangle(const double a[3], const double b[3], const double c[3], double Dss, double Dds,
                           double Dn, double nu, bool hs, TriDev& t, bool sides = true)
{
    t.Dss = Dss;
    t.Dds = Dds;
    t.Dn = Dn;
    t.K8 = 1.0 / (8.0 * M_PI * (1.0 - nu));
    build_frame(a, b, c, t.real);
    if (!hs) return;
    const double ai[3] = {a[0], a[1], -a[2]}, bi[3] = {b[0], b[1], -b[2]}, ci[3] = {c[0], c[1], -c[2]};
    build_frame(ai, bi, ci, t.image);
    if (!sides) return;
    build_side(a, b, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[0]);
    build_side(b, c, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[1]);
    build_side(c, a, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[2]);
}

}  // namespace cad
