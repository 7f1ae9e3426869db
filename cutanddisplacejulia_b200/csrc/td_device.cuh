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
// The closed-form angular-dislocation terms come from tde_closed_form.cuh.
//
// Data layout: everything that depends only on the triangle (frames, angles,
// per-dislocation constants of every closed-form term, slip rotations) is
// computed once per triangle by td_setup_kernel into a TriDev record; the pair
// kernels stage one TriDev at a time in shared memory and every thread of the
// block (one observation point each) reads it as a broadcast.
#pragma once
#include <cfloat>
#include <cstddef>
#include <cstdint>

#include "tde_closed_form.cuh"

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
    T skip;              // 1: the side adds nothing (beta test)
    T ey1[3], ey2[3], ey3[3];
    T PA[3];
    T PAlo[3];           // as P2lo
    T y1B, y2B, y3B;
    T beta;
    T cs[3][3];          // ADCS slip of each unit mode m (Dn, Dss, Dds), component g
    T cd[3][3];          // the same scaled by 1 / (4 pi (1 - nu)) for displacements
    ang_dis_strain_fsc_k<T> ks[2][2];   // [0: beta, 1: pi - beta][0: at PA, 1: at PB]
    ang_dis_disp_fsc_k<T> kd[2][2];     // [0: beta, 1: beta - pi][0: at PA, 1: at PB]
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
    const R den = out ? Ra + a : rho2, num = out ? R(1.0) : Ra - a;
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

// Strain of unit slip n, strike, dip (TDCS xx, yy, zz, xy, xz, yz) and the
// displacement (its solid-angle part included) of frame f at TDCS (x, y, z).
// K8 = 1 / (8 pi (1 - nu)).  In the segment's own axes (n = TD normal,
// m = t x n in the plane, t along the side) the offset is (x, e, 0), the
// Hessian of V is H, and a unit Burgers vector b gives
//   strain -1/(4 pi) sym(b w) K + (1/(4 pi) - 2 K8) sym((b x t) grad V) - K8 (b.w) H
//   displacement 1/(4 pi) (b x t) V - K8 ((b x t) V + (b.w) grad V)
// with w = (-e, x, 0) and grad V = (-x K, -e K, T).
template <bool STRAIN, bool DISP, typename R>
CAD_HD void td_unit(const FrameT<R>& f, R x, R y, R z, R K8, R E[3][6], R U[3][3])
{
    const R k1 = R(kInv4Pi), ka = k1 - R(2.0) * K8;
    const R h = R(-1.0) * K8;   // (ka - k1) / 2
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
        // solid angle of the triangle seen from the point
        const R one = -x * ((dy[1] - dy[0]) * (dz[2] - dz[0]) - (dz[1] - dz[0]) * (dy[2] - dy[0]));
        const R ab = x2 + dy[0] * dy[1] + dz[0] * dz[1];
        const R ac = x2 + dy[0] * dy[2] + dz[0] * dz[2];
        const R bc = x2 + dy[1] * dy[2] + dz[1] * dz[2];
        const R two = Rv[0] * Rv[1] * Rv[2] + ab * Rv[2] + ac * Rv[1] + bc * Rv[0];
        const R Fi = R(-2.0) * k1 * cad_atan2(one, two);
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
            const R Hnn = x2 * g.I - g.K, Hmm = e2 * g.I - g.K;
            const R Htt = -(Hnn + Hmm);
            const R hT = R(0.5) * ka * g.T;
            // b = n
            const R nnn = e * (k1 * g.K + K8 * Hnn), nmm = e * (ka * g.K + K8 * Hmm), ntt = K8 * e * Htt;
            const R nnm = x * (h * g.K + K8 * e2 * g.I), nmt = -hT - K8 * e2 * g.Q, nnt = -K8 * e * x * g.Q;
            // b = m
            const R mmm = x * (-k1 * g.K - K8 * Hmm), mnn = x * (-ka * g.K - K8 * Hnn), mtt = -K8 * x * Htt;
            const R mnm = -e * (h * g.K + K8 * x2 * g.I), mnt = hT + K8 * x2 * g.Q, mmt = K8 * x * e * g.Q;
            // b = t: only nt and mt
            const R tnt = R(0.5) * k1 * g.K * e, tmt = R(-0.5) * k1 * g.K * x;
            const R yy = ty * ty, zz = tz * tz, yz = ty * tz, dd = zz - yy;
            E[0][0] += nnn;
            E[0][1] += nmm * zz + ntt * yy + R(2.0) * nmt * yz;
            E[0][2] += nmm * yy + ntt * zz - R(2.0) * nmt * yz;
            E[0][3] += nnm * tz + nnt * ty;
            E[0][4] += nnt * tz - nnm * ty;
            E[0][5] += (ntt - nmm) * yz + nmt * dd;
            // b = m and b = t in TDCS, then unit strike = (tz m + ty t), unit dip = (-ty m + tz t)
            const R r1 = mmm * zz + mtt * yy + R(2.0) * mmt * yz, r2 = mmm * yy + mtt * zz - R(2.0) * mmt * yz;
            const R r3 = mnm * tz + mnt * ty, r4 = mnt * tz - mnm * ty, r5 = (mtt - mmm) * yz + mmt * dd;
            const R q1 = R(2.0) * tmt * yz, q3 = tnt * ty, q4 = tnt * tz, q5 = tmt * dd;
            E[1][0] += tz * mnn;
            E[1][1] += tz * r1 + ty * q1;
            E[1][2] += tz * r2 - ty * q1;
            E[1][3] += tz * r3 + ty * q3;
            E[1][4] += tz * r4 + ty * q4;
            E[1][5] += tz * r5 + ty * q5;
            E[2][0] += -ty * mnn;
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
// Observation point -> ADCS of a side, relative to PA.
template <typename R>
CAD_HD void to_adcs(const FscSideT<R>& s, double X, double Y, double Z, R& x, R& y, R& z)
{
    R dX, dY, dZ;
    rel_origin(s.PA, s.PAlo, X, Y, Z, dX, dY, dZ);
    x = add_rn(add_rn(mul_rn(s.ey1[0], dX), mul_rn(s.ey2[0], dY)), mul_rn(s.ey3[0], dZ));
    y = add_rn(add_rn(mul_rn(s.ey1[1], dX), mul_rn(s.ey2[1], dY)), mul_rn(s.ey3[1], dZ));
    z = add_rn(add_rn(mul_rn(s.ey1[2], dX), mul_rn(s.ey2[2], dY)), mul_rn(s.ey3[2], dZ));
}

// The FP64 free-surface strain groups are called out of line: each then gets
// the whole register file, which spills far less than one inlined body (the
// FP32 groups fit inline).
#ifdef __CUDACC__
#define CAD_OUTLINE static __host__ __device__ __noinline__
#else
#define CAD_OUTLINE static inline
#endif
CAD_OUTLINE void fsc_strain_g0_f64(const ang_dis_strain_fsc_k<double>& k, double y1, double y2, double y3, double* v)
{
    ang_dis_strain_fsc_g0(k, y1, y2, y3, v);
}
CAD_OUTLINE void fsc_strain_g1_f64(const ang_dis_strain_fsc_k<double>& k, double y1, double y2, double y3, double* v)
{
    ang_dis_strain_fsc_g1(k, y1, y2, y3, v);
}
CAD_OUTLINE void fsc_strain_g2_f64(const ang_dis_strain_fsc_k<double>& k, double y1, double y2, double y3, double* v)
{
    ang_dis_strain_fsc_g2(k, y1, y2, y3, v);
}

template <typename R>
CAD_HD void fsc_strain_eval(const ang_dis_strain_fsc_k<R>& k, R y1, R y2, R y3, R v[18])
{
    if constexpr (sizeof(R) == sizeof(double)) {
        fsc_strain_g0_f64(k, y1, y2, y3, v);
        fsc_strain_g1_f64(k, y1, y2, y3, v + 6);
        fsc_strain_g2_f64(k, y1, y2, y3, v + 12);
    } else {
        ang_dis_strain_fsc_g0(k, y1, y2, y3, v);
        ang_dis_strain_fsc_g1(k, y1, y2, y3, v + 6);
        ang_dis_strain_fsc_g2(k, y1, y2, y3, v + 12);
    }
}

// One side's harmonic correction to the strain, added into E (EFCS).
template <typename R>
CAD_HD void fsc_strain(const FscSideT<R>& s, double X, double Y, double Z, R Dss, R Dds, R Dn, R E[3][6])
{
    R x, y, z;
    to_adcs(s, X, Y, Z, x, y, z);
    const bool flip = mul_rn(s.beta, x) >= 0.0;
    const int c = flip ? 1 : 0;
    const R f = flip ? R(-1.0) : R(1.0);
    // d = (term at PB) - (term at PA), formed before any slip product: far
    // from the side the two terms nearly cancel, and differencing them first
    // keeps the products from rounding the two halves differently.
    R d[18];
    fsc_strain_eval(s.ks[c][0], f * x, f * y, z, d);
#pragma unroll
    for (int q = 0; q < 18; ++q) d[q] = -d[q];
    {
        R v[18];
        fsc_strain_eval(s.ks[c][1], f * (x - s.y1B), f * (y - s.y2B), z - s.y3B, v);
#pragma unroll
        for (int q = 0; q < 18; ++q) d[q] += v[q];
    }
    R T[3][6];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        // configuration flip negates the first two ADCS slip components and
        // the 13 / 23 strain components
        const R c0 = f * s.cs[m][0], c1 = f * s.cs[m][1], c2 = s.cs[m][2];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const R fk = (k >= 4) ? f : R(1.0);
            const R h = (k >= 3) ? R(0.5) : R(1.0);
            T[m][k] = h * fk * (c0 * d[k] + c1 * d[6 + k] + c2 * d[12 + k]);
        }
    }
    const R AFlip[9] = {s.ey1[0], s.ey1[1], s.ey1[2], s.ey2[0], s.ey2[1], s.ey2[2], s.ey3[0], s.ey3[1], s.ey3[2]};
    const R slip[3] = {Dn, Dss, Dds};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        tensor_rot(T[m], AFlip);
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] += T[m][k];
    }
}

// The same correction as a linear map of the side's Burgers vector: G[j] is
// the EFCS strain of a unit Burgers vector along EFCS axis j.  A side shared
// by two triangles is traversed in opposite directions, and the reversed
// side's map is the negative of this one (the two dislocation segments
// cancel), so one evaluation per mesh edge serves both triangles.
template <typename R>
CAD_HD void fsc_strain_map(const FscSideT<R>& s, double X, double Y, double Z, R G[3][6])
{
    R x, y, z;
    to_adcs(s, X, Y, Z, x, y, z);
    const bool flip = mul_rn(s.beta, x) >= 0.0;
    const int c = flip ? 1 : 0;
    const R f = flip ? R(-1.0) : R(1.0);
    R d[18];
    fsc_strain_eval(s.ks[c][0], f * x, f * y, z, d);
#pragma unroll
    for (int q = 0; q < 18; ++q) d[q] = -d[q];
    {
        R v[18];
        fsc_strain_eval(s.ks[c][1], f * (x - s.y1B), f * (y - s.y2B), z - s.y3B, v);
#pragma unroll
        for (int q = 0; q < 18; ++q) d[q] += v[q];
    }
    const R AFlip[9] = {s.ey1[0], s.ey1[1], s.ey1[2], s.ey2[0], s.ey2[1], s.ey2[2], s.ey3[0], s.ey3[1], s.ey3[2]};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        // ADCS slip components of a unit Burgers vector along EFCS axis j (as
        // build_side forms them: the j-th frame vector ey(j+1))
        const R c0 = f * AFlip[3 * j], c1 = f * AFlip[3 * j + 1], c2 = AFlip[3 * j + 2];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const R fk = (k >= 4) ? f : R(1.0);
            const R h = (k >= 3) ? R(0.5) : R(1.0);
            G[j][k] = h * fk * (c0 * d[k] + c1 * d[6 + k] + c2 * d[12 + k]);
        }
        tensor_rot(G[j], AFlip);
    }
}

// E[m] += sign * (the map G applied to the EFCS Burgers vector of unit mode m
// of the triangle with frame `real`), for the modes with non-zero slip.
template <typename R>
CAD_HD void fsc_apply_map(const R G[3][6], R sign, const FrameT<R>& real, R Dss, R Dds, R Dn, R E[3][6])
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

// One side's harmonic correction to the displacement, added into U (EFCS).
template <typename R>
CAD_HD void fsc_disp(const FscSideT<R>& s, double X, double Y, double Z, R Dss, R Dds, R Dn, R U[3][3])
{
    R x, y, z;
    to_adcs(s, X, Y, Z, x, y, z);
    const int c = mul_rn(s.beta, x) >= 0.0 ? 1 : 0;
    R uA[9], uB[9];
    ang_dis_disp_fsc(s.kd[c][0], x, y, z, uA);
    ang_dis_disp_fsc(s.kd[c][1], x - s.y1B, y - s.y2B, z - s.y3B, uB);
    const R slip[3] = {Dn, Dss, Dds};
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(slip[m] != 0.0)) continue;
        R u[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            u[d] = s.cd[m][0] * (uB[3 * d] - uA[3 * d]) + s.cd[m][1] * (uB[3 * d + 1] - uA[3 * d + 1]) +
                   s.cd[m][2] * (uB[3 * d + 2] - uA[3 * d + 2]);
        // ADCS -> EFCS: rows (ey1, ey2, ey3) as in the reference's VxR, VyR, VzR
        U[m][0] += s.ey1[0] * u[0] + s.ey1[1] * u[1] + s.ey1[2] * u[2];
        U[m][1] += s.ey2[0] * u[0] + s.ey2[1] * u[1] + s.ey2[2] * u[2];
        U[m][2] += s.ey3[0] * u[0] + s.ey3[1] * u[1] + s.ey3[2] * u[2];
    }
}

// The free-surface displacement of side s at (X, Y, Z) for a unit Burgers
// vector along EFCS axis j, without the factor 1 / (4 pi (1 - nu)):
// Gu[j][c] = sum_d ey_c[d] sum_g ey_j[g] (uB - uA)[3 d + g] (fsc_disp with
// cs = ey_j).  As for the strain map, the reversed side's map is the
// negative of this one.
template <typename R>
CAD_HD void fsc_disp_map(const FscSideT<R>& s, double X, double Y, double Z, R Gu[3][3])
{
    R x, y, z;
    to_adcs(s, X, Y, Z, x, y, z);
    const int c = mul_rn(s.beta, x) >= 0.0 ? 1 : 0;
    R uA[9], uB[9];
    ang_dis_disp_fsc(s.kd[c][0], x, y, z, uA);
    ang_dis_disp_fsc(s.kd[c][1], x - s.y1B, y - s.y2B, z - s.y3B, uB);
    const R* ey[3] = {s.ey1, s.ey2, s.ey3};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        R u[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            u[d] = ey[j][0] * (uB[3 * d] - uA[3 * d]) + ey[j][1] * (uB[3 * d + 1] - uA[3 * d + 1]) +
                   ey[j][2] * (uB[3 * d + 2] - uA[3 * d + 2]);
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) Gu[j][cc] = ey[cc][0] * u[0] + ey[cc][1] * u[1] + ey[cc][2] * u[2];
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

// The geometry of side PA -> PB (frame, beta test, closed-form constants);
// its slip coefficients cs, cd are left zero.
CAD_HD void build_side_geom(const double PA[3], const double PB[3], double nu, FscSide& s)
{
    for (int m = 0; m < 3; ++m)
        for (int g = 0; g < 3; ++g) s.cs[m][g] = s.cd[m][g] = 0.0;
    const double S[3] = {sub_rn(PB[0], PA[0]), sub_rn(PB[1], PA[1]), sub_rn(PB[2], PA[2])};
    const double Sv = norm3_rn(S[0], S[1], S[2]);
    const double beta = acos(-S[2] / Sv);
    s.beta = beta;
    s.skip = ((fabs(beta) < DBL_EPSILON) || (fabs(M_PI - beta) < DBL_EPSILON) || (fabs(1.0 / tan(beta)) > 5e3)) ? 1.0 : 0.0;
    for (int i = 0; i < 3; ++i) { s.PA[i] = PA[i]; s.PAlo[i] = 0.0; }
    if (s.skip != 0.0) return;
    const double n1 = norm3_rn(S[0], S[1], 0.0);
    const double e1[3] = {S[0] / n1, S[1] / n1, 0.0 / n1};
    const double e3[3] = {-0.0, -0.0, -1.0};
    double e2[3];
    cross3_rn(e3, e1, e2);
    for (int i = 0; i < 3; ++i) { s.ey1[i] = e1[i]; s.ey2[i] = e2[i]; s.ey3[i] = e3[i]; }
    s.y1B = add_rn(add_rn(mul_rn(e1[0], S[0]), mul_rn(e2[0], S[1])), mul_rn(e3[0], S[2]));
    s.y2B = add_rn(add_rn(mul_rn(e1[1], S[0]), mul_rn(e2[1], S[1])), mul_rn(e3[1], S[2]));
    s.y3B = add_rn(add_rn(mul_rn(e1[2], S[0]), mul_rn(e2[2], S[1])), mul_rn(e3[2], S[2]));
    const double a_end[2] = {-PA[2], -PB[2]};
    const double pibs = M_PI - beta, pibd = -M_PI + beta;
    for (int e = 0; e < 2; ++e) {
        ang_dis_strain_fsc_setup(cos(beta), sin(beta), 1.0 / tan(beta), nu, a_end[e], s.ks[0][e]);
        ang_dis_strain_fsc_setup(cos(pibs), sin(pibs), 1.0 / tan(pibs), nu, a_end[e], s.ks[1][e]);
        ang_dis_disp_fsc_setup(cos(beta), sin(beta), 1.0 / tan(beta), 1.0 / tan(beta / 2.0), nu, a_end[e],
                               s.kd[0][e]);
        ang_dis_disp_fsc_setup(cos(pibd), sin(pibd), 1.0 / tan(pibd), 1.0 / tan(pibd / 2.0), nu, a_end[e],
                               s.kd[1][e]);
    }
}

CAD_HD void build_side(const double PA[3], const double PB[3], const Frame& real, double Dss, double Dds,
                       double Dn, double nu, FscSide& s)
{
    build_side_geom(PA, PB, nu, s);
    if (s.skip != 0.0) return;
    // unit-mode slip vectors: TDCS (n, s, d) -> EFCS -> ADCS
    const double slip[3] = {Dn, Dss, Dds};
    const double* axes[3] = {real.Vn, real.Vs, real.Vd};
    for (int m = 0; m < 3; ++m) {
        double w[3];
        for (int i = 0; i < 3; ++i) w[i] = mul_rn(axes[m][i], slip[m]);
        for (int g = 0; g < 3; ++g) {
            s.cs[m][g] = add_rn(add_rn(mul_rn(s.ey1[g], w[0]), mul_rn(s.ey2[g], w[1])), mul_rn(s.ey3[g], w[2]));
            s.cd[m][g] = s.cs[m][g] / 4.0 / M_PI / sub_rn(1.0, nu);
        }
    }
}

// Side PA -> PB carrying the net Burgers vector B (EFCS) of every triangle side
// on that mesh edge, as unit mode 0 (evaluate with Dn = 1, Dss = Dds = 0).  The
// slip coefficients follow build_side's for w = B.
CAD_HD void build_side_burgers(const double PA[3], const double PB[3], const double B[3], double nu, FscSide& s)
{
    build_side_geom(PA, PB, nu, s);
    if (s.skip != 0.0) return;
    for (int g = 0; g < 3; ++g) {
        s.cs[0][g] = add_rn(add_rn(mul_rn(s.ey1[g], B[0]), mul_rn(s.ey2[g], B[1])), mul_rn(s.ey3[g], B[2]));
        s.cd[0][g] = s.cs[0][g] / 4.0 / M_PI / sub_rn(1.0, nu);
    }
}

// ------------------------------------------------------------ pair drivers
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

// Half-space strain with the free-surface corrections of the triangle's sides
// read from per-edge maps (fsc_strain_map): entry (edge e, value q) of this
// observation point at G[e * ge + q * gq]; code[sd] = +-(e + 1) for side sd
// traversed along / against edge e's direction, 0 for no correction.
CAD_HD void pair_strain_edges(const TriDev& t, double X, double Y, double Z, const double* G, int64_t gq, int64_t ge,
                              const int* code, double E[3][6])
{
#pragma unroll
    for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int k = 0; k < 6; ++k) E[m][k] = 0.0;
    strain_fs<false>(t.real, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
#pragma unroll 1
    for (int sd = 0; sd < 3; ++sd) {
        const int c = code[sd];
        if (c == 0) continue;
        const int64_t e = (int64_t)(c > 0 ? c : -c) - 1;
        double Gm[3][6];
#pragma unroll
        for (int q = 0; q < 18; ++q) Gm[q / 6][q % 6] = G[e * ge + q * gq];
        fsc_apply_map(Gm, c > 0 ? 1.0 : -1.0, t.real, t.Dss, t.Dds, t.Dn, E);
    }
    strain_fs<true>(t.image, X, Y, Z, t.Dss, t.Dds, t.Dn, t.K8, E);
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

CAD_HD void build_triangle(const double a[3], const double b[3], const double c[3], double Dss, double Dds,
                           double Dn, double nu, bool hs, TriDev& t)
{
    t.Dss = Dss;
    t.Dds = Dds;
    t.Dn = Dn;
    t.K8 = 1.0 / (8.0 * M_PI * (1.0 - nu));
    build_frame(a, b, c, t.real);
    if (!hs) return;
    const double ai[3] = {a[0], a[1], -a[2]}, bi[3] = {b[0], b[1], -b[2]}, ci[3] = {c[0], c[1], -c[2]};
    build_frame(ai, bi, ci, t.image);
    build_side(a, b, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[0]);
    build_side(b, c, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[1]);
    build_side(c, a, t.real, t.Dss, t.Dds, t.Dn, nu, t.side[2]);
}

}  // namespace cad
