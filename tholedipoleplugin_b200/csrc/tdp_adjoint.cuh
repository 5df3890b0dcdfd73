// tdp_adjoint.cuh -- per-pair reverse-mode building blocks of the
// TholeDipoleForce evaluation (reference semantics, FP64), shared by the box
// adjoint (tdp_adjoint.cu) and the batched-cluster adjoint (tdp_batch.cu).
// See tdp_adjoint.cu for the chain they differentiate.
#pragma once

#include "tdp_frames.cuh"
#include "tdp_kernels.cuh"

#include <math.h>

namespace tdp {
namespace adj {

struct Dual {
    double v, d;
};
__device__ __forceinline__ Dual mk(double v, double d = 0.0) { return {v, d}; }
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator-(Dual a) { return {-a.v, -a.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return {a.v * b.v, a.v * b.d + a.d * b.v}; }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    double iv = 1.0 / b.v;
    return {a.v * iv, (a.d - a.v * iv * b.d) * iv};
}
__device__ __forceinline__ Dual operator+(Dual a, double b) { return {a.v + b, a.d}; }
__device__ __forceinline__ Dual operator+(double a, Dual b) { return {a + b.v, b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, double b) { return {a.v - b, a.d}; }
__device__ __forceinline__ Dual operator-(double a, Dual b) { return {a - b.v, -b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, double b) { return {a.v * b, a.d * b}; }
__device__ __forceinline__ Dual operator*(double a, Dual b) { return {a * b.v, a * b.d}; }
__device__ __forceinline__ Dual& operator+=(Dual& a, Dual b) { return a = a + b; }
__device__ __forceinline__ Dual& operator-=(Dual& a, Dual b) { return a = a - b; }
__device__ __forceinline__ Dual dexp(Dual a) {
    double e = exp(a.v);
    return {e, e * a.d};
}
__device__ __forceinline__ double dexp(double a) { return exp(a); }
__device__ __forceinline__ double val(double a) { return a; }
__device__ __forceinline__ double val(Dual a) { return a.v; }
__device__ __forceinline__ double der(double) { return 0.0; }
__device__ __forceinline__ double der(Dual a) { return a.d; }
// min(t_i, t_j) of the damping (RTDF.cpp:206, :662).  It has a kink where the
// factors are equal; there the symmetric subgradient is used (each side gets
// half), which is what a central difference sees and which sums to the exact
// derivative when both factors move together.
__device__ __forceinline__ double tmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ Dual tmin(Dual a, Dual b) {
    if (a.v < b.v) return a;
    if (b.v < a.v) return b;
    return {a.v, 0.5 * (a.d + b.d)};
}
template <class T> __device__ __forceinline__ T cst(double v);
template <> __device__ __forceinline__ double cst<double>(double v) { return v; }
template <> __device__ __forceinline__ Dual cst<Dual>(double v) { return mk(v); }

template <class T>
struct V3T {
    T x, y, z;
};
typedef V3T<double> V3;
__device__ __forceinline__ V3 ld(const double* p) { return {p[0], p[1], p[2]}; }

// Thole factors of the pair energy routine (RTDF.cpp:204-220).
template <class T>
__device__ __forceinline__ void energy_damping(double r, double r2, double damp_r2, T tI, T tK, T& tc, T& td0, T& td1,
                                               T& dtc, T& dtd0, T& dtd1) {
    tc = td0 = td1 = dtc = dtd0 = dtd1 = cst<T>(1.0);
    if (r2 < damp_r2) {
        T dmp = tI * tK;
        if (fabs(val(dmp)) > 1.0e-5) {
            T a = tmin(tI, tK);
            T u = cst<T>(r) / dmp;
            T au3 = a * u * u * u;
            T e = dexp(-au3);
            tc = 1.0 - e;
            td0 = 1.0 - e * (1.0 + 1.5 * au3);
            td1 = 1.0 - e;
            dtc = 1.0 - e * (1.0 + 1.5 * au3);
            dtd0 = 1.0 - e * (1.0 + au3 + 1.5 * au3 * au3);
            dtd1 = 1.0 - e * (1.0 + au3);
        }
    }
}

// Damped 1/r^3 and 3/r^5 of getAndScaleInverseRs (RTDF.cpp:646-676).
template <class T>
__device__ __forceinline__ void field_damping(double r, double r2, double damp_r2, T ti, T tj, T& rr3, T& rr5) {
    double rI = 1.0 / r, r2I = rI * rI;
    rr3 = cst<T>(rI * r2I);
    rr5 = cst<T>(3.0 * rI * r2I * r2I);
    if (r2 < damp_r2) {
        T dmp = ti * tj;
        if (val(dmp) != 0.0) {
            T pg = tmin(ti, tj);
            T ratio = cst<T>(r) / dmp;
            ratio = ratio * ratio * ratio;
            T damp = -pg * ratio;
            if (val(damp) > -50.0) {
                T e = dexp(damp);
                rr3 = rr3 * (1.0 - e);
                rr5 = rr5 * (1.0 - (1.0 - damp) * e);
            }
        }
    }
}

// One pair of calculateElectrostaticPairIxn in its canonical orientation
// (I lower index, d = p_K - p_I), contracted with the cotangents:
//   l = gE*energy + cf.qf + ctI.qtI + ctK.qtJ
// where cf = FR^T (gF_K - gF_I), ctI = FR^T gT_I, ctK = FR^T gT_K are the
// force/torque cotangents brought into the QI frame.  Same operations and
// frame convention as pair_energy (tdp_pairs.cuh).
template <class T>
__device__ T pair_loss(double dx, double dy, double dz, bool yzd, T qI, const T* mI, const T* uIl, T tI, T qK,
                       const T* mK, const T* uKl, T tK, double mS, double iS, double damp_r2, double rv4p,
                       double rv4f, bool mutual, double gE, V3 gFI, V3 gFK, V3 gTI, V3 gTK) {
    double r2 = dx * dx + dy * dy + dz * dz;
    double r = sqrt(r2);
    double rinv = 1.0 / r;
    double zx = dx * rinv, zy = dy * rinv, zz = dz * rinv;
    double xx = zx, xy = zy, xz = zz;
    if (yzd) xx += 1.0;
    else xy += 1.0;
    double dt = zx * xx + zy * xy + zz * xz;
    xx -= zx * dt;
    xy -= zy * dt;
    xz -= zz * dt;
    double xn = sqrt(xx * xx + xy * xy + xz * xz);
    if (xn > 0.0) {
        xx /= xn;
        xy /= xn;
        xz /= xn;
    }
    double yx = zy * xz - zz * xy, yy = zz * xx - zx * xz, yz = zx * xy - zy * xx;
    // Force rotation rows (Y.y, Z.y, X.y), (Y.z, Z.z, X.z), (Y.x, Z.x, X.x).
    double FR[3][3] = {{yy, zy, xy}, {yz, zz, xz}, {yx, zx, xx}};
    double gd[3] = {gFK.x - gFI.x, gFK.y - gFI.y, gFK.z - gFI.z};
    double gti[3] = {gTI.x, gTI.y, gTI.z}, gtk[3] = {gTK.x, gTK.y, gTK.z};
    double cf[3], cti[3], ctk[3];
    for (int b = 0; b < 3; b++) {
        cf[b] = FR[0][b] * gd[0] + FR[1][b] * gd[1] + FR[2][b] * gd[2];
        cti[b] = FR[0][b] * gti[0] + FR[1][b] * gti[1] + FR[2][b] * gti[2];
        ctk[b] = FR[0][b] * gtk[0] + FR[1][b] * gtk[1] + FR[2][b] * gtk[2];
    }
    T uI0 = xx * uIl[0] + xy * uIl[1] + xz * uIl[2];
    T uI1 = yx * uIl[0] + yy * uIl[1] + yz * uIl[2];
    T uI2 = zx * uIl[0] + zy * uIl[1] + zz * uIl[2];
    T uJ0 = xx * uKl[0] + xy * uKl[1] + xz * uKl[2];
    T uJ1 = yx * uKl[0] + yy * uKl[1] + yz * uKl[2];
    T uJ2 = zx * uKl[0] + zy * uKl[1] + zz * uKl[2];
    T QI0 = qI, QJ0 = qK;
    T QI1 = xx * mI[0] + xy * mI[1] + xz * mI[2];
    T QI2 = yx * mI[0] + yy * mI[1] + yz * mI[2];
    T QI3 = zx * mI[0] + zy * mI[1] + zz * mI[2];
    T QJ1 = xx * mK[0] + xy * mK[1] + xz * mK[2];
    T QJ2 = yx * mK[0] + yy * mK[1] + yz * mK[2];
    T QJ3 = zx * mK[0] + zy * mK[1] + zz * mK[2];
    double rv1 = rinv, rv2 = rv1 * rinv, rv3 = rv2 * rinv;
    double rv4 = rv4p * (rv3 * rinv) + rv4f;
    T tc, td0, td1, dtc, dtd0, dtd1;
    energy_damping<T>(r, r2, damp_r2, tI, tK, tc, td0, td1, dtc, dtd0, dtd1);

    double eP = rv1 * mS, dP = -0.5 * mS * rv2;
    T Vij0 = eP * QJ0, Vji0 = eP * QI0, VijR0 = dP * QJ0, VjiR0 = dP * QI0;
    eP = rv2 * mS;
    T eU = (rv2 * iS) * tc;
    dP = -rv3 * mS;
    T dU = (-2.0 * rv3 * iS) * dtc;
    Vij0 = Vij0 - (eP * QJ1 + eU * uJ0);
    T Vji1 = -(eP * QI0);
    VijR0 = VijR0 - (dP * QJ1 + dU * uJ0);
    T VjiR1 = -(dP * QI0);
    T Vjid0 = -(eU * QI0);
    T Vij1 = eP * QJ0;
    Vji0 = Vji0 + eP * QI1 + eU * uI0;
    T VijR1 = dP * QJ0;
    VjiR0 = VjiR0 + dP * QI1 + dU * uI0;
    T Vijd0 = eU * QJ0;
    eP = -2.0 * rv3 * mS;
    eU = (-2.0 * rv3 * iS) * td0;
    dP = 3.0 * rv4 * mS;
    dU = (6.0 * rv4 * iS) * dtd0;
    Vij1 = Vij1 + eP * QJ1 + eU * uJ0;
    Vji1 = Vji1 + eP * QI1 + eU * uI0;
    VijR1 = VijR1 + dP * QJ1 + dU * uJ0;
    VjiR1 = VjiR1 + dP * QI1 + dU * uI0;
    Vijd0 = Vijd0 + eU * QJ1;
    Vjid0 = Vjid0 + eU * QI1;
    eP = rv3 * mS;
    eU = (rv3 * iS) * td1;
    dP = -1.5 * rv4 * mS;
    dU = (-3.0 * rv4 * iS) * dtd1;
    T Vij2 = eP * QJ2 + eU * uJ1, Vji2 = eP * QI2 + eU * uI1;
    T VijR2 = dP * QJ2 + dU * uJ1, VjiR2 = dP * QI2 + dU * uI1;
    T Vijd1 = eU * QJ2, Vjid1 = eU * QI2;
    T Vij3 = eP * QJ3 + eU * uJ2, Vji3 = eP * QI3 + eU * uI2;
    T VijR3 = dP * QJ3 + dU * uJ2, VjiR3 = dP * QI3 + dU * uI2;
    T Vijd2 = eU * QJ3, Vjid2 = eU * QI3;

    T energy = 0.5 * (QI0 * Vij0 + QJ0 * Vji0) + 0.5 * (QI1 * Vij1 + QJ1 * Vji1) + 0.5 * (QI2 * Vij2 + QJ2 * Vji2) +
               0.5 * (QI3 * Vij3 + QJ3 * Vji3);
    T fIZ = QI0 * VijR0 + QI1 * VijR1 + QI2 * VijR2 + QI3 * VijR3;
    T fJZ = QJ0 * VjiR0 + QJ1 * VjiR1 + QJ2 * VjiR2 + QJ3 * VjiR3;
    T EIX = QI3 * Vij1 - QI1 * Vij3, EIY = QI1 * Vij2 - QI2 * Vij1, EIZ = QI2 * Vij3 - QI3 * Vij2;
    T EJX = QJ3 * Vji1 - QJ1 * Vji3, EJY = QJ1 * Vji2 - QJ2 * Vji1, EJZ = QJ2 * Vji3 - QJ3 * Vji2;
    T iEIX = uI2 * Vijd0 - uI0 * Vijd2, iEJX = uJ2 * Vjid0 - uJ0 * Vjid2;
    T iEIY = uI0 * Vijd1 - uI1 * Vijd0, iEJY = uJ0 * Vjid1 - uJ1 * Vjid0;
    if (mutual) {
        T eC = (-4.0 * rv3 * iS) * td0;
        T dC = (6.0 * rv4 * iS) * dtd0;
        iEIX += eC * uI2 * uJ0;
        iEJX += eC * uJ2 * uI0;
        iEIY -= eC * uI1 * uJ0;
        iEJY -= eC * uJ1 * uI0;
        fIZ += dC * uI0 * uJ0;
        fJZ += dC * uJ0 * uI0;
        eC = (2.0 * rv3 * iS) * td1;
        dC = (-3.0 * rv4 * iS) * dtd1;
        iEIX -= eC * uI0 * uJ2;
        iEJX -= eC * uJ0 * uI2;
        iEIY += eC * uI0 * uJ1;
        iEJY += eC * uJ0 * uI1;
        fIZ += dC * (uI1 * uJ1 + uI2 * uJ2);
        fJZ += dC * (uJ1 * uI1 + uJ2 * uI2);
    }
    T qf0 = rinv * (EIY + EJY + iEIY + iEJY);
    T qf1 = -rinv * (EIX + EJX + iEIX + iEJX);
    T qf2 = -(fJZ + fIZ);
    T l = gE * energy + cf[0] * qf0 + cf[1] * qf1 + cf[2] * qf2;
    l = l - (cti[0] * EIX + cti[1] * EIY + cti[2] * EIZ) - (ctk[0] * EJX + ctk[1] * EJY + ctk[2] * EJZ);
    return l;
}

__device__ __forceinline__ V3 min_image(const PairParams& P, V3 d) {
    if (!P.periodic) return d;
    const V3 f = {round_fold(d.x, P.box[0], P.inv_box[0]), round_fold(d.y, P.box[1], P.inv_box[1]),
                  round_fold(d.z, P.box[2], P.inv_box[2])};
    if (!near_tie(f.x, __double2hiint(P.half_box_tol[0])) && !near_tie(f.y, __double2hiint(P.half_box_tol[1])) &&
        !near_tie(f.z, __double2hiint(P.half_box_tol[2])))
        return f;
    return {fold_d(d.x, P.box[0], P.inv_box[0]), fold_d(d.y, P.box[1], P.inv_box[1]),
            fold_d(d.z, P.box[2], P.inv_box[2])};
}

// |d|^2 with its roundings spelled out: passes that divide the pairs between
// them by r^2 < damp_r2 have to agree to the last bit.
__device__ __forceinline__ double norm2(V3 d) { return fma(d.z, d.z, fma(d.y, d.y, d.x * d.x)); }

struct AtomData {
    const double* pos;     // n*3
    const double* q;       // n
    const double* lab;     // n*3
    const double* mu;      // n*3
    const double* thole;   // n
    const double2* yz;     // raw (y, z) for the QI frame test (NULL: taken from pos)
};

template <class T>
__device__ __forceinline__ V3T<T> cross3(V3T<T> a, V3T<T> b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <class T>
__device__ __forceinline__ T dot3(V3T<T> a, V3T<T> b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
template <class T>
__device__ __forceinline__ V3T<T> axpy(T a, V3T<T> x, V3T<T> y) { return {a * x.x + y.x, a * x.y + y.y, a * x.z + y.z}; }
template <class T>
__device__ __forceinline__ V3T<T> scl(T a, V3T<T> x) { return {a * x.x, a * x.y, a * x.z}; }
template <class T>
__device__ __forceinline__ V3T<T> add3(V3T<T> a, V3T<T> b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class T>
__device__ __forceinline__ V3T<T> sub3v(V3T<T> a, V3T<T> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
// Transpose of the permuted back rotation: a . perm(v) = permT(a) . v with
// perm(v) = (v_y, v_z, v_x).
template <class T>
__device__ __forceinline__ V3T<T> permT(V3T<T> a) { return {a.z, a.x, a.y}; }
// 1/sqrt(x): rsqrt in either arithmetic.
__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }

// Closed-form VJP of the pair routine with respect to one atom's (q, m_lab,
// mu_ind) and, with DAMP, its Thole factor, for rInvVec[4] = 0 and a pair off
// the x axis: the derivatives of
//   l = gE e + gF . F + gF' . F' + gT . tau + gT' . tau'
// (primed: the partner's), by reverse mode through the lab-frame form of the
// routine (the energy walk of tdp_sym.cu has the expressions).  d points from
// the atom to its partner; an atom with the higher index negates both charges
// and the force (sg = -1), as there.  With A, B, C, D the X coefficients of
// V, V', Vd, Vd', K = A m + B m' + C u + D u' and
//   f = (K.X/r + S0) X - K/r,  S0 = mS q q'/r^2 + 2 (mS c_m + iS t0 c_u)/r^3,
//   c_m = q' m_0 - q m'_0,  c_u = q' u_0 - q u'_0,
// the cotangents follow from c = sg permT(gF' - gF), t = permT(gT):
//   K~ = ((c.X) X - c)/r,  V~ = gE m/2 + m x t,  V'~ = gE m'/2 + m' x t',
//   A~ = K~.m + V~.X,  B~ = K~.m' + V'~.X,  C~ = K~.u,  D~ = K~.u',
// and the rest is the chain through A..D, c_m, c_u.  About 210 operations
// (260 with damping), where evaluating the routine with the atom's multipoles
// set to unit vectors and a dual number for the Thole factor takes about
// 4,500 (256 clusters, FP64: reverse pass 2.5 -> 1.1 ms; 12,288-atom box:
// k_pair_vjp_slow 896 -> 255 us, k_pair_vjp_fast 1927 -> 1561 us).  lam: 2
// (Mutual) or 0.  acc[0..6] += dq, dm[3], du[3], acc[7] += dt.
template <class T, bool DAMP>
__device__ __forceinline__ void pair_vjp_me(V3T<T> d, T sg, T q, V3T<T> m, V3T<T> u, T t, T qo, V3T<T> mo, V3T<T> uo,
                                            T to, T mS, T iS, T damp_r2, T lam, T gE, V3T<T> gF, V3T<T> gFo,
                                            V3T<T> gT, V3T<T> gTo, T* acc) {
    typedef V3T<T> W;
    const T rho2 = d.y * d.y + d.z * d.z, r2 = d.x * d.x + rho2;
    const T rinv = rsq(r2), xs = rinv * rsq(rho2), ndxs = -d.x * xs;
    const W X = {rho2 * xs, ndxs * d.y, ndxs * d.z};
    const T qi = sg * q, qj = sg * qo;
    const T mi0 = dot3(X, m), ui0 = dot3(X, u), mj0 = dot3(X, mo), uj0 = dot3(X, uo);
    T x = 0, e = 0, tc = 1, w = 1, t0 = 1;
    bool damped = false;
    if (DAMP && r2 < damp_r2) {
        const T dmp = t * to;
        if (fabs(dmp) > T(1.0e-5)) {
            const T v = r2 * rinv / dmp;
            damped = true;
            x = (t < to ? t : to) * v * v * v;
            e = exp(-x);
            tc = T(1) - e;
            w = T(1) - (T(1) + x) * e;
            t0 = T(1) - (T(1) + T(1.5) * x) * e;
        }
    }
    const T rv2 = rinv * rinv, rv3 = rv2 * rinv, n3 = T(-3) * rv3;
    const T sw = iS * w, sc = iS * tc, mv2 = mS * rv2, cv2 = sc * rv2;
    const T lj0 = mj0 + lam * uj0, li0 = mi0 + lam * ui0;
    const T A = mv2 * qj + n3 * (mS * mj0 + sw * uj0), C = cv2 * qj + n3 * sw * lj0;
    const W V = axpy(A, X, scl(rv3, axpy(mS, mo, scl(sc, uo))));
    const W c = scl(sg, permT(sub3v(gFo, gF))), tI = permT(gT), tK = permT(gTo);
    const T cx = dot3(c, X), hE = T(0.5) * gE;
    const W Kb = scl(rinv, sub3v(scl(cx, X), c));
    const W Ub = axpy(hE, mo, cross3(mo, tK));
    const T Bb = dot3(Kb, mo) + dot3(Ub, X), Db = dot3(Kb, uo);
    const T cmb = mS * (T(2) * rv3 * cx + hE * rv2), cub = iS * (T(2) * rv3 * t0 * cx + hE * rv2 * tc);
    const T mi0b = n3 * (mS * Bb + sw * Db) + cmb * qj, ui0b = n3 * sw * (Bb + lam * Db) + cub * qj;
    const W gm = add3(axpy(hE, V, cross3(tI, V)), axpy(A, Kb, axpy(rv3 * mS, Ub, scl(mi0b, X))));
    const W gu = axpy(C, Kb, axpy(rv3 * sc, Ub, scl(ui0b, X)));
    acc[0] += sg * (mv2 * cx * qj + mS * gE * rinv * qj - mv2 * Bb - cv2 * Db - cmb * mj0 - cub * uj0);
    acc[1] += gm.x;
    acc[2] += gm.y;
    acc[3] += gm.z;
    acc[4] += gu.x;
    acc[5] += gu.y;
    acc[6] += gu.z;
    if (DAMP && damped) {
        const W Vb = axpy(hE, m, cross3(m, tI));
        const T Ab = dot3(Kb, m) + dot3(Vb, X), Cb = dot3(Kb, u);
        const T cu = qj * ui0 - qi * uj0;
        const T tcb = rv3 * (dot3(Vb, uo) + dot3(Ub, u)) + rv2 * (hE * cu + qj * Cb - qi * Db);
        const T wb = n3 * (uj0 * Ab + ui0 * Bb + lj0 * Cb + li0 * Db);
        const T xb = iS * e * (tcb + x * wb + (T(1.5) * x - T(0.5)) * (T(2) * rv3 * cu * cx));
        // x = min(t, t') r^3 / (t t')^3; the symmetric subgradient at t = t' (tmin).
        acc[7] += xb * x / t * (t < to ? T(-2) : to < t ? T(-3) : T(-2.5));
    }
}

// The VJP of a pair on the x axis, or of one with 1/r^4 terms, by the routine
// itself: it is bilinear in the two atoms' multipoles, so each derivative is
// the routine with this atom's multipoles set to unit vectors; the Thole
// factor's takes a dual number.  Rare and out of line, so that it does not set
// its callers' registers.
static __device__ __noinline__ void visit_pair_routine(const PairParams& P, const AtomData& A, const double* g,
                                                const double* gT, double gE, bool meI, int I, int K, V3 d, bool yzd,
                                                double mS, double iS, double* acc) {
    const double rv4p = P.rinv4_power, rv4f = P.rinv4_fill;
    const double damp_r2 = P.damp_r2 == 0.0f ? 0.0 : (double)P.damp_r2;
    V3 gFI = ld(g + 3 * I), gFK = ld(g + 3 * K), gTI = ld(gT + 3 * I), gTK = ld(gT + 3 * K);
    double oq = A.q[meI ? K : I];
    double om[3] = {A.lab[3 * (meI ? K : I)], A.lab[3 * (meI ? K : I) + 1], A.lab[3 * (meI ? K : I) + 2]};
    double ou[3] = {A.mu[3 * (meI ? K : I)], A.mu[3 * (meI ? K : I) + 1], A.mu[3 * (meI ? K : I) + 2]};
    double tI = A.thole[I], tK = A.thole[K];
    for (int a = 0; a < 7; a++) {
        double bq = a == 0 ? 1.0 : 0.0;
        double bm[3] = {a == 1 ? 1.0 : 0.0, a == 2 ? 1.0 : 0.0, a == 3 ? 1.0 : 0.0};
        double bu[3] = {a == 4 ? 1.0 : 0.0, a == 5 ? 1.0 : 0.0, a == 6 ? 1.0 : 0.0};
        double l = meI ? pair_loss<double>(d.x, d.y, d.z, yzd, bq, bm, bu, tI, oq, om, ou, tK, mS, iS, damp_r2, rv4p,
                                           rv4f, P.mutual, gE, gFI, gFK, gTI, gTK)
                       : pair_loss<double>(d.x, d.y, d.z, yzd, oq, om, ou, tI, bq, bm, bu, tK, mS, iS, damp_r2, rv4p,
                                           rv4f, P.mutual, gE, gFI, gFK, gTI, gTK);
        acc[a] += l;
    }
    // Thole-factor derivative: dual number seeded on my t.
    Dual dq[2], dm[2][3], du[2][3];
    for (int s = 0; s < 2; s++) {
        int at = s == 0 ? I : K;
        dq[s] = mk(A.q[at]);
        for (int c = 0; c < 3; c++) {
            dm[s][c] = mk(A.lab[3 * at + c]);
            du[s][c] = mk(A.mu[3 * at + c]);
        }
    }
    Dual dtI = mk(tI, meI ? 1.0 : 0.0), dtK = mk(tK, meI ? 0.0 : 1.0);
    Dual l = pair_loss<Dual>(d.x, d.y, d.z, yzd, dq[0], dm[0], du[0], dtI, dq[1], dm[1], du[1], dtK, mS, iS, damp_r2,
                             rv4p, rv4f, P.mutual, gE, gFI, gFK, gTI, gTK);
    acc[7] += l.d;
}

__device__ inline void visit_pair(const PairParams& P, const AtomData& A, const double* g, const double* gT, double gE,
                           int me, int j, double mS, double iS, double* acc) {
    const bool meI = me < j;
    const int I = meI ? me : j, K = meI ? j : me;
    V3 d = min_image(P, {A.pos[3 * K] - A.pos[3 * I], A.pos[3 * K + 1] - A.pos[3 * I + 1],
                         A.pos[3 * K + 2] - A.pos[3 * I + 2]});
    bool yzd;
    if (A.yz) {
        const double2 yzI = A.yz[I], yzK = A.yz[K];
        yzd = (yzI.x != yzK.x) || (yzI.y != yzK.y);
    } else {
        yzd = (A.pos[3 * I + 1] != A.pos[3 * K + 1]) || (A.pos[3 * I + 2] != A.pos[3 * K + 2]);
    }
    const double rv4p = P.rinv4_power, rv4f = P.rinv4_fill;
    const double damp_r2 = P.damp_r2 == 0.0f ? 0.0 : (double)P.damp_r2;
    if (rv4p == 0.0 && rv4f == 0.0 && yzd && d.y * d.y + d.z * d.z >= 1.0e-12) {
        const double sg = meI ? 1.0 : -1.0;
        pair_vjp_me<double, true>({sg * d.x, sg * d.y, sg * d.z}, sg, A.q[me], ld(A.lab + 3 * me), ld(A.mu + 3 * me),
                                  A.thole[me], A.q[j], ld(A.lab + 3 * j), ld(A.mu + 3 * j), A.thole[j], mS, iS,
                                  damp_r2, P.mutual ? 2.0 : 0.0, gE, ld(g + 3 * me), ld(g + 3 * j), ld(gT + 3 * me),
                                  ld(gT + 3 * j), acc);
        return;
    }
    visit_pair_routine(P, A, g, gT, gE, meI, I, K, d, yzd, mS, iS, acc);
}

// Derivatives of the damped rr3 and rr5 (field_damping) with respect to the
// Thole factor t of one side (to: the other's), zero where that side's pairs are not damped.
__device__ __forceinline__ void field_damping_dt(double r, double rinv, double t, double to, double& d3,
                                                 double& d5) {
    d3 = d5 = 0.0;
    const double dmp = t * to;
    if (dmp == 0.0) return;
    const double v = r / dmp, x = (t < to ? t : to) * v * v * v;
    if (!(x < 50.0)) return;
    // rr3 = (1 - e^-x)/r^3, rr5 = 3 (1 - (1 + x) e^-x)/r^5, x = min(t, to) r^3/(t to)^3.
    const double xt = x / t * (t < to ? -2.0 : to < t ? -3.0 : -2.5) * exp(-x), i2 = rinv * rinv;
    d3 = xt * rinv * i2;
    d5 = 3.0 * x * xt * rinv * i2 * i2;
}

// d/dt_k of m (lambda_i . f_ik + lambda_k . f_ki), f_ik = -[d (rr3 q_k - rr5 lab_k.d) + lab_k rr3], d = p_k - p_i.
__device__ __forceinline__ double fixed_vjp_dt(const AtomData& A, V3 d, double r, V3 li, V3 lk, int k, int i, double m) {
    double d3v, d5v;
    field_damping_dt(r, 1.0 / r, A.thole[k], A.thole[i], d3v, d5v);
    const V3 mk_ = ld(A.lab + 3 * k), mi = ld(A.lab + 3 * i);
    const double lid = dot3(li, d), lkd = dot3(lk, d);
    return m * (d5v * (lid * dot3(mk_, d) + lkd * dot3(mi, d)) -
                d3v * (lid * A.q[k] + dot3(li, mk_) - lkd * A.q[i] + dot3(lk, mi)));
}

// Contribution of the pair (i, k) with M scale m to atom k's
// d/d(q_k, lab_k, t_k) of lambda . Efix (k_fixed_vjp), added to acc[5].
__device__ __forceinline__ void fixed_vjp_visit(const PairParams& P, const AtomData& A, const double* lam, int k,
                                                int i, double m, double* acc) {
    const double damp_r2 = (double)P.damp_r2;
    const V3 lk = ld(lam + 3 * k);
    V3 d = min_image(P, {A.pos[3 * k] - A.pos[3 * i], A.pos[3 * k + 1] - A.pos[3 * i + 1],
                         A.pos[3 * k + 2] - A.pos[3 * i + 2]});  // p_k - p_i
    double r2 = norm2(d), r = sqrt(r2);
    V3 li = ld(lam + 3 * i);
    double rr3, rr5;
    field_damping<double>(r, r2, damp_r2, A.thole[i], A.thole[k], rr3, rr5);
    double ldd = li.x * d.x + li.y * d.y + li.z * d.z;
    // Each term is rounded before m, so that the pair and its correction by -1 cancel exactly.
    const double a = rr5 * ldd;
    acc[0] -= m * __dmul_rn(rr3, ldd);  // d(lambda_i . f_ik)/dq_k
    acc[1] += m * __dadd_rn(a * d.x, -__dmul_rn(rr3, li.x));
    acc[2] += m * __dadd_rn(a * d.y, -__dmul_rn(rr3, li.y));
    acc[3] += m * __dadd_rn(a * d.z, -__dmul_rn(rr3, li.z));
    // t_k enters f_ik and f_ki (only within the damping range).
    if (!(r2 < damp_r2)) return;
    acc[4] += fixed_vjp_dt(A, d, r, li, lk, k, i, m);
}

// fixed_vjp_visit of a unit-scale pair within the damping range, nothing beyond.
__device__ __forceinline__ void fixed_vjp_damped(const PairParams& P, const AtomData& A, const double* lam, int k,
                                                 int i, double* acc) {
    const V3 d = min_image(P, {A.pos[3 * k] - A.pos[3 * i], A.pos[3 * k + 1] - A.pos[3 * i + 1],
                               A.pos[3 * k + 2] - A.pos[3 * i + 2]});
    if (norm2(d) < (double)P.damp_r2) fixed_vjp_visit(P, A, lam, k, i, 1.0, acc);
}

// d/dt_k of the pair (k, j) terms of lambda^T T(t) mu with I scale s
// (k_matvec_t_vjp).  Undamped pairs do not depend on t.
__device__ __forceinline__ double matvec_t_visit(const PairParams& P, const AtomData& A, const double* lam, int k,
                                                 int j, double s) {
    const double damp_r2 = (double)P.damp_r2;
    V3 d = min_image(P, {A.pos[3 * j] - A.pos[3 * k], A.pos[3 * j + 1] - A.pos[3 * k + 1],
                         A.pos[3 * j + 2] - A.pos[3 * k + 2]});
    double r2 = d.x * d.x + d.y * d.y + d.z * d.z, r = sqrt(r2);
    if (!(r2 < damp_r2)) return 0.0;
    double d3v, d5v;
    field_damping_dt(r, 1.0 / r, A.thole[k], A.thole[j], d3v, d5v);
    V3 lk = ld(lam + 3 * k), uk = ld(A.mu + 3 * k);
    V3 lj = ld(lam + 3 * j), uj = ld(A.mu + 3 * j);
    // lambda_k.(T_kj mu_j) + lambda_j.(T_jk mu_k); T_kj v = -rr3 v + rr5 (v.d) d.
    double a1 = (lk.x * d.x + lk.y * d.y + lk.z * d.z) * (uj.x * d.x + uj.y * d.y + uj.z * d.z);
    double b1 = lk.x * uj.x + lk.y * uj.y + lk.z * uj.z;
    double a2 = (lj.x * d.x + lj.y * d.y + lj.z * d.z) * (uk.x * d.x + uk.y * d.y + uk.z * d.z);
    double b2 = lj.x * uk.x + lj.y * uk.y + lj.z * uk.z;
    return s * (d5v * (a1 + a2) - d3v * (b1 + b2));
}

}  // namespace adj
}  // namespace tdp
