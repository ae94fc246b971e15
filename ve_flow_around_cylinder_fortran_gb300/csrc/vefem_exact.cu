// Exact (linearised) element Jacobian by forward-mode differentiation of the
// Gauss-point physics, in FP32 (the inexact-Newton "precision form") or FP64.
//
// At a Gauss point the weak-form term of test node i and equation e is linear
// in the test function: TERM(i,e) = sum_k c_ek(q) psi_k(i), psi = (phi, dphi/dx,
// dphi/dy), where the coefficients c (6 equations x 3) depend on the 20
// interpolated quantities q (u, v: value, x/y gradient, Laplacian; p and the
// three stress components: value, x/y gradient) and on Wi (through the
// arclength unknown).  Each unknown x(j,f) enters q linearly through chi(j) =
// (phi_j, dphi_j/dx, dphi_j/dy, Laplacian phi_j).  Hence
//     dR(i,e)/dx(j,f) = sum_gp WET sum_k psi_k(i) sum_s (dc_ek/dq_fs) chi_s(j).
// This replaces the 56 residual evaluations of the forward difference; it is
// the derivative the FD approximates (they differ by the FD truncation error).
//
// A CTA takes NE elements at a time (persistent: it walks a list of work
// items, each a run of consecutive elements of one mesh; a single mesh is the
// one-instance case):
//   1  state, geometry (from the mesh's table) and the 20 interpolants;
//   2  D[gp][d][e*3+k] = WET dc_ek/dq_d, a thread per direction, in four groups
//      of warps (velocity, stress, stress gradient, Wi).  A group's duals are
//      only the quantities that depend on its own seeds, the others plain
//      numbers (coef_tangent), and c is formed once (the physics source's
//      test_node, asked for unit test functions, does it three times with the
//      nine-node divisions of the FD's rounding).  The pressure and the
//      Laplacians enter the momentum residual linearly: no evaluation at all;
//   3  a thread per (field f, test node i, R equations): the test side
//      sum_k psi_k(i) D in registers (each is used by this thread only), then the
//      nine trial nodes; coalesced stores through shared memory.
// Bound: FP64 by its pipe, 2 lanes per clock and SM; FP32 by shared-memory
// reads in part 3 (105 reads for 240 multiply-adds with R = 6; a thread per
// equation made 52 for 40) and by latency in part 2.
// Kernel alone, SQRT form: FP32 2.5 -> 0.65 ms per 40,000 elements; residual and
// FP64 Jacobian 4,408 -> 2,046 us on 5,000 quads (e-PTT, T form), 7,176 -> 2,263
// us (Giesekus, SQRT).  FP32 error against 64 bits 7.8e-7 -> 1.0e-7: the state
// enters as differences over the element.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "vefem_dual.cuh"
#include "vefem_internal.h"
#include "vefem_physics.cuh"

namespace vefem {

__constant__ double x_bfn[9][9];

cudaError_t upload_tables_exact(const GaussTables &t, cudaStream_t s)
{
    return cudaMemcpyToSymbolAsync(x_bfn, t.bfn, sizeof(t.bfn), 0, cudaMemcpyHostToDevice, s);
}

constexpr int EX_NDIR = 21;      // 20 interpolated quantities + the arclength unknown

// direction index of quantity s (0 value, 1 d/dx, 2 d/dy, 3 Laplacian) of field f
__device__ __forceinline__ int qdir(int f, int s)
{
    return f == 0 ? s : (f == 1 ? 4 + s : 8 + 3 * (f - 2) + s);
}

template <class T>
struct __align__(4 * sizeof(T)) Chi {
    T p, x, y, l;                // phi, dphi/dx, dphi/dy, Laplacian
};

// Tangent of a value that may not depend on the seeds.
__device__ __forceinline__ float tangent(float) { return 0.0f; }
__device__ __forceinline__ double tangent(double) { return 0.0; }
template <class T> __device__ __forceinline__ T tangent(const Dual<T> &a) { return a.d; }
__device__ __forceinline__ float value(float a) { return a; }
__device__ __forceinline__ double value(double a) { return a; }
template <class T> __device__ __forceinline__ T value(const Dual<T> &a) { return a.v; }

// 1/x and 1/sqrt(x), one division (or root) for value and tangent
__device__ __forceinline__ float inv(float x) { return 1.0f / x; }
__device__ __forceinline__ double inv(double x) { return 1.0 / x; }
template <class T> __device__ __forceinline__ Dual<T> inv(const Dual<T> &a)
{
    const T r = inv(a.v);
    return Dual<T>(r, -(r * r) * a.d);
}
__device__ __forceinline__ float inv_sqrt(float x) { return 1.0f / sqrtf(x); }
__device__ __forceinline__ double inv_sqrt(double x) { return ::rsqrt(x); }
template <class T> __device__ __forceinline__ Dual<T> inv_sqrt(const Dual<T> &a)
{
    const T r = inv_sqrt(a.v);
    return Dual<T>(r, (T)-0.5 * (r * r) * (r * a.d));
}

// What the closed-form directions (pressure, Laplacians) need of a point.
template <class T>
struct MomentumFactors {
    T u1, u2;       // tlsme ReN (U1, U2): momentum residual in the momentum equations
    T tm, ts;       // in the continuity and (with the sign) the stress equations
};

// dst[e*3 + k] = w * tangent of c_ek (gauss_point and test_node of the physics
// source, coefficients of phi, dphi/dx, dphi/dy instead of nine test nodes).
// RU, RS, RG, RW: types of the velocity, stress, stress-gradient and Wi
// values, Dual where the seeds are.  The constitutive residual is symmetric
// (C21 = C12 up to rounding), and so is used once.
template <int FORM, int SPEC, class T, class RU, class RS, class RG, class RW>
__device__ __forceinline__ MomentumFactors<T>
coef_tangent(const KParams &prm, const RU U1, const RU U2, const RU GU11, const RU GU21, const RU GU12, const RU GU22,
             const RS S11, const RS S12, const RS S22, const RG X11, const RG Y11, const RG X12, const RG Y12,
             const RG X22, const RG Y22, const RW Wi, T dPx, T dPy, T lap1, T lap2, T H2, T w, const Chi<T> *chi,
             T *dst)
{
    const T be = (T)prm.BvN, Re = (T)prm.ReN, Ve = (T)prm.VeN, Df = (T)prm.DfN, dt = (T)prm.dt;
    const T om = (T)1 - be, half = (T)0.5, one = (T)1, two = (T)2, rH2 = inv(H2);
    // setFlowKinematics
    const auto tr = GU11 + GU22;
    const auto gt11 = (GU11 - GU22) * half, gt22 = -gt11;
    const auto Gd11 = gt11 + gt11, Gd12 = GU12 + GU21;
    const auto a11 = U1 * X11 + U2 * Y11, a12 = U1 * X12 + U2 * Y12, a22 = U1 * X22 + U2 * Y22;
    const auto ddG = (Gd11 * Gd11 + Gd12 * Gd12) * two;
    const auto rWi = inv(Wi);
    const auto rr = rWi * om;
    typedef decltype(U1 * S11 * X11 * Wi) R;          // depends on anything
    R f2 = R((T)0);
    R C11, C12, C22, C33 = R((T)0);
    typedef decltype(S11 * S11 * Wi) RF;
    RF fT = RF((T)0), f3 = RF((T)0);
    R P11, P12, P22, divT1, divT2;                    // stress without pressure
    RF ddT, ddC;
    const auto ddS = S11 * S11 + two * (S12 * S12) + S22 * S22;
    if constexpr (FORM == FORM_T) {
        const auto trT = S11 + S22;
        const T rom = inv(om);
        R MD = R((T)0);
        const bool fene = prm.model == FENE_CR || prm.model == FENE_P;
        const T rVe = inv(prm.model == FENE_P ? Ve : Ve - two);
        if (fene) {
            const auto k = Wi * (rom * rVe);
            MD = U1 * (k * (X11 + X22)) + U2 * (k * (Y11 + Y22));
        }
        RF f1 = RF(one);
        switch (prm.model) {
        case L_PTT:
        case M_L_PTT: fT = (Wi * trT) * (Ve * rom) + one; break;
        case E_PTT:
        case M_E_PTT: fT = exp((Wi * trT) * (Ve * rom)); break;
        case GIESEKUS: fT = RF(Wi * (Ve * rom)); f3 = fT; break;
        default: fT = (Wi * trT) * (rom * rVe) + one; break;
        }
        R term_I = R((T)0);
        if (prm.model == M_L_PTT || prm.model == M_E_PTT || prm.model == FENE_CR) f1 = fT;
        if (prm.model == GIESEKUS) {
            f2 = R(one);
        } else if (fene) {
            const R q = MD * inv(fT);
            f2 = fT - Wi * q;
            if (prm.model == FENE_P) term_I = q;
        } else {
            f2 = R(fT);
        }
        P11 = S11 + be * Gd11;
        P12 = S12 + be * Gd12;
        P22 = S22 - be * Gd11;
        const auto u11 = a11 - two * (gt11 * S11 + GU21 * S12);
        const auto u12 = a12 - (GU21 * S22 + GU12 * S11);          // gt11 + gt22 = 0
        const auto u22 = a22 - two * (GU12 * S12 + gt22 * S22);
        const auto fo = f1 * om;
        C11 = Wi * u11 + f3 * (S11 * S11 + S12 * S12) + f2 * S11 - fo * (Gd11 + term_I);
        C12 = Wi * u12 + f3 * (S12 * (S11 + S22)) + f2 * S12 - fo * Gd12;
        C22 = Wi * u22 + f3 * (S12 * S12 + S22 * S22) + f2 * S22 - fo * (term_I - Gd11);
        if (prm.model == FENE_P) C33 = -(fo * term_I);
        divT1 = R(X11 + Y12);
        divT2 = R(X12 + Y22);
        ddT = RF(ddS);
        ddC = RF(ddS);
    } else {
        const auto c11 = S11 * S11 + S12 * S12, c12 = S12 * (S11 + S22), c22 = S12 * S12 + S22 * S22;
        const auto d11x = two * (X11 * S11 + X12 * S12), d11y = two * (Y11 * S11 + Y12 * S12);
        const auto d22x = two * (X12 * S12 + X22 * S22), d22y = two * (Y12 * S12 + Y22 * S22);
        const auto d12x = X11 * S12 + X12 * (S11 + S22) + S12 * X22;
        const auto d12y = Y11 * S12 + Y12 * (S11 + S22) + S12 * Y22;
        const auto trC = c11 + c22;
        typedef decltype(S11 * S11) RC;
        typedef decltype(S11 * X11) RD;
        RC f = RC(one), f1 = RC(one), g1 = RC(one), g2 = RC(one);
        RD e1x = RD((T)0), e1y = RD((T)0), e2x = RD((T)0), e2y = RD((T)0);
        T f3c = (T)0;
        switch (prm.model) {
        case L_PTT:
        case M_L_PTT: f = Ve * (trC - two) + one; break;
        case E_PTT:
        case M_E_PTT: f = exp(Ve * (trC - two)); break;
        case GIESEKUS: f = RC(one - two * Ve); f3c = Ve; break;
        default: f = (Ve - two) * inv(Ve - trC); break;
        }
        f1 = prm.model == GIESEKUS ? RC(one - Ve) : (prm.model == FENE_P ? RC(one) : f);
        if (prm.model != L_PTT && prm.model != E_PTT && prm.model != GIESEKUS) {
            // f_T' per trace of c: VeN, VeN f_T, f_T / (VeN - tr c)
            const RC k = prm.model == M_L_PTT ? RC(Ve) : (prm.model == M_E_PTT ? RC(Ve * f) : RC(f * inv(Ve - trC)));
            g2 = f;
            e2x = k * (d11x + d22x);
            e2y = k * (d11y + d22y);
            if (prm.model != FENE_P) {
                g1 = f;
                e1x = e2x;
                e1y = e2y;
            }
        }
        fT = RF(f);
        f2 = R(f);
        const auto T11 = rr * (g2 * c11 - g1), T12 = rr * (g2 * c12), T22 = rr * (g2 * c22 - g1), T33 = rr * g1;
        P11 = T11 + be * Gd11;
        P12 = T12 + be * Gd12;
        P22 = T22 - be * Gd11;
        divT1 = rr * (e2x * c11 + g2 * d11x - e1x + e2y * c12 + g2 * d12y);
        divT2 = rr * (e2x * c12 + g2 * d12x + e2y * c22 + g2 * d22y - e1y);
        const auto rden = inv(S11 + S22);
        const auto W12 = (S12 * Gd11 - S11 * GU12 + S22 * GU21) * rden;
        const auto u11 = a11 - (S11 * gt11 + S12 * GU21) - W12 * S12;
        const auto u12 = a12 - (S11 * GU12 + S12 * gt22) - W12 * S22;
        const auto u22 = a22 - (S12 * GU12 + S22 * gt22) + W12 * S12;
        const auto f1d = f1 * inv(S11 * S22 - S12 * S12);
        // (f3 S^3 + f2 S - f1 S^-1) / 2
        C11 = Wi * u11 + half * (f3c * (S11 * c11 + S12 * c12) + f * S11 - f1d * S22);
        C12 = Wi * u12 + half * (f3c * (S11 * c12 + S12 * c22) + (f + f1d) * S12);
        C22 = Wi * u22 + half * (f3c * (S12 * c12 + S22 * c22) + f * S22 - f1d * S11);
        ddT = T11 * T11 + two * (T12 * T12) + T22 * T22 + T33 * T33;
        ddC = RF(c11 * c11 + two * (c12 * c12) + c22 * c22);
        f3 = RF(f3c);
    }
    // strongFormMomentum
    R M1 = -(divT1 + (be * lap1 - dPx)), M2 = -(divT2 + (be * lap2 - dPy));
    RU rc1 = RU((T)0), rc2 = RU((T)0);
    if constexpr (!(SPEC & SPEC_RE0)) {
        rc1 = Re * (U1 * GU11 + U2 * GU21);
        rc2 = Re * (U1 * GU12 + U2 * GU22);
        M1 = M1 + rc1;
        M2 = M2 + rc2;
    }
    // setStabilizationTerms
    RU ts = RU((T)0);
#pragma unroll
    for (int n = 0; n < 9; n++) ts = ts + fabs(U1 * chi[n].x + U2 * chi[n].y);
    const auto ha = (rr * rr + half * ddT) * inv(half * ddG + one) * (rH2 * rH2);   // (Ha / H^2)^2
    R tq = R(ha + (be * rH2) * (be * rH2));
    if constexpr (!(SPEC & SPEC_RE0)) {
        const auto q = Re * ts;
        tq = tq + (q * q + (Re / dt) * (Re / dt));
    }
    const R tm = inv_sqrt(tq);
    const R tic = H2 * (tq * tm);
    RF tda = RF(half * ddS);
    if constexpr (FORM == FORM_T) tda = tda + rr * rr;
    RF td = RF((T)0);
    if (!(Df > (T)1.0e-12)) td = H2 * inv_sqrt(tda);
    const R mag = sqrt(half * (C11 * C11 + two * (C12 * C12) + C22 * C22 + C33 * C33));
    const R tdm = td * mag;
    const auto wt = Wi * ts;
    const R b6 = tdm * rH2;
    R tcq = wt * wt + half * (Wi * Wi * ddG) + f2 * f2 + half * (f3 * f3 * ddC) + b6 * b6 + (Wi * Wi) * ((one / dt) * (one / dt));
    if constexpr (!(SPEC & SPEC_DF0)) tcq = tcq + (Df * rH2) * (Df * rH2);
    const R tc = inv_sqrt(tcq);
    // LSCE in the momentum equations: gradient coefficients
    R kx1, ky1, kx2, ky2;
    if constexpr (FORM == FORM_T) {
        kx1 = -(tc * C11);
        ky1 = -(tc * C12);
        kx2 = ky1;
        ky2 = -(tc * C22);
    } else {
        // (S . grad phi) : with WTensor2D's quotient (S12 (C22 - C11) + C12 (S11 - S22)) / (S11 + S22)
        const R Y = (S12 * (C22 - C11) + C12 * (S11 - S22)) * inv(S11 + S22);
        const R al = -(tc * rr);
        const R m = C12 - Y, q = C12 + Y;
        kx1 = al * (S11 * C11 + S12 * m);
        ky1 = al * (S12 * C11 + S22 * m);
        kx2 = al * (S11 * q + S12 * C22);
        ky2 = al * (S12 * q + S22 * C22);
    }
    const R ic = tic * tr;
    auto put = [&](int e, auto k0, auto k1, auto k2) {
        dst[e * 3] = w * tangent(k0);
        dst[e * 3 + 1] = w * tangent(k1);
        dst[e * 3 + 2] = w * tangent(k2);
    };
    MomentumFactors<T> mf;
    if constexpr (!(SPEC & SPEC_RE0)) {
        const R v1 = tm * Re * U1, v2 = tm * Re * U2;
        put(0, rc1, P11 + ic + v1 * M1 + kx1, P12 + v2 * M1 + ky1);
        put(1, rc2, P12 + v1 * M2 + kx2, P22 + ic + v2 * M2 + ky2);
        mf.u1 = value(v1);
        mf.u2 = value(v2);
    } else {
        put(0, (T)0, P11 + ic + kx1, P12 + ky1);
        put(1, (T)0, P12 + kx2, P22 + ic + ky2);
        mf.u1 = mf.u2 = (T)0;
    }
    const R tM1 = tm * M1, tM2 = tm * M2;
    put(2, tr, tM1, tM2);
    R s1, s2;
    if constexpr (FORM == FORM_T) {
        s1 = om * tM1;
        s2 = om * tM2;
        mf.ts = om * value(tm);
    } else {
        s1 = Wi * tM1;
        s2 = Wi * tM2;
        mf.ts = value(Wi) * value(tm);
    }
    mf.tm = value(tm);
    const R l0 = FORM == FORM_T ? R(one) : R(half * (tc * fT) + one);
    const R l1 = tc * (Wi * U1), l2 = tc * (Wi * U2);
    const R dd = tdm + Df;
    put(3, l0 * C11, l1 * C11 + dd * X11 - s1, l2 * C11 + dd * Y11);
    put(4, l0 * C12, l1 * C12 + dd * X12 - s2, l2 * C12 + dd * Y12 - s1);
    put(5, l0 * C22, l1 * C22 + dd * X22, l2 * C22 + dd * Y22 - s2);
    return mf;
}

// Elements at a time, threads, equations per contraction thread and CTAs per
// SM: the groups' direction counts (54, 27, 54, 9 per element) fill 18.1 of 20
// warps with 4 elements, 13.5 of 16 with 3 (FP64: 95 KB of shared memory a CTA,
// two per SM; 4 would leave one).
template <class T> struct ExCfg;
template <> struct ExCfg<float> { static constexpr int NE = 4, THREADS = 224, R = 6, CTAS = 2; };
template <> struct ExCfg<double> { static constexpr int NE = 3, THREADS = 256, R = 2, CTAS = 2; };

template <class T>
struct ExSmem {
    static constexpr int NE = ExCfg<T>::NE;
    Chi<T> chi[NE][9][9];
    T D[NE][9][EX_NDIR][18];     // reused as the output stage [NE][2916]
    T tl[NE][54];                // node 0's values, the others' differences from them
    T ip[NE][9][20];             // quantities in direction order
    T hw[NE][9][2];              // H^2, weight
};

template <class T, int FORM, int SPEC>
__device__ __forceinline__ void exact_elements(const ElemArgs &a, const KParams &prm, T *__restrict__ es,
                                               T *__restrict__ as, const int e0, const int ne, ExSmem<T> &sm)
{
    constexpr int NT = ExCfg<T>::THREADS, NE = ExCfg<T>::NE, NW = NT / 32;
    const int t = threadIdx.x, lane = t & 31;
    for (int i = t; i < ne * 54; i += NT) {
        const int el = i / 54, pos = i - 54 * el, inod = pos / 6, f = pos - 6 * inod;
        // relative to the element's first node (the gradients see differences
        // only): FP32 then rounds the variation over the element, not the value
        const double *tl = a.TL + (size_t)f * a.nnodes;
        const double t0 = tl[a.conn[e0 + el]];
        sm.tl[el][pos] = inod == 0 ? (T)t0 : (T)(tl[a.conn[inod * a.nel + e0 + el]] - t0);
    }
    for (int i = t; i < ne * 81; i += NT) {
        const int gp = i / 9, n = i - 9 * gp;                       // gp over all elements
        const double *r = a.geo + ((size_t)e0 * 9 + gp) * GEO_REC + n;
        Chi<T> c;
        c.p = (T)x_bfn[gp % 9][n];
        c.x = (T)r[0];
        c.y = (T)r[9];
        c.l = (T)(r[18] + r[27]);
        sm.chi[gp / 9][gp % 9][n] = c;
        if (n < 2) sm.hw[gp / 9][gp % 9][n] = (T)r[36];             // r + n: H^2, weight
    }
    __syncthreads();
    // interpolants: value, x, y, Laplacian of u and v; value, x, y of the others
    for (int i = t; i < ne * 9 * 20; i += NT) {
        const int gp = i / 20, d = i - 20 * gp, el = gp / 9;
        const int f = d < 8 ? d / 4 : 2 + (d - 8) / 3, k = d < 8 ? d % 4 : (d - 8) % 3;
        const T *c = reinterpret_cast<const T *>(&sm.chi[el][gp % 9][0]) + k;
        T v = (T)0;
#pragma unroll
        for (int n = 1; n < 9; n++) v += sm.tl[el][n * 6 + f] * c[4 * n];
        sm.ip[el][gp % 9][d] = k == 0 ? sm.tl[el][f] + v : v;
    }
    __syncthreads();
    {
        typedef Dual<T> X;
        T Wi = (T)prm.WiN, dWi = (T)0;
        if (prm.nex > 0) {
            dWi = (T)prm.Wi0;
            Wi = dWi * (T)a.EU[prm.nex - 1];
        }
        const int ns = (ne * 27 + 31) / 32, nu = (ne * 54 + 31) / 32, nw = (ne * 9 + 31) / 32;
        for (int wt = t >> 5; wt < ns + 2 * nu + nw; wt += NW) {
            // warp tasks: stress, velocity, stress gradient, Wi
            if (wt < ns) {
                const int k = wt * 32 + lane, gp = k / 3, d = k - 3 * gp;
                if (k < ne * 27) {
                    const int el = gp / 9, g = gp % 9;
                    const T *q = sm.ip[el][g];
                    coef_tangent<FORM, SPEC, T, T, X, T, T>(
                        prm, q[0], q[4], q[1], q[2], q[5], q[6], X(q[11], d == 0 ? (T)1 : (T)0),
                        X(q[14], d == 1 ? (T)1 : (T)0), X(q[17], d == 2 ? (T)1 : (T)0), q[12], q[13], q[15], q[16],
                        q[18], q[19], Wi, q[9], q[10], q[3], q[7], sm.hw[el][g][0], sm.hw[el][g][1], sm.chi[el][g],
                        sm.D[el][g][11 + 3 * d]);
                }
            } else if (wt < ns + nu) {
                const int k = (wt - ns) * 32 + lane, gp = k / 6, d = k - 6 * gp;
                if (k < ne * 54) {
                    const int el = gp / 9, g = gp % 9;
                    const T *q = sm.ip[el][g];
                    auto sd = [&](int i, int at) { return X(q[at], d == i ? (T)1 : (T)0); };
                    coef_tangent<FORM, SPEC, T, X, T, T, T>(
                        prm, sd(0, 0), sd(3, 4), sd(1, 1), sd(2, 2), sd(4, 5), sd(5, 6), q[11], q[14], q[17], q[12],
                        q[13], q[15], q[16], q[18], q[19], Wi, q[9], q[10], q[3], q[7], sm.hw[el][g][0],
                        sm.hw[el][g][1], sm.chi[el][g], sm.D[el][g][d < 3 ? d : d + 1]);
                }
            } else if (wt < ns + 2 * nu) {
                const int k = (wt - ns - nu) * 32 + lane, gp = k / 6, d = k - 6 * gp;
                if (k < ne * 54) {
                    const int el = gp / 9, g = gp % 9;
                    const T *q = sm.ip[el][g];
                    auto sd = [&](int i, int at) { return X(q[at], d == i ? (T)1 : (T)0); };
                    coef_tangent<FORM, SPEC, T, T, T, X, T>(
                        prm, q[0], q[4], q[1], q[2], q[5], q[6], q[11], q[14], q[17], sd(0, 12), sd(1, 13), sd(2, 15),
                        sd(3, 16), sd(4, 18), sd(5, 19), Wi, q[9], q[10], q[3], q[7], sm.hw[el][g][0],
                        sm.hw[el][g][1], sm.chi[el][g], sm.D[el][g][12 + 3 * (d / 2) + d % 2]);
                }
            } else {
                const int gp = (wt - ns - 2 * nu) * 32 + lane;
                if (gp < ne * 9) {
                    const int el = gp / 9, g = gp % 9;
                    const T *q = sm.ip[el][g];
                    const T w = sm.hw[el][g][1];
                    const MomentumFactors<T> m = coef_tangent<FORM, SPEC, T, T, T, T, X>(
                        prm, q[0], q[4], q[1], q[2], q[5], q[6], q[11], q[14], q[17], q[12], q[13], q[15], q[16],
                        q[18], q[19], X(Wi, dWi), q[9], q[10], q[3], q[7], sm.hw[el][g][0], w, sm.chi[el][g],
                        sm.D[el][g][20]);
                    // pressure: -p in the stress, grad p in the momentum residual;
                    // Laplacians: -beta there
                    const T be = (T)prm.BvN;
                    T *dp = sm.D[el][g][8], *dx = sm.D[el][g][9], *dy = sm.D[el][g][10];
                    T *l1 = sm.D[el][g][3], *l2 = sm.D[el][g][7];
#pragma unroll
                    for (int k = 0; k < 18; k++) {
                        const T v1 = k == 1 ? m.u1 : k == 2 ? m.u2 : k == 7 ? m.tm : k == 10 || k == 14 ? -m.ts : (T)0;
                        const T v2 = k == 4 ? m.u1 : k == 5 ? m.u2 : k == 8 ? m.tm : k == 13 || k == 17 ? -m.ts : (T)0;
                        dp[k] = k == 1 || k == 5 ? -w : (T)0;
                        dx[k] = w * v1;
                        dy[k] = w * v2;
                        l1[k] = -(be * w) * v1;
                        l2[k] = -(be * w) * v2;
                    }
                }
            }
        }
    }
    __syncthreads();

    // contraction; f is the slowest index, so a warp agrees on the Laplacian
    constexpr int R = ExCfg<T>::R, PARTS = 6 / R, TASKS = NE * 54 * PARTS, ROUNDS = (TASKS + NT - 1) / NT;
    T acc[ROUNDS][R][9];
#pragma unroll
    for (int it = 0; it < ROUNDS; it++) {
        const int k = it * NT + t;
        const int f = k / (NE * 9 * PARTS), m = k - f * (NE * 9 * PARTS);
        const int el = m / (9 * PARTS), i = (m / PARTS) % 9, part = m % PARTS;
#pragma unroll
        for (int r = 0; r < R; r++)
#pragma unroll
            for (int j = 0; j < 9; j++) acc[it][r][j] = (T)0;
        if (k < TASKS && el < ne) {
            const int q0 = qdir(f, 0);
            const bool lap = f < 2;
#pragma unroll 1
            for (int g = 0; g < 9; g++) {
                const Chi<T> p = sm.chi[el][g][i];
                const T *d = sm.D[el][g][q0] + part * (3 * R);
                T c0[R], c1[R], c2[R];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    c0[r] = p.p * d[3 * r] + p.x * d[3 * r + 1] + p.y * d[3 * r + 2];
                    c1[r] = p.p * d[18 + 3 * r] + p.x * d[18 + 3 * r + 1] + p.y * d[18 + 3 * r + 2];
                    c2[r] = p.p * d[36 + 3 * r] + p.x * d[36 + 3 * r + 1] + p.y * d[36 + 3 * r + 2];
                }
#pragma unroll
                for (int j = 0; j < 9; j++) {
                    const Chi<T> c = sm.chi[el][g][j];
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        T v = acc[it][r][j];
                        v += c0[r] * c.p;
                        v += c1[r] * c.x;
                        v += c2[r] * c.y;
                        acc[it][r][j] = v;
                    }
                }
                if (lap) {
#pragma unroll
                    for (int r = 0; r < R; r++)
                        c0[r] = p.p * d[54 + 3 * r] + p.x * d[54 + 3 * r + 1] + p.y * d[54 + 3 * r + 2];
#pragma unroll
                    for (int j = 0; j < 9; j++) {
                        const T l = sm.chi[el][g][j].l;
#pragma unroll
                        for (int r = 0; r < R; r++) acc[it][r][j] += c0[r] * l;
                    }
                }
            }
        }
    }
    if (prm.nex > 0) {
        for (int k = t; k < ne * 54; k += NT) {
            const int el = k / 54, i = (k % 54) / 6, e = k % 6;
            T v = (T)0;
            for (int g = 0; g < 9; g++) {
                const Chi<T> p = sm.chi[el][g][i];
                const T *d = sm.D[el][g][20] + e * 3;
                v += p.p * d[0] + p.x * d[1] + p.y * d[2];
            }
            as[(size_t)(e0 + el) * 54 + i * 6 + e] = v;
        }
    }
    __syncthreads();
    T *stage = &sm.D[0][0][0][0];
#pragma unroll
    for (int it = 0; it < ROUNDS; it++) {
        const int k = it * NT + t;
        const int f = k / (NE * 9 * PARTS), m = k - f * (NE * 9 * PARTS);
        const int el = m / (9 * PARTS), i = (m / PARTS) % 9, part = m % PARTS;
        if (k < TASKS && el < ne) {
#pragma unroll
            for (int r = 0; r < R; r++)
#pragma unroll
                for (int j = 0; j < 9; j++)
                    stage[el * 2916 + (i * 9 + j) * 36 + (part * R + r) * 6 + f] = acc[it][r][j];
        }
    }
    __syncthreads();
    T *out = es + (size_t)e0 * 2916;
    for (int o = t; o < ne * 2916; o += NT) out[o] = stage[o];
}

// persistent form over the work items of many meshes; each item is a run of
// consecutive elements of one mesh (the element-batch tile of its size class)
template <class T, int FORM, int SPEC>
__global__ void __launch_bounds__(ExCfg<T>::THREADS, ExCfg<T>::CTAS)
k_exact_batched(const BatchInst *__restrict__ insts, const WorkItem *__restrict__ work, int nwork)
{
    extern __shared__ __align__(32) unsigned char smraw[];
    ExSmem<T> &sm = *reinterpret_cast<ExSmem<T> *>(smraw);
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = work[w];
        const ElemArgs a = insts[it.inst].ea;
        const KParams prm = insts[it.inst].prm;
        T *es = static_cast<T *>(insts[it.inst].es);
        T *as = static_cast<T *>(insts[it.inst].as);
        const int e_end = min(it.e0 + it.count, a.nel);
        for (int e = it.e0; e < e_end; e += ExCfg<T>::NE) {
            exact_elements<T, FORM, SPEC>(a, prm, es, as, e, min(ExCfg<T>::NE, e_end - e), sm);
            __syncthreads();
        }
    }
}

template <class T, int FORM, int SPEC>
static cudaError_t go_exact_batched(const BatchInst *insts, const WorkItem *work, int nwork,
                                    int grid, cudaStream_t s)
{
    const size_t smem = sizeof(ExSmem<T>);
    cudaError_t e = cudaFuncSetAttribute(k_exact_batched<T, FORM, SPEC>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_exact_batched<T, FORM, SPEC><<<grid, ExCfg<T>::THREADS, smem, s>>>(insts, work, nwork);
    return cudaGetLastError();
}

// Elements per work item of nel elements in all (a mesh, a batch).  In FP64 a mesh
// of a few elements per SM takes as long as one SM does, most of it the FP64 pipe's
// time for the SM's elements, so they are spread evenly.  Residual, then Jacobian,
// T form, 150 / 300 / 450 quads: 145 / 213 / 372 us with one element to an item,
// 184 / 189 / 316 with two, 204 / 209 / 215 with three (a kernel of one element at a
// time took 222 / 347 / 471).  FP32 gains nothing by it (40 to 900 quads within 5%).
int exact_elements_per_item(int elem_size, int64_t nel, int sms)
{
    if (elem_size == 4) return ExCfg<float>::NE;
    return (int)std::min<int64_t>(ExCfg<double>::NE, std::max<int64_t>(1, (nel + sms - 1) / std::max(1, sms)));
}

template <class T>
cudaError_t launch_exact_batched(const BatchInst *insts, const WorkItem *work, int nwork,
                                 int form, int spec, int grid, cudaStream_t s)
{
    if (nwork <= 0) return cudaSuccess;
#define GO(F, SP)                                                                              if (form == F && spec == SP) return go_exact_batched<T, F, SP>(insts, work, nwork, grid, s);
    GO(FORM_T, 0) GO(FORM_T, SPEC_RE0) GO(FORM_T, SPEC_DF0) GO(FORM_T, SPEC_RE0 | SPEC_DF0)
    GO(FORM_SQRT, 0) GO(FORM_SQRT, SPEC_RE0) GO(FORM_SQRT, SPEC_DF0)
    GO(FORM_SQRT, SPEC_RE0 | SPEC_DF0)
#undef GO
    return cudaErrorInvalidValue;
}

template <class T, int FORM, int SPEC>
static int occ_exact()
{
    const size_t smem = sizeof(ExSmem<T>);
    if (cudaFuncSetAttribute(k_exact_batched<T, FORM, SPEC>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return 0;
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_exact_batched<T, FORM, SPEC>,
                                                  ExCfg<T>::THREADS, smem);
    return n;
}

int exact_batched_ctas_per_sm(int elem_size, int form, int spec)
{
#define OC(F, SP)                                                                              if (form == F && spec == SP)                                                                   return elem_size == 4 ? occ_exact<float, F, SP>() : occ_exact<double, F, SP>();
    OC(FORM_T, 0) OC(FORM_T, SPEC_RE0) OC(FORM_T, SPEC_DF0) OC(FORM_T, SPEC_RE0 | SPEC_DF0)
    OC(FORM_SQRT, 0) OC(FORM_SQRT, SPEC_RE0) OC(FORM_SQRT, SPEC_DF0)
    OC(FORM_SQRT, SPEC_RE0 | SPEC_DF0)
#undef OC
    return 0;
}

template cudaError_t launch_exact_batched<float>(const BatchInst *, const WorkItem *, int, int,
                                                 int, int, cudaStream_t);
template cudaError_t launch_exact_batched<double>(const BatchInst *, const WorkItem *, int, int,
                                                  int, int, cudaStream_t);

}  // namespace vefem
