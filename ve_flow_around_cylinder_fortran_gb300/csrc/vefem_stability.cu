// Linear-stability assembly: the A and B matrices of the generalised
// eigenproblem for spanwise-periodic 3-D perturbations (Neq = 10 per node:
// Ux, Uy, Uz, P, Txx, Txy, Tyy, Txz, Tyz, Tzz) of a steady 2-D base state,
// for many wavenumbers at once (setEquationsBulkStability,
// Equations_Stability_mod.F90:20-226; T form).
//
// The perturbation residual is linear in the perturbation, with the base
// state's quantities as coefficients, and at a Gauss point its weak-form
// term for test node i is linear in the test function's (phi, dphi/dx,
// dphi/dy):  TERM(i, e) = sum_k psi_k(i) c_ek(q).  The coefficients c depend
// linearly on 33 interpolated perturbation quantities q (velocity: value,
// x/y gradient, Laplacian; pressure and the six stresses: value, x/y
// gradient); the z-derivatives follow from the values and the wavenumber K
// (setExtraFlowUnknownsStability, Element_Calculations_Stability_mod.F90:280-311).
// The element matrices are therefore
//     A(i,e; j,f) = sum_gp WET sum_k psi_k(i) sum_s D[gp][q(f,s)][e][k] chi_s(j)
// with D = dc/dq obtained by evaluating c at unit q.  A is a quadratic
// polynomial in K and B does not depend on it, so the kernel builds the
// element blocks of B and of A at K = 0, +1, -1 once, and the scatter forms
// A(K) = A0 + K (A+ - A-)/2 + K^2 ((A+ + A-)/2 - A0) for every requested
// wavenumber while it sums the element blocks in element order.
//
// FP64 throughout.  Base quantities per Gauss point follow strongFormEquations
// with the stability problem's dimension N = 3 (traceless kinematics) and
// setStabilizationTerms; the perturbation physics restates
// setFlowQuantitiesStability, strongFormConEQ_Stability (L-PTT, m-L-PTT,
// e-PTT, m-e-PTT, Giesekus), strongFormMomentumStability and the terms of
// momentumStabilityT, momentumStability3D, continuityStability and
// stressStabilityT (Residuals_Stability_mod.F90:34-188).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "vefem.h"
#include "vefem_ctx.h"
#include "vefem_internal.h"
#include "vefem_physics.cuh"

namespace vefem {

namespace {

constexpr int ST_NEQ = 10;
constexpr int ST_NQ = 33;          // perturbation quantities
constexpr int ST_THREADS = 256;
constexpr int ST_BLK = 8100;       // 90 x 90 element block

__constant__ double s_w[9];
__constant__ double s_bfn[9][9], s_dfdc[9][9], s_dfde[9][9], s_d2c[9][9], s_d2e[9][9], s_d2ce[9][9];

// base quantities a Gauss point needs (StabBase) -- 3x3 tensors as the reference holds them
struct StabBase {
    double U[3];
    double GU[3][3], GUT[3][3], G_dot[3][3];
    double S[3][3], dT[3][3][3];
    double CE[3][3];                   // Con_EQ
    double f[3], g[2], fT;
    double tlsme, tlsic, tlsce, tdcs, mag;
    double WET;
};

__device__ __forceinline__ double tr3(const double A[3][3]) { return A[0][0] + A[1][1] + A[2][2]; }

// doubleDotProduct (Tools_mod.F90:262-280): sum_ij A(i,j) B(j,i)
__device__ __forceinline__ double ddot(const double A[3][3], const double B[3][3])
{
    double s = 0.0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) s = s + A[i][j] * B[j][i];
    return s;
}

__device__ __forceinline__ void mm3(const double A[3][3], const double B[3][3], double C[3][3])
{
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double s = 0.0;
            for (int k = 0; k < 3; k++) s = s + A[i][k] * B[k][j];
            C[i][j] = s;
        }
}

// stress component of unknown i - istart (getStressComponent, Tools_mod.F90:769-793)
__device__ __forceinline__ void stress_jk(int c, int &j, int &k)
{
    const int J[6] = {0, 0, 1, 0, 1, 2}, K[6] = {0, 1, 1, 2, 2, 2};
    j = J[c];
    k = K[c];
}

// Base state at Gauss point ig of an element: setFlowUnknownsStability on
// TEMP_TL_b, strongFormEquations(Problem_Stability) (N = 3), setStabilizationTerms.
__device__ void stab_base(const KParams &p, const double *tlb /* [9][10] */, const double *dFx,
                          const double *dFy, const double *d2x, const double *d2y, double H2,
                          double WET, int ig, StabBase &b)
{
    const double WiN = p.WiN, BvN = p.BvN, VeN = p.VeN, ReN = p.ReN, DfN = p.DfN, dt = p.dt;
    double GU[3][3] = {}, G2U[3][3] = {}, U[3] = {}, dP[3] = {}, P = 0.0;
    double S[3][3] = {}, dS[3][3][3] = {};
    for (int i = 0; i < 3; i++) {
        double u = 0.0, gx = 0.0, gy = 0.0, hx = 0.0, hy = 0.0, px = 0.0, py = 0.0;
        for (int n = 0; n < 9; n++) {
            const double t = tlb[n * ST_NEQ + i];
            u = u + t * s_bfn[ig][n];
            gx = gx + t * dFx[n];
            gy = gy + t * dFy[n];
            hx = hx + t * d2x[n];
            hy = hy + t * d2y[n];
        }
        U[i] = u;
        GU[0][i] = gx;
        GU[1][i] = gy;
        G2U[0][i] = hx;
        G2U[1][i] = hy;
    }
    {
        double pv = 0.0, px = 0.0, py = 0.0;
        for (int n = 0; n < 9; n++) {
            const double t = tlb[n * ST_NEQ + 3];
            pv = pv + t * s_bfn[ig][n];
            px = px + t * dFx[n];
            py = py + t * dFy[n];
        }
        P = pv;
        dP[0] = px;
        dP[1] = py;
    }
    for (int c = 0; c < 6; c++) {
        int j, k;
        stress_jk(c, j, k);
        double v = 0.0, gx = 0.0, gy = 0.0;
        for (int n = 0; n < 9; n++) {
            const double t = tlb[n * ST_NEQ + 4 + c];
            v = v + t * s_bfn[ig][n];
            gx = gx + t * dFx[n];
            gy = gy + t * dFy[n];
        }
        S[j][k] = v;
        S[k][j] = v;
        dS[j][k][0] = gx;
        dS[j][k][1] = gy;
        dS[k][j][0] = gx;
        dS[k][j][1] = gy;
    }
    // setFlowKinematics, N = 3
    double GUT[3][3], Gd[3][3], GUtr[3][3], GUTtr[3][3], Gdtr[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) GUT[i][j] = GU[j][i];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Gd[i][j] = GU[i][j] + GUT[i][j];
    const double trg = tr3(GU);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) GUtr[i][j] = GU[i][j] - trg * (i == j ? 1.0 : 0.0) / 3.0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) GUTtr[i][j] = GUtr[j][i];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Gdtr[i][j] = GUtr[i][j] + GUTtr[i][j];
    // conEQ_* (Constitutive_Models_mod.F90:96-268), models restated for stability
    const double trT = tr3(S);
    const bool fene = p.model == FENE_CR || p.model == FENE_P;
    double fT = 1.0, f0 = 1.0, f1 = 1.0, f2 = 0.0, g0 = 1.0, g1 = 1.0, termI = 0.0;
    if (p.model == L_PTT || p.model == M_L_PTT) {
        fT = 1.0 + (VeN * WiN * trT) / (1.0 - BvN);
    } else if (p.model == E_PTT || p.model == M_E_PTT) {
        fT = exp(VeN * WiN * trT / (1.0 - BvN));
    } else if (p.model == FENE_CR) {   // N = 2, the base problem's dimension
        fT = 1.0 + ((WiN * trT / (1.0 - BvN))) / (VeN - 2.0);
    } else if (p.model == FENE_P) {
        fT = 1.0 + (WiN * trT / (1.0 - BvN)) / VeN;
    } else {  // GIESEKUS
        fT = VeN * WiN / (1.0 - BvN);
    }
    if (p.model == GIESEKUS) {
        f2 = fT;
    } else if (p.model == M_L_PTT || p.model == M_E_PTT) {
        f0 = fT; f1 = fT; g0 = fT; g1 = fT;
    } else if (fene) {
        // setFENEMaterialDerivative (steady): U . grad f_T from the trace of grad T
        double df[3] = {0.0, 0.0, 0.0};
        for (int i = 0; i < 3; i++)
            for (int c = 0; c < 3; c++) df[c] = df[c] + dS[i][i][c];
        const double den = p.model == FENE_P ? VeN : (VeN - 2.0);
        for (int c = 0; c < 3; c++) df[c] = (WiN / (1.0 - BvN)) * df[c] / den;
        double MD = 0.0;
        for (int i = 0; i < 3; i++) MD = MD + U[i] * df[i];
        f1 = fT - (WiN * MD / fT);
        if (p.model == FENE_CR) {
            f0 = fT; g0 = fT; g1 = fT;
        } else {
            g1 = fT;
            termI = MD / fT;
        }
    } else {
        f1 = fT;
    }
    // upper-convected derivative (steady) and Con_EQ
    double UCD[3][3] = {}, M1[3][3], M2[3][3], T2[3][3];
    for (int k = 0; k < 3; k++)
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) UCD[i][j] = UCD[i][j] + U[k] * dS[i][j][k];
    mm3(GUTtr, S, M1);
    mm3(S, GUtr, M2);
    mm3(S, S, T2);
    double CE[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            const double ucd = UCD[i][j] - M1[i][j] - M2[i][j];
            double c = WiN * ucd + f2 * T2[i][j];
            c = c + f1 * S[i][j];
            c = c - f0 * (1.0 - BvN) * (Gdtr[i][j] + termI * (i == j ? 1.0 : 0.0));
            CE[i][j] = c;
        }
    // setStabilizationTerms
    double tsugn = 0.0;
    for (int n = 0; n < 9; n++) tsugn = tsugn + fabs(U[0] * dFx[n] + U[1] * dFy[n]);
    const double ddT = ddot(S, S), ddG = ddot(Gdtr, Gdtr);
    double Ha = sqrt(((1.0 - BvN) / WiN) * ((1.0 - BvN) / WiN) + 0.5 * ddT);
    Ha = Ha / sqrt(1.0 + 0.5 * ddG);
    const double t1 = ReN / dt, t2 = ReN * tsugn, t3 = BvN / H2, t4 = Ha / H2;
    double tlsme = t1 * t1 + t2 * t2 + t3 * t3 + t4 * t4;
    tlsme = 1.0 / sqrt(tlsme);
    double tdcs = 0.5 * ddot(S, S);
    tdcs = tdcs + ((1.0 - BvN) / WiN) * ((1.0 - BvN) / WiN);
    tdcs = H2 / sqrt(tdcs);
    if (DfN > 1.0e-12) tdcs = 0.0;
    double mag = sqrt(0.5 * ddot(CE, CE));
    const double s1 = WiN / dt, s2 = WiN * tsugn, s3 = WiN * sqrt(0.5 * ddG), s4 = f1;
    const double s5 = f2 * sqrt(0.5 * ddT), s6 = tdcs * mag / H2, s7 = DfN / H2;
    double tlsce = s1 * s1 + s2 * s2 + s3 * s3 + s4 * s4 + s5 * s5 + s6 * s6 + s7 * s7;
    tlsce = 1.0 / sqrt(tlsce);

    for (int i = 0; i < 3; i++) {
        b.U[i] = U[i];
        for (int j = 0; j < 3; j++) {
            b.GU[i][j] = GU[i][j];
            b.GUT[i][j] = GUT[i][j];
            b.G_dot[i][j] = Gd[i][j];
            b.S[i][j] = S[i][j];
            b.CE[i][j] = CE[i][j];
            for (int k = 0; k < 3; k++) b.dT[i][j][k] = dS[i][j][k];
        }
    }
    b.f[0] = f0; b.f[1] = f1; b.f[2] = f2; b.g[0] = g0; b.g[1] = g1; b.fT = fT;
    b.tlsme = tlsme;
    b.tlsic = H2 / tlsme;
    b.tlsce = tlsce;
    b.tdcs = tdcs;
    b.mag = mag;
    b.WET = WET;
    (void)P; (void)dP; (void)G2U;
}

// Coefficients c_a[e][k], c_b[e][k] (k: phi, dphi/dx, dphi/dy) of the
// perturbation's weak-form terms at one Gauss point for unit quantity q.
__device__ void stab_coef(const KParams &p, const StabBase &b, double K, int kz, int q,
                          double ca[ST_NEQ][3], double cb[ST_NEQ][3])
{
    const double WiN = p.WiN, BvN = p.BvN, ReN = p.ReN, DfN = p.DfN, VeN = p.VeN;
    double U[3] = {}, GU[3][3] = {}, G2U[3][3] = {}, P = 0.0, dP[3] = {};
    double S[3][3] = {}, dT[3][3][3] = {};
    // unit interpolant q: velocity i: value, d/dx, d/dy, Laplacian (x and y parts summed)
    if (q < 12) {
        const int i = q / 4, s = q % 4;
        if (s == 0) U[i] = 1.0;
        else if (s == 1) GU[0][i] = 1.0;
        else if (s == 2) GU[1][i] = 1.0;
        else G2U[0][i] = 1.0;
    } else if (q < 15) {
        const int s = q - 12;
        if (s == 0) P = 1.0;
        else dP[s - 1] = 1.0;
    } else {
        const int c = (q - 15) / 3, s = (q - 15) % 3;
        int j, k;
        stress_jk(c, j, k);
        if (s == 0) {
            S[j][k] = 1.0;
            S[k][j] = 1.0;
        } else {
            dT[j][k][s - 1] = 1.0;
            dT[k][j][s - 1] = 1.0;
        }
    }
    if (kz) {   // setExtraFlowUnknownsStability, real split, N = z
        GU[2][0] = -K * U[0];
        GU[2][1] = -K * U[1];
        GU[2][2] = K * U[2];
        dP[2] = -K * P;
        for (int a = 0; a < 3; a++)
            for (int c = 0; c < 3; c++) dT[a][c][2] = -K * S[a][c];
        dT[0][2][2] = K * S[0][2];
        dT[2][0][2] = dT[0][2][2];
        dT[1][2][2] = K * S[1][2];
        dT[2][1][2] = dT[1][2][2];
        for (int i = 0; i < 3; i++) G2U[2][i] = -(K * K) * U[i];
    }
    // setFlowKinematics
    double GUT[3][3], Gd[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) GUT[i][j] = GU[j][i];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Gd[i][j] = GU[i][j] + GUT[i][j];
    // conEQ_*_Stability (Constitutive_Models_Stability_mod.F90:96-289)
    const double trT = tr3(S);
    const bool fene = p.model == FENE_CR || p.model == FENE_P;
    double fT = 0.0, f0 = 0.0, f1 = 0.0, termI = 0.0, termIt = 0.0;
    if (p.model == L_PTT || p.model == M_L_PTT) fT = VeN * WiN * trT / (1.0 - BvN);
    else if (p.model == E_PTT || p.model == M_E_PTT) fT = b.fT * VeN * WiN * trT / (1.0 - BvN);
    else if (p.model == FENE_CR) fT = (WiN * trT / (1.0 - BvN)) / (VeN - 2.0);
    else if (p.model == FENE_P) fT = (WiN * trT / (1.0 - BvN)) / VeN;
    if (p.model == M_L_PTT || p.model == M_E_PTT || p.model == FENE_CR) f0 = fT;
    if (p.model != GIESEKUS) f1 = fT;
    if (fene) {
        // setFENEMaterialDerivativeStability (:294-328)
        double dfb[3] = {0.0, 0.0, 0.0}, dfd[3] = {0.0, 0.0, 0.0};
        for (int i = 0; i < 3; i++)
            for (int c = 0; c < 3; c++) {
                dfb[c] = dfb[c] + b.dT[i][i][c];
                dfd[c] = dfd[c] + dT[i][i][c];
            }
        const double den = p.model == FENE_P ? VeN : (VeN - 2.0);
        for (int c = 0; c < 3; c++) {
            dfb[c] = (WiN / (1.0 - BvN)) * dfb[c] / den;
            dfd[c] = (WiN / (1.0 - BvN)) * dfd[c] / den;
        }
        double MD = 0.0;
        for (int i = 0; i < 3; i++) {
            const double term = ((b.fT) * dfd[i] - fT * dfb[i]) / (b.fT);
            MD = MD + U[i] * dfb[i] + b.U[i] * term;
        }
        f1 = fT - WiN * MD / (b.fT);
        if (p.model == FENE_P) {
            termI = MD / (b.fT);
            termIt = -(1.0 - BvN) * fT / (b.fT);
        }
    }
    // setStressTensorStability: P_tot (C_Tensor of the perturbation is not used below)
    double Pt[3][3];
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) Pt[i][j] = S[i][j] + BvN * Gd[i][j] - P * (i == j ? 1.0 : 0.0);
    // setUCDStability
    double UCD[3][3] = {}, M1[3][3], M2[3][3], M3[3][3], M4[3][3];
    for (int k = 0; k < 3; k++)
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++) UCD[i][j] = UCD[i][j] + b.U[k] * dT[i][j][k] + U[k] * b.dT[i][j][k];
    mm3(b.GUT, S, M1);
    mm3(GUT, b.S, M2);
    mm3(b.S, GU, M3);
    mm3(S, b.GU, M4);
    double SbSd[3][3], SdSb[3][3], SbSb[3][3], CE[3][3];
    mm3(b.S, S, SbSd);
    mm3(S, b.S, SdSb);
    mm3(b.S, b.S, SbSb);
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            const double ucd = UCD[i][j] - M1[i][j] - M2[i][j] - M3[i][j] - M4[i][j];
            const double tT = b.f[2] * (SbSd[i][j] + SdSb[i][j]) + 0.0 * SbSb[i][j] + f1 * b.S[i][j]
                              + b.f[1] * S[i][j];
            const double tG = b.f[0] * Gd[i][j] + f0 * b.G_dot[i][j];
            CE[i][j] = WiN * ucd + tT - (1.0 - BvN) * (tG + termI * (i == j ? 1.0 : 0.0));
        }
    // strongFormMomentumStability
    double Mom[3], mt[3];
    for (int i = 0; i < 3; i++) {
        double divT = 0.0;
        for (int j = 0; j < 3; j++) divT = divT + dT[j][i][j];
        const double divP = -dP[i] + divT + BvN * (G2U[0][i] + G2U[1][i] + G2U[2][i]);
        double c1 = 0.0, c2 = 0.0;
        for (int k = 0; k < 3; k++) c1 = c1 + b.U[k] * GU[k][i];
        for (int k = 0; k < 3; k++) c2 = c2 + U[k] * b.GU[k][i];
        Mom[i] = ReN * (c1 + c2) - divP;
        mt[i] = ReN * U[i];
    }
    const double Cont = tr3(GU);
    const double magd = ddot(b.CE, CE) / (2.0 * b.mag + 1.0e-12);
    double ceqt[3][3];     // Con_EQ_time (strongFormConEQ_Stability :85-93)
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            double c = WiN * S[i][j];
            if (fene) c = c - WiN * fT * b.S[i][j] / (b.fT);
            ceqt[i][j] = c + termIt * (i == j ? 1.0 : 0.0);
        }
    double conv[3];
    for (int i = 0; i < 3; i++) {
        double c1 = 0.0, c2 = 0.0;
        for (int k = 0; k < 3; k++) c1 = c1 + b.U[k] * GU[k][i];
        for (int k = 0; k < 3; k++) c2 = c2 + U[k] * b.GU[k][i];
        conv[i] = c1 + c2;
    }
    // momentumStabilityT + momentumStability3D
    const double lme[2] = {b.tlsme * ReN * b.U[0], b.tlsme * ReN * b.U[1]};   // LSMEMomentum per dphi
    for (int i = 0; i < 3; i++) {
        const double k3 = (i == 2) ? -K : K;
        ca[i][0] = ReN * conv[i] - k3 * Pt[i][2];
        cb[i][0] = mt[i];
        for (int c = 0; c < 2; c++) {
            ca[i][1 + c] = Pt[i][c] + lme[c] * Mom[i] + (i == c ? b.tlsic * Cont : 0.0)
                           - b.tlsce * CE[c][i];
            cb[i][1 + c] = lme[c] * mt[i] - b.tlsce * ceqt[c][i];
        }
    }
    // continuityStability
    ca[3][0] = Cont;
    cb[3][0] = 0.0;
    for (int c = 0; c < 2; c++) {
        ca[3][1 + c] = b.tlsme * Mom[c];
        cb[3][1 + c] = b.tlsme * mt[c];
    }
    // stressStabilityT
    for (int cc = 0; cc < 6; cc++) {
        int j, k;
        stress_jk(cc, j, k);
        const int e = 4 + cc;
        ca[e][0] = CE[j][k];
        cb[e][0] = ceqt[j][k];
        for (int c = 0; c < 2; c++) {
            double lm = -(k == c ? Mom[j] : 0.0);
            double lt = -(k == c ? mt[j] : 0.0);
            if (j != k) {
                lm = lm - (j == c ? Mom[k] : 0.0);
                lt = lt - (j == c ? mt[k] : 0.0);
            }
            const double lce = b.tlsce * WiN * b.U[c];
            const double dcs = b.tdcs * b.dT[j][k][c];
            ca[e][1 + c] = DfN * dT[j][k][c] + b.tlsme * lm * (1.0 - BvN) + lce * CE[j][k] + dcs * magd;
            cb[e][1 + c] = b.tlsme * lt * (1.0 - BvN) + lce * ceqt[j][k];
        }
    }
    // TERM_RES_b = -TERM_RES_b
    for (int e = 0; e < ST_NEQ; e++)
        for (int c = 0; c < 3; c++) cb[e][c] = -cb[e][c];
}

struct StabArgs {
    int nel, nnodes;
    const int32_t *conn;
    const double *xy;
    const double *TLb;      // [10][nnodes] embedded base state
    double *es;             // [nel][4][ST_BLK]: B, A(0), A(+1), A(-1), block layout
    int kz;
};

// quantity index of field f, basis component s (0 value, 1 d/dx, 2 d/dy, 3 Laplacian)
__device__ __forceinline__ int st_q(int f, int s)
{
    return f < 3 ? f * 4 + s : (f == 3 ? 12 + s : 15 + (f - 4) * 3 + s);
}

constexpr int ST_JCH = 3;                                            // test nodes per chunk
constexpr int ST_CH_OUT = ST_JCH * 900;                              // outputs per chunk (2700)
constexpr int ST_PER_T = (ST_CH_OUT + ST_THREADS - 1) / ST_THREADS;  // outputs per thread (11)
constexpr int ST_A2 = ST_NQ + 1;                                     // row stride of A2

// Shared memory: D and DB [9][33][10][3] coefficient derivatives (A at one K
// and, from the same evaluations at K = 0, B), A2 [30][ST_A2] the test-side
// contraction of one Gauss point for one chunk of three test nodes, and the
// base quantities of the 9 Gauss points.
__host__ __device__ constexpr size_t st_smem_doubles()
{
    return (size_t)2 * 9 * ST_NQ * ST_NEQ * 3 + (size_t)ST_JCH * ST_NEQ * ST_A2;
}

__global__ void __launch_bounds__(ST_THREADS)
k_stability(const StabArgs a, const KParams prm)
{
    extern __shared__ __align__(16) double sm[];
    double *D = sm;                                   // [9][33][10][3]
    double *DB = D + 9 * ST_NQ * ST_NEQ * 3;          // [9][33][10][3]
    double *A2 = DB + 9 * ST_NQ * ST_NEQ * 3;         // [30][ST_A2]
    StabBase *base = reinterpret_cast<StabBase *>(A2 + ST_JCH * ST_NEQ * ST_A2);
    __shared__ double s_tlb[9 * ST_NEQ];
    __shared__ double s_dFx[9][9], s_dFy[9][9], s_lap[9][9], s_H2[9], s_W[9];
    __shared__ double s_d2x[9][9], s_d2y[9][9];
    const int t = threadIdx.x;
    for (int e = blockIdx.x; e < a.nel; e += gridDim.x) {
        if (t < 9 * ST_NEQ) {
            const int n = t / ST_NEQ, f = t % ST_NEQ;
            s_tlb[t] = a.TLb[(size_t)f * a.nnodes + a.conn[n * a.nel + e]];
        } else if (t >= 96 && t < 105) {
            const int ig = t - 96;
            double x[9], y[9], fx[9], fy[9], sx[9], sy[9];
            for (int n = 0; n < 9; n++) {
                const int gn = a.conn[n * a.nel + e];
                x[n] = a.xy[gn];
                y[n] = a.xy[a.nnodes + gn];
            }
            auto go = geometry(s_bfn[ig], s_dfdc[ig], s_dfde[ig], s_d2c[ig], s_d2e[ig], s_d2ce[ig],
                               s_w[ig], x, y, fx, fy, sx, sy);
            for (int n = 0; n < 9; n++) {
                s_dFx[ig][n] = fx[n];
                s_dFy[ig][n] = fy[n];
                s_d2x[ig][n] = sx[n];
                s_d2y[ig][n] = sy[n];
                s_lap[ig][n] = sx[n] + sy[n];
            }
            s_H2[ig] = go.H2;
            s_W[ig] = go.WET;
        }
        __syncthreads();
        if (t < 9)
            stab_base(prm, s_tlb, s_dFx[t], s_dFy[t], s_d2x[t], s_d2y[t], s_H2[t], s_W[t], t, base[t]);
        __syncthreads();
        double *out = a.es + (size_t)e * 4 * ST_BLK;
        // element block m: 0 B (K = 0), 1 A(0), 2 A(+1), 3 A(-1); layout
        // ((jnod*9 + inod)*10 + jeq)*10 + ieq: row (jnod, jeq) = equation of test node
        // jnod, column (inod, ieq) = unknown of trial node inod.  The K = 0
        // evaluations give both B and A(0).
        for (int m = 0; m < 4; m++) {
            const double K = m == 2 ? 1.0 : (m == 3 ? -1.0 : 0.0);
            if (m != 1) {
                for (int w = t; w < 9 * ST_NQ; w += ST_THREADS) {
                    const int gp = w / ST_NQ, q = w % ST_NQ;
                    double ca[ST_NEQ][3], cb[ST_NEQ][3];
                    stab_coef(prm, base[gp], K, a.kz, q, ca, cb);
                    double *da = D + (size_t)w * ST_NEQ * 3, *db = DB + (size_t)w * ST_NEQ * 3;
                    for (int e2 = 0; e2 < ST_NEQ; e2++)
                        for (int c = 0; c < 3; c++) {
                            da[e2 * 3 + c] = ca[e2][c];
                            if (m == 0) db[e2 * 3 + c] = cb[e2][c];
                        }
                }
                __syncthreads();
            }
            const double *Dm = m == 0 ? DB : D;
            for (int j0 = 0; j0 < 9; j0 += ST_JCH) {
                double acc[ST_PER_T];
#pragma unroll
                for (int r = 0; r < ST_PER_T; r++) acc[r] = 0.0;
                for (int gp = 0; gp < 9; gp++) {
                    // test side: A2[(jn - j0)*10 + je][q] = WET sum_k psi_k(jn) D[gp][q][je][k]
                    const double w = base[gp].WET;
                    for (int it = t; it < ST_JCH * ST_NEQ * ST_NQ; it += ST_THREADS) {
                        const int row = it / ST_NQ, q = it % ST_NQ;
                        const int jn = j0 + row / ST_NEQ, je = row % ST_NEQ;
                        const double *dd = Dm + ((size_t)(gp * ST_NQ + q) * ST_NEQ + je) * 3;
                        A2[row * ST_A2 + q] = w * (s_bfn[gp][jn] * dd[0] + s_dFx[gp][jn] * dd[1]
                                                   + s_dFy[gp][jn] * dd[2]);
                    }
                    __syncthreads();
                    // trial side; chunk output c = ((jn - j0)*9 + inod)*100 + jeq*10 + ieq
#pragma unroll
                    for (int r = 0; r < ST_PER_T; r++) {
                        const int c = t + r * ST_THREADS;
                        if (c < ST_CH_OUT) {
                            const int ji = c / 100, rr = c % 100;
                            const int jl = ji / 9, in = ji % 9;
                            const int je = rr / 10, ie = rr % 10;
                            const double *a2 = A2 + (jl * ST_NEQ + je) * ST_A2;
                            const int q0 = st_q(ie, 0);
                            double v = a2[q0] * s_bfn[gp][in] + a2[q0 + 1] * s_dFx[gp][in]
                                       + a2[q0 + 2] * s_dFy[gp][in];
                            if (ie < 3) v = v + a2[q0 + 3] * s_lap[gp][in];
                            acc[r] = acc[r] + v;
                        }
                    }
                    __syncthreads();
                }
#pragma unroll
                for (int r = 0; r < ST_PER_T; r++) {
                    const int c = t + r * ST_THREADS;
                    if (c < ST_CH_OUT) out[(size_t)m * ST_BLK + j0 * 900 + c] = acc[r];
                }
            }
        }
    }
}

// one thread per AIJ entry of a node-pair block of the 10-unknown pattern
__global__ void k_stability_gather(const GatherArgs g, const int64_t *__restrict__ rowptr10,
                                   const int32_t *__restrict__ boff10, const double *__restrict__ es,
                                   int nk, const double *__restrict__ kw, double *const *A,
                                   double *B)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)g.nblocks * 100) return;
    const int blk = (int)(t / 100), r = (int)(t % 100);
    const int jeq = r / 10, ieq = r % 10;
    const int64_t slot = rowptr10[(int64_t)g.brow[blk] * ST_NEQ + jeq] + boff10[blk] + ieq;
    double sb = 0.0, s0 = 0.0, sp = 0.0, sn = 0.0;
    for (int c = g.bptr[blk]; c < g.bptr[blk + 1]; c++) {
        const int64_t con = g.bcon[c];                    // e*81 + jnod*9 + inod
        const int64_t e = con / 81, ji = con % 81;
        const double *src = es + (size_t)e * 4 * ST_BLK + ji * 100 + r;
        sb = sb + src[0];
        s0 = s0 + src[ST_BLK];
        sp = sp + src[2 * ST_BLK];
        sn = sn + src[3 * ST_BLK];
    }
    if (B) B[slot] = B[slot] + sb;
    const double a1 = (sp - sn) * 0.5, a2 = (sp + sn) * 0.5 - s0;
    for (int k = 0; k < nk; k++) {   // A(K) = s0 + K (a1 + K a2), two FMAs per wavenumber
        const double K = kw[k];
        A[k][slot] = A[k][slot] + __fma_rn(K, __fma_rn(K, a2, a1), s0);
    }
}

// ---------------------------------------------------------------------------
// Planar base states (W = Txz = Tyz = Tzz = 0, what updateStabilityArrays
// embeds).  Most of the 10 x 10 x 33 x 3 coefficients above are then
// structural zeros: in-plane and out-of-plane unknowns couple only through
// the wavenumber, A's linear and quadratic parts in K and B act on values
// only.  128 (equation, unknown) pairs are left of 400 for B and the three
// coefficients A0, A1, A2 of A(K) = A0 + K A1 + K^2 A2.
//
// The general kernel is bound by the FP64 pipe (76% active) on 4.4 M
// instructions per element: coefficients evaluated at 33 unit quantities and
// three wavenumbers, 4 x 8100 outputs.  Here they are written down once per
// Gauss point (k_planar_coef, a thread per point) and contracted pair by pair
// (k_planar_contract: 0.24 M multiply-adds per element), and the scatter reads
// 83 KB per element instead of 259.  20,000 quads, 16 wavenumbers and B:
// 184.6 -> 14.5 ms.  The line between the routes is the check of the four
// out-of-plane base fields (k_nonplanar, one pass over 2.6 MB): the pairs left
// out are exact zeros for a planar base and for no other.

constexpr int PL_NV = 17, PL_NS = 41, PL_NM = 70;        // pairs of velocity, stress/pressure, value type
constexpr int PL_NP = PL_NV + PL_NS + PL_NM;             // 128
// pairs that are nonzero without FENE (velocity, stress) and with Re = 0 besides (value type)
constexpr int PL_NV0 = 15, PL_NS0 = 38, PL_NM0 = 46;
// record of a Gauss point: coefficients [4 s][3 k][17], [3][3][41], [3 k][70],
// each pair-fastest, then dphi/dx, dphi/dy and the Laplacian of the 9 nodes
constexpr int PL_OS = 12 * PL_NV, PL_OM = PL_OS + 9 * PL_NS, PL_OG = PL_OM + 3 * PL_NM;
constexpr int PL_REC = PL_OG + 27;                       // 810 doubles
constexpr int PL_OUT = 81 * PL_NP;                       // outputs per element

struct PlPair {
    signed char m, e, f;    // matrix 0 B, 1 A0, 2 A1, 3 A2; equation; unknown
};
// Order of the pairs: those that need FENE (or Re, value type) come last.
static const PlPair PL_PAIRS[PL_NP] = {
    // velocity type, A0: u1, u2 in m1 m2 c 11 12 22; u3 in m3 13 23; FENE: u1, u2 in 33
    {1, 0, 0}, {1, 1, 0}, {1, 3, 0}, {1, 4, 0}, {1, 5, 0}, {1, 6, 0},
    {1, 0, 1}, {1, 1, 1}, {1, 3, 1}, {1, 4, 1}, {1, 5, 1}, {1, 6, 1},
    {1, 2, 2}, {1, 7, 2}, {1, 8, 2}, {1, 9, 0}, {1, 9, 1},
    // stress type, A0: p, s11, s12, s22 in m1 m2 c 11 12 22; s33 in m1 m2 11 12 22 33; s13, s23
    // in m3 13 23; A1: u3 in m1, m2; FENE: s11, s12, s22 in 33
    {1, 0, 3}, {1, 1, 3}, {1, 3, 3}, {1, 4, 3}, {1, 5, 3}, {1, 6, 3},
    {1, 0, 4}, {1, 1, 4}, {1, 3, 4}, {1, 4, 4}, {1, 5, 4}, {1, 6, 4},
    {1, 0, 5}, {1, 1, 5}, {1, 3, 5}, {1, 4, 5}, {1, 5, 5}, {1, 6, 5},
    {1, 0, 6}, {1, 1, 6}, {1, 3, 6}, {1, 4, 6}, {1, 5, 6}, {1, 6, 6},
    {1, 0, 9}, {1, 1, 9}, {1, 4, 9}, {1, 5, 9}, {1, 6, 9}, {1, 9, 9},
    {1, 2, 7}, {1, 7, 7}, {1, 8, 7}, {1, 2, 8}, {1, 7, 8}, {1, 8, 8},
    {2, 0, 2}, {2, 1, 2}, {1, 9, 4}, {1, 9, 5}, {1, 9, 6},
    // value type: A1
    {2, 0, 7}, {2, 1, 8}, {2, 2, 0}, {2, 2, 1}, {2, 2, 3}, {2, 2, 9}, {2, 3, 2}, {2, 3, 7}, {2, 3, 8},
    {2, 4, 7}, {2, 4, 2}, {2, 5, 7}, {2, 5, 8}, {2, 5, 2}, {2, 6, 8}, {2, 6, 2}, {2, 9, 2},
    {2, 7, 0}, {2, 7, 3}, {2, 7, 9}, {2, 8, 1}, {2, 8, 3}, {2, 8, 9},
    // A2
    {3, 0, 0}, {3, 1, 1}, {3, 2, 2}, {3, 3, 0}, {3, 3, 1}, {3, 4, 0}, {3, 5, 0}, {3, 5, 1}, {3, 6, 1},
    {3, 7, 2}, {3, 8, 2},
    // B
    {0, 0, 4}, {0, 0, 5}, {0, 1, 5}, {0, 1, 6}, {0, 2, 7}, {0, 2, 8}, {0, 4, 4}, {0, 5, 5}, {0, 6, 6},
    {0, 7, 7}, {0, 8, 8}, {0, 9, 9},
    // B, Re only
    {0, 0, 0}, {0, 1, 1}, {0, 2, 2}, {0, 3, 0}, {0, 3, 1}, {0, 4, 0}, {0, 5, 0}, {0, 5, 1}, {0, 6, 1},
    {0, 7, 2}, {0, 8, 2},
    // B, FENE only
    {0, 0, 6}, {0, 0, 9}, {0, 1, 4}, {0, 1, 9}, {0, 4, 6}, {0, 4, 9}, {0, 5, 4}, {0, 5, 6}, {0, 5, 9},
    {0, 6, 4}, {0, 6, 9}, {0, 9, 4}, {0, 9, 6}};

// Values the coefficients of one unit quantity are made of.
struct PlUnit {
    double C11, C12, C22, C33;       // constitutive residual
    double M1, M2;                   // momentum residual
    double P11, P12, P22, div, conv1, conv2;
};

// flag = 1 when any base value lies out of the plane (a NaN counts)
__global__ void k_nonplanar(int nnodes, const double *__restrict__ TLb, int *flag)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnodes) return;
    bool any = TLb[(size_t)2 * nnodes + i] != 0.0;
    for (int f = 7; f < 10; f++) any |= TLb[(size_t)f * nnodes + i] != 0.0;
    if (any) *flag = 1;
}

constexpr int PC_EL = 14, PC_THREADS = 128;   // 14 elements x 9 points: 126 of 128 lanes

__global__ void __launch_bounds__(PC_THREADS)
k_planar_coef(const StabArgs a, const KParams prm, double *__restrict__ rec)
{
    __shared__ double s_tlb[PC_EL][9 * ST_NEQ];
    const int t = threadIdx.x, e0 = blockIdx.x * PC_EL;
    for (int u = t; u < PC_EL * 9 * ST_NEQ; u += PC_THREADS) {
        const int el = u / (9 * ST_NEQ), q = u % (9 * ST_NEQ);
        if (e0 + el < a.nel)
            s_tlb[el][q] = a.TLb[(size_t)(q % ST_NEQ) * a.nnodes + a.conn[(q / ST_NEQ) * a.nel + e0 + el]];
    }
    __syncthreads();
    const int el = t / 9, gp = t % 9, e = e0 + el;
    if (el >= PC_EL || e >= a.nel) return;
    double *r = rec + ((size_t)e * 9 + gp) * PL_REC;
    StabBase b;
    {
        double x[9], y[9], fx[9], fy[9], sx[9], sy[9];
        for (int n = 0; n < 9; n++) {
            const int gn = a.conn[n * a.nel + e];
            x[n] = a.xy[gn];
            y[n] = a.xy[a.nnodes + gn];
        }
        const auto go = geometry(s_bfn[gp], s_dfdc[gp], s_dfde[gp], s_d2c[gp], s_d2e[gp], s_d2ce[gp], s_w[gp], x, y,
                                 fx, fy, sx, sy);
        for (int n = 0; n < 9; n++) {
            r[PL_OG + n] = fx[n];
            r[PL_OG + 9 + n] = fy[n];
            r[PL_OG + 18 + n] = sx[n] + sy[n];
        }
        stab_base(prm, s_tlb[el], fx, fy, sx, sy, go.H2, go.WET, gp, b);
    }
    const double W = b.WET, Wi = prm.WiN, be = prm.BvN, om = 1.0 - prm.BvN, Re = prm.ReN, Df = prm.DfN, VeN = prm.VeN;
    const double z = a.kz ? 1.0 : 0.0;
    const double U1 = b.U[0], U2 = b.U[1];
    const double g11 = b.GU[0][0], g21 = b.GU[1][0], g12 = b.GU[0][1], g22 = b.GU[1][1];
    const double S11 = b.S[0][0], S12 = b.S[0][1], S22 = b.S[1][1];
    const double X11 = b.dT[0][0][0], X12 = b.dT[0][1][0], X22 = b.dT[1][1][0];
    const double Y11 = b.dT[0][0][1], Y12 = b.dT[0][1][1], Y22 = b.dT[1][1][1];
    const double f0 = b.f[0], f1 = b.f[1], f2 = b.f[2];
    const double tm = b.tlsme, tc = b.tlsce, a1 = tm * Re * U1, a2 = tm * Re * U2;
    const double b1 = tc * Wi * U1, b2 = tc * Wi * U2, to = tm * om;
    const double md = b.tdcs / (2.0 * b.mag + 1.0e-12);   // tdcs x magnitude derivative per CE : CE'
    const double c33 = -2.0 * om * f0;                    // CE'(3,3) per K u3
    // f_T and what follows from it per unit trace of the stress perturbation
    const bool fene = prm.model == FENE_CR || prm.model == FENE_P;
    double cT = 0.0;
    if (prm.model == L_PTT || prm.model == M_L_PTT) cT = VeN * Wi / om;
    else if (prm.model == E_PTT || prm.model == M_E_PTT) cT = b.fT * VeN * Wi / om;
    else if (prm.model == FENE_CR) cT = Wi / om / (VeN - 2.0);
    else if (prm.model == FENE_P) cT = Wi / om / VeN;
    const bool mod = prm.model == M_L_PTT || prm.model == M_E_PTT || prm.model == FENE_CR;
    const double h0 = mod ? cT : 0.0;                     // f_0' per trace
    double h1 = prm.model == GIESEKUS ? 0.0 : cT;         // f_1' per trace, trace_x, trace_y, u1, u2
    double h1x = 0.0, h1y = 0.0, h1u = 0.0, h1v = 0.0;
    double tI = 0.0, tIx = 0.0, tIy = 0.0, tIu = 0.0, tIv = 0.0, tIt = 0.0;
    if (fene) {
        const double kap = Wi / om / (prm.model == FENE_P ? VeN : VeN - 2.0);
        const double d1 = kap * (X11 + X22), d2 = kap * (Y11 + Y22);      // grad f_T of the base
        const double mv = -(cT / b.fT) * (U1 * d1 + U2 * d2);
        h1 -= Wi * mv / b.fT;
        h1x = -Wi * (U1 * kap) / b.fT;
        h1y = -Wi * (U2 * kap) / b.fT;
        h1u = -Wi * d1 / b.fT;
        h1v = -Wi * d2 / b.fT;
        if (prm.model == FENE_P) {
            tI = mv / b.fT;
            tIx = U1 * kap / b.fT;
            tIy = U2 * kap / b.fT;
            tIu = d1 / b.fT;
            tIv = d2 / b.fT;
            tIt = -om * cT / b.fT;
        }
    }
    // coefficients of the in-plane equations for one unit quantity: component s
    // of unknown f; dx, dy: the quantity is the x or y derivative of stress
    // component dc (diffusion term)
    auto emit = [&](int f, int s, const PlUnit &u, int dc, double dx, double dy) {
        const double mg = md * (b.CE[0][0] * u.C11 + (b.CE[0][1] + b.CE[1][0]) * u.C12 + b.CE[1][1] * u.C22
                                + b.CE[2][2] * u.C33);
        auto put = [&](int e, double k0, double k1, double k2) {
            double *d;
            int np;
            const int eq = e < 2 ? e : e - 1;                           // 0 1 3 4 5 6 -> 0..5
            if (f < 2) {
                d = r + s * 3 * PL_NV + (e == 9 ? 15 + f : f * 6 + eq);
                np = PL_NV;
            } else {
                int at;
                if (e == 9) at = f == 9 ? 29 : 38 + (f - 4);
                else if (f == 9) at = 24 + (e < 2 ? e : e - 2);         // 0 1 4 5 6 -> 0..4
                else at = (f - 3) * 6 + eq;
                d = r + PL_OS + s * 3 * PL_NS + at;
                np = PL_NS;
            }
            d[0] = W * k0;
            d[np] = W * k1;
            d[2 * np] = W * k2;
        };
        put(0, Re * u.conv1, u.P11 + a1 * u.M1 + b.tlsic * u.div - tc * u.C11, u.P12 + a2 * u.M1 - tc * u.C12);
        put(1, Re * u.conv2, u.P12 + a1 * u.M2 - tc * u.C12, u.P22 + a2 * u.M2 + b.tlsic * u.div - tc * u.C22);
        if (f != 9) put(3, u.div, tm * u.M1, tm * u.M2);
        put(4, u.C11, (dc == 4 ? Df * dx : 0.0) - to * u.M1 + b1 * u.C11 + X11 * mg,
            (dc == 4 ? Df * dy : 0.0) + b2 * u.C11 + Y11 * mg);
        put(5, u.C12, (dc == 5 ? Df * dx : 0.0) - to * u.M2 + b1 * u.C12 + X12 * mg,
            (dc == 5 ? Df * dy : 0.0) - to * u.M1 + b2 * u.C12 + Y12 * mg);
        put(6, u.C22, (dc == 6 ? Df * dx : 0.0) + b1 * u.C22 + X22 * mg,
            (dc == 6 ? Df * dy : 0.0) - to * u.M2 + b2 * u.C22 + Y22 * mg);
        if (f != 3) put(9, u.C33, (dc == 9 ? Df * dx : 0.0) + b1 * u.C33, (dc == 9 ? Df * dy : 0.0) + b2 * u.C33);
    };
    {   // u1: value, x, y, Laplacian
        PlUnit u = {Wi * X11 + h1u * S11 - om * tIu, Wi * X12 + h1u * S12, Wi * X22 + h1u * S22 - om * tIu, -om * tIu,
                    Re * g11, Re * g12, 0.0, 0.0, 0.0, 0.0, g11, g12};
        emit(0, 0, u, -1, 0.0, 0.0);
        u = {-2.0 * (Wi * S11 + om * f0), -Wi * S12, 0.0, 0.0, Re * U1, 0.0, 2.0 * be, 0.0, 0.0, 1.0, U1, 0.0};
        emit(0, 1, u, -1, 0.0, 0.0);
        u = {-2.0 * Wi * S12, -Wi * S22 - om * f0, 0.0, 0.0, Re * U2, 0.0, 0.0, be, 0.0, 0.0, U2, 0.0};
        emit(0, 2, u, -1, 0.0, 0.0);
        u = {0.0, 0.0, 0.0, 0.0, -be, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        emit(0, 3, u, -1, 0.0, 0.0);
        // u2
        u = {Wi * Y11 + h1v * S11 - om * tIv, Wi * Y12 + h1v * S12, Wi * Y22 + h1v * S22 - om * tIv, -om * tIv,
             Re * g21, Re * g22, 0.0, 0.0, 0.0, 0.0, g21, g22};
        emit(1, 0, u, -1, 0.0, 0.0);
        u = {0.0, -Wi * S11 - om * f0, -2.0 * Wi * S12, 0.0, 0.0, Re * U1, 0.0, be, 0.0, 0.0, 0.0, U1};
        emit(1, 1, u, -1, 0.0, 0.0);
        u = {0.0, -Wi * S12, -2.0 * (Wi * S22 + om * f0), 0.0, 0.0, Re * U2, 0.0, 0.0, 2.0 * be, 1.0, 0.0, U2};
        emit(1, 2, u, -1, 0.0, 0.0);
        u = {0.0, 0.0, 0.0, 0.0, 0.0, -be, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        emit(1, 3, u, -1, 0.0, 0.0);
        // p
        u = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, -1.0, 0.0, -1.0, 0.0, 0.0, 0.0};
        emit(3, 0, u, -1, 0.0, 0.0);
        u = {0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        emit(3, 1, u, -1, 0.0, 0.0);
        u = {0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        emit(3, 2, u, -1, 0.0, 0.0);
        // stresses: the trace part of s11, s22, s33 first
        const double t11 = h1 * S11 - om * (2.0 * h0 * g11 + tI), t12 = h1 * S12 - om * h0 * (g12 + g21);
        const double t22 = h1 * S22 - om * (2.0 * h0 * g22 + tI), t33 = -om * tI;
        u = {t11 - 2.0 * Wi * g11 + 2.0 * f2 * S11 + f1, t12 - Wi * g12 + f2 * S12, t22, t33, 0.0, 0.0, 1.0, 0.0, 0.0,
             0.0, 0.0, 0.0};
        emit(4, 0, u, -1, 0.0, 0.0);
        u = {-2.0 * Wi * g21 + 2.0 * f2 * S12, -Wi * (g11 + g22) + f2 * (S11 + S22) + f1,
             -2.0 * Wi * g12 + 2.0 * f2 * S12, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0};
        emit(5, 0, u, -1, 0.0, 0.0);
        u = {t11, t12 - Wi * g21 + f2 * S12, t22 - 2.0 * Wi * g22 + 2.0 * f2 * S22 + f1, t33, 0.0, 0.0, 0.0, 0.0, 1.0,
             0.0, 0.0, 0.0};
        emit(6, 0, u, -1, 0.0, 0.0);
        u = {t11, t12, t22, t33 + f1, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        emit(9, 0, u, -1, 0.0, 0.0);
        // their x and y derivatives
        for (int s = 1; s <= 2; s++) {
            const double wu = Wi * (s == 1 ? U1 : U2), hx = s == 1 ? h1x : h1y, ix = om * (s == 1 ? tIx : tIy);
            const double q11 = hx * S11 - ix, q12 = hx * S12, q22 = hx * S22 - ix;
            const double dx = s == 1 ? 1.0 : 0.0, dy = 1.0 - dx;
            u = {wu + q11, q12, q22, -ix, -dx, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            emit(4, s, u, 4, dx, dy);
            u = {0.0, wu, 0.0, 0.0, -dy, -dx, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            emit(5, s, u, 5, dx, dy);
            u = {q11, q12, wu + q22, -ix, 0.0, -dy, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            emit(6, s, u, 6, dx, dy);
            u = {q11, q12, q22, wu - ix, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            emit(9, s, u, 9, dx, dy);
        }
    }
    // out-of-plane unknowns in A0: m3, 13, 23 per (C13, C23, M3, P13, P23, conv3)
    auto emit3 = [&](double *d, int np, int stride, double C13, double C23, double M3, double P13, double P23,
                     double conv3, double d13x, double d13y, double d23x, double d23y) {
        const double k[3][3] = {{Re * conv3, P13 + a1 * M3 - tc * C13, P23 + a2 * M3 - tc * C23},
                                {C13, Df * d13x - to * M3 + b1 * C13, Df * d13y + b2 * C13},
                                {C23, Df * d23x + b1 * C23, Df * d23y - to * M3 + b2 * C23}};
        for (int e = 0; e < 3; e++)
            for (int c = 0; c < 3; c++) d[c * np + e * stride] = W * k[e][c];
    };
    {
        double *v = r + 12;                              // u3
        emit3(v, PL_NV, 1, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
        emit3(v + 3 * PL_NV, PL_NV, 1, -Wi * S11 - om * f0, -Wi * S12, Re * U1, be, 0.0, U1, 0.0, 0.0, 0.0, 0.0);
        emit3(v + 6 * PL_NV, PL_NV, 1, -Wi * S12, -Wi * S22 - om * f0, Re * U2, 0.0, be, U2, 0.0, 0.0, 0.0, 0.0);
        emit3(v + 9 * PL_NV, PL_NV, 1, 0.0, 0.0, -be, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
        double *q = r + PL_OS + 30;                      // s13, then s23
        emit3(q, PL_NS, 1, -Wi * g11 + f2 * S11 + f1, -Wi * g12 + f2 * S12, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0);
        emit3(q + 3 * PL_NS, PL_NS, 1, Wi * U1, 0.0, -1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0);
        emit3(q + 6 * PL_NS, PL_NS, 1, Wi * U2, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0);
        q += 3;
        emit3(q, PL_NS, 1, -Wi * g21 + f2 * S12, -Wi * g22 + f2 * S22 + f1, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0);
        emit3(q + 3 * PL_NS, PL_NS, 1, 0.0, Wi * U1, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0);
        emit3(q + 6 * PL_NS, PL_NS, 1, 0.0, Wi * U2, -1.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0);
        // A1: u3 in m1 and m2 (its x or y derivative in the value term, its value in the gradient terms)
        for (int i = 0; i < 2; i++) {
            double *d = r + PL_OS + 36 + i;
            for (int c = 0; c < 9; c++) d[c * PL_NS] = 0.0;
            d[(1 + i) * 3 * PL_NS] = -W * be;
            d[(1 + i) * PL_NS] = W * z * b.tlsic;
        }
    }
    // value type
    auto val = [&](int i, double k0, double k1, double k2) {
        double *d = r + PL_OM + i;
        d[0] = W * k0;
        d[PL_NM] = W * k1;
        d[2 * PL_NM] = W * k2;
    };
    const double mg3 = md * b.CE[2][2] * c33, of = om * f0;
    val(0, -1.0, -z * a1, -z * a2);
    val(1, -1.0, -z * a1, -z * a2);
    val(2, 0.0, -z * (be + tc * of), 0.0);
    val(3, 0.0, 0.0, -z * (be + tc * of));
    val(4, -1.0, -z * a1, -z * a2);
    val(5, 1.0, z * a1, z * a2);
    val(6, z, 0.0, 0.0);
    val(7, 0.0, -z * tm, 0.0);
    val(8, 0.0, 0.0, -z * tm);
    val(9, 0.0, z * to, 0.0);
    val(10, 0.0, z * X11 * mg3, z * Y11 * mg3);
    val(11, 0.0, 0.0, z * to);
    val(12, 0.0, z * to, 0.0);
    val(13, 0.0, z * X12 * mg3, z * Y12 * mg3);
    val(14, 0.0, 0.0, z * to);
    val(15, 0.0, z * X22 * mg3, z * Y22 * mg3);
    val(16, z * c33, z * b1 * c33, z * b2 * c33);
    val(17, z * of, z * b1 * of, z * b2 * of);
    val(18, 0.0, z * to, 0.0);
    val(19, 0.0, -z * to, 0.0);
    val(20, z * of, z * b1 * of, z * b2 * of);
    val(21, 0.0, 0.0, z * to);
    val(22, 0.0, 0.0, -z * to);
    const double zb = z * be, zt = -z * to * be;
    val(23, zb, a1 * zb, a2 * zb);
    val(24, zb, a1 * zb, a2 * zb);
    val(25, 2.0 * zb, a1 * zb, a2 * zb);
    val(26, 0.0, tm * zb, 0.0);
    val(27, 0.0, 0.0, tm * zb);
    val(28, 0.0, zt, 0.0);
    val(29, 0.0, 0.0, zt);
    val(30, 0.0, zt, 0.0);
    val(31, 0.0, 0.0, zt);
    val(32, 0.0, zt, 0.0);
    val(33, 0.0, 0.0, zt);
    // B (its sign: TERM_RES_b = -TERM_RES_b); w: the FENE part per trace
    const double w0 = fene ? -Wi * cT / b.fT : 0.0;
    const double w11 = w0 * S11 + tIt, w12 = w0 * S12, w22 = w0 * S22 + tIt;
    auto mom = [&](int i, double c1, double c2) { val(i, 0.0, tc * c1, tc * c2); };
    auto str = [&](int i, double c) { val(i, -c, -b1 * c, -b2 * c); };
    mom(34, Wi + w11, w12);
    mom(35, 0.0, Wi);
    mom(36, Wi, 0.0);
    mom(37, w12, Wi + w22);
    mom(38, Wi, 0.0);
    mom(39, 0.0, Wi);
    str(40, Wi + w11);
    str(41, Wi);
    str(42, Wi + w22);
    str(43, Wi);
    str(44, Wi);
    str(45, Wi + tIt);
    val(46, -Re, -a1 * Re, -a2 * Re);
    val(47, -Re, -a1 * Re, -a2 * Re);
    val(48, -Re, -a1 * Re, -a2 * Re);
    val(49, 0.0, -tm * Re, 0.0);
    val(50, 0.0, 0.0, -tm * Re);
    val(51, 0.0, to * Re, 0.0);
    val(52, 0.0, 0.0, to * Re);
    val(53, 0.0, to * Re, 0.0);
    val(54, 0.0, 0.0, to * Re);
    val(55, 0.0, to * Re, 0.0);
    val(56, 0.0, 0.0, to * Re);
    mom(57, w11, w12);
    mom(58, w11, w12);
    mom(59, w12, w22);
    mom(60, w12, w22);
    str(61, w11);
    str(62, w11);
    str(63, w12);
    str(64, w12);
    str(65, w12);
    str(66, w22);
    str(67, w22);
    str(68, tIt);
    str(69, tIt);
}

constexpr int PK_WARPS = 8;

// One (test node, pair) of an element: 9 trial nodes, NS components
template <int NS>
__device__ __forceinline__ void planar_pair(const double *__restrict__ rec, const double *__restrict__ phi,
                                            int off, int np, int pair, int i, double *__restrict__ out)
{
    double acc[9];
#pragma unroll
    for (int j = 0; j < 9; j++) acc[j] = 0.0;
#pragma unroll 1
    for (int gp = 0; gp < 9; gp++) {
        const double *r = rec + gp * PL_REC, *d = r + off + pair, *g = r + PL_OG, *p = phi + gp * 9;
        const double p0 = p[i], p1 = g[i], p2 = g[9 + i];
        double c[NS];
#pragma unroll
        for (int s = 0; s < NS; s++)
            c[s] = p0 * d[(3 * s) * np] + p1 * d[(3 * s + 1) * np] + p2 * d[(3 * s + 2) * np];
#pragma unroll
        for (int j = 0; j < 9; j++) {
            acc[j] += c[0] * p[j];
            if constexpr (NS > 1) acc[j] += c[1] * g[j];
            if constexpr (NS > 2) acc[j] += c[2] * g[9 + j];
            if constexpr (NS > 3) acc[j] += c[3] * g[18 + j];
        }
    }
#pragma unroll
    for (int j = 0; j < 9; j++) out[(size_t)(i * 9 + j) * PL_NP] = acc[j];
}

// A CTA per element: its records in shared memory, a lane per (test node,
// pair), the lanes of a warp on one type.  40 multiply-adds per Gauss point and
// lane against ~50 shared loads, most of them broadcasts: an FP64 instruction
// holds the pipe for 16 clocks of the SM, so the loads hide.
__global__ void __launch_bounds__(PK_WARPS * 32)
k_planar_contract(const double *__restrict__ rec_all, double *__restrict__ es, int nv, int ns, int nm)
{
    extern __shared__ __align__(16) double rec[];
    __shared__ double phi[81];
    const double2 *src = reinterpret_cast<const double2 *>(rec_all + (size_t)blockIdx.x * 9 * PL_REC);
    for (int u = threadIdx.x; u < 9 * PL_REC / 2; u += PK_WARPS * 32) reinterpret_cast<double2 *>(rec)[u] = src[u];
    if (threadIdx.x < 81) phi[threadIdx.x] = s_bfn[threadIdx.x / 9][threadIdx.x % 9];
    __syncthreads();
    double *out = es + (size_t)blockIdx.x * PL_OUT;
    const int lane = threadIdx.x & 31;
    const int wv = (nv * 9 + 31) / 32, ws = (ns * 9 + 31) / 32, wm = (nm * 9 + 31) / 32;
    for (int w = threadIdx.x >> 5; w < wv + ws + wm; w += PK_WARPS) {
        if (w < wv) {
            const int k = w * 32 + lane;
            if (k < nv * 9) planar_pair<4>(rec, phi, 0, PL_NV, k % nv, k / nv, out + k % nv);
        } else if (w < wv + ws) {
            const int k = (w - wv) * 32 + lane;
            if (k < ns * 9) planar_pair<3>(rec, phi, PL_OS, PL_NS, k % ns, k / ns, out + PL_NV + k % ns);
        } else {
            const int k = (w - wv - ws) * 32 + lane;
            if (k < nm * 9) planar_pair<1>(rec, phi, PL_OM, PL_NM, k % nm, k / nm, out + PL_NV + PL_NS + k % nm);
        }
    }
}

// Where a pair's sum goes: B or A0 at equation x unknown `r`, or the K (pw 1) or
// K^2 (pw 2) part of the `dep`-th of the 36 entries of a block that depend on K.
constexpr int PL_DEP = 36;
struct PlMap {
    unsigned char n;                               // pairs that are not identically zero
    unsigned char pair[PL_NP], m[PL_NP], at[PL_NP]; // pair; matrix; r or dep
    unsigned char dr[PL_DEP], dpw[PL_DEP];
};

constexpr int PG_THREADS = 256, PG_BLK = 16;       // node-pair blocks at a time
constexpr int PG_OWN = (PG_BLK * 100 + PG_THREADS - 1) / PG_THREADS;       // entries per thread
constexpr int PG_DEP = (PG_BLK * PL_DEP + PG_THREADS - 1) / PG_THREADS;    // K-dependent ones

// Scatter: a CTA per row node sums its blocks' pairs in element order and writes
// its 10 rows of B and of A(K) for every wavenumber.  Only 36 of a block's 100
// entries depend on K, in one power each: they are evaluated on full warps into
// shared memory (a thread per entry, K in two multiply-adds whatever the entry
// holds, spent 6.5 ms of FP64 pipe on 20,000 quads x 16 wavenumbers, more than
// the 2.6 ms of writing 17.5 GB), and the rows are written from there in the
// order they are stored.  store: leave out reading the matrices.
// Scatter of that case 9.2 -> 5.1 ms, the call 18.6 -> 14.5 ms.
__global__ void __launch_bounds__(PG_THREADS)
k_planar_gather(const GatherArgs g, const PlMap map, const int64_t *__restrict__ rowptr10,
                const int32_t *__restrict__ boff10, const double *__restrict__ es, int nk,
                const double *__restrict__ kw, double *const *__restrict__ A, double *__restrict__ B, int store)
{
    __shared__ PlMap s_map;
    __shared__ double s_v[PG_BLK * 100], s_b[PG_BLK * 100], s_x[PG_BLK * PL_DEP];
    __shared__ int s_id[PG_BLK][4], s_n[PG_BLK], s_c0[PG_BLK], s_off[PG_BLK];
    __shared__ int64_t s_row[ST_NEQ];
    const int t = threadIdx.x;
    for (int u = t; u < (int)sizeof(PlMap); u += PG_THREADS)
        reinterpret_cast<unsigned char *>(&s_map)[u] = reinterpret_cast<const unsigned char *>(&map)[u];
    if (t < ST_NEQ) s_row[t] = rowptr10[(int64_t)blockIdx.x * ST_NEQ + t];
    const int b1 = g.nbptr[blockIdx.x + 1];
    for (int b0 = g.nbptr[blockIdx.x]; b0 < b1; b0 += PG_BLK) {
        const int nb = min(PG_BLK, b1 - b0), wide = nb * ST_NEQ, count = nb * 100;
        __syncthreads();
        if (t < nb) {
            const int4 *rp = reinterpret_cast<const int4 *>(g.brec + b0 + t);
            const int4 head = rp[0], ids = rp[1];
            s_c0[t] = head.z;
            s_n[t] = head.w;
            s_off[t] = boff10[b0 + t];
            s_id[t][0] = ids.x; s_id[t][1] = ids.y; s_id[t][2] = ids.z; s_id[t][3] = ids.w;
        }
        for (int i = t; i < count; i += PG_THREADS) s_v[i] = s_b[i] = 0.0;
        __syncthreads();
        const int np = s_map.n;
        for (int i = t; i < nb * np; i += PG_THREADS) {
            const int b = i / np, q = i - b * np, n = s_n[b];
            const double *src = es + s_map.pair[q];
            double x = 0.0;
            for (int k = 0; k < n; k++)
                x += src[(size_t)(k < 4 ? s_id[b][k] : g.bcon[s_c0[b] + k]) * PL_NP];
            const int m = s_map.m[q], at = s_map.at[q];
            if (m >= 2)
                s_x[b * PL_DEP + at] = x;
            else
                (m == 0 ? s_b : s_v)[at / ST_NEQ * wide + b * ST_NEQ + at % ST_NEQ] = x;
        }
        __syncthreads();
        int64_t slot[PG_OWN];
#pragma unroll
        for (int u = 0; u < PG_OWN; u++) {
            const int i = t + u * PG_THREADS;
            if (i >= count) continue;
            const int jeq = i / wide, c = i - jeq * wide, b = c / ST_NEQ;
            slot[u] = s_row[jeq] + s_off[b] + c - b * ST_NEQ;
            if (B) B[slot[u]] = store ? s_b[i] : B[slot[u]] + s_b[i];
        }
        int at[PG_DEP];
        double v0[PG_DEP], vx[PG_DEP];
        bool sq[PG_DEP];
#pragma unroll
        for (int u = 0; u < PG_DEP; u++) {
            const int d = t + u * PG_THREADS;
            at[u] = -1;
            if (d >= nb * PL_DEP) continue;
            const int b = d / PL_DEP, j = d - b * PL_DEP, r = s_map.dr[j];
            at[u] = r / ST_NEQ * wide + b * ST_NEQ + r % ST_NEQ;
            v0[u] = s_v[at[u]];
            vx[u] = s_x[d];
            sq[u] = s_map.dpw[j] == 2;
        }
        for (int k = 0; k < nk; k++) {
            const double K = kw[k], K2 = K * K;
            double *Ak = A[k];
            __syncthreads();
#pragma unroll
            for (int u = 0; u < PG_DEP; u++)
                if (at[u] >= 0) s_v[at[u]] = __fma_rn(sq[u] ? K2 : K, vx[u], v0[u]);
            __syncthreads();
#pragma unroll
            for (int u = 0; u < PG_OWN; u++) {
                const int i = t + u * PG_THREADS;
                if (i < count) Ak[slot[u]] = store ? s_v[i] : Ak[slot[u]] + s_v[i];
            }
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side

__global__ void k_boff10(int n, const int32_t *__restrict__ boff6, int32_t *__restrict__ boff10)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) boff10[i] = boff6[i] / 6 * 10;
}

cudaError_t stab_upload_tables(const GaussTables &t, cudaStream_t s)
{
    cudaError_t e = cudaSuccess;
#define UP(sym, src)                                                                       \
    if (e == cudaSuccess) e = cudaMemcpyToSymbolAsync(sym, src, sizeof(src), 0, cudaMemcpyHostToDevice, s);
    UP(s_w, t.w)
    UP(s_bfn, t.bfn)
    UP(s_dfdc, t.dfdc)
    UP(s_dfde, t.dfde)
    UP(s_d2c, t.d2fdc2)
    UP(s_d2e, t.d2fde2)
    UP(s_d2ce, t.d2fdce)
#undef UP
    return e;
}

}  // namespace vefem

using namespace vefem;

namespace {

int sfail(vefem_ctx *c, int code, const std::string &m)
{
    c->err = m;
    return code;
}

#define SCK(call)                                                                          \
    do {                                                                                   \
        cudaError_t _e = (call);                                                           \
        if (_e != cudaSuccess)                                                             \
            return sfail(ctx, VEFEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

// The 10-unknown pattern from the frozen 6-unknown one: every node-pair block
// becomes a 10 x 10 block, the extra (arclength) columns and rows are dropped.
int stab_pattern(vefem_ctx *ctx)
{
    if (!ctx->h_rowptr10.empty()) return VEFEM_OK;
    const int64_t nn = ctx->nnodes;
    std::vector<int64_t> rp(nn * ST_NEQ + 1, 0);
    std::vector<int32_t> ci;
    for (int64_t n = 0; n < nn; n++) {
        const int64_t r0 = ctx->h_rowptr[n * 6], r1 = ctx->h_rowptr[n * 6 + 1];
        std::vector<int32_t> cols;
        for (int64_t s = r0; s < r1; s++) {
            const int32_t c = ctx->h_colind[s];
            if (c < nn * 6 && c % 6 == 0) cols.push_back(c / 6);
        }
        for (int q = 0; q < ST_NEQ; q++) {
            for (int32_t cn : cols)
                for (int f = 0; f < ST_NEQ; f++) ci.push_back(cn * ST_NEQ + f);
            rp[n * ST_NEQ + q + 1] = (int64_t)ci.size();
        }
    }
    ctx->h_rowptr10.swap(rp);
    ctx->h_colind10.swap(ci);
    SCK(cudaMalloc((void **)&ctx->d_rowptr10, ctx->h_rowptr10.size() * sizeof(int64_t)));
    SCK(cudaMemcpy(ctx->d_rowptr10, ctx->h_rowptr10.data(), ctx->h_rowptr10.size() * sizeof(int64_t),
                   cudaMemcpyHostToDevice));
    SCK(cudaMalloc((void **)&ctx->d_boff10, std::max(1, ctx->nblocks) * sizeof(int32_t)));
    if (ctx->nblocks > 0)
        k_boff10<<<(ctx->nblocks + 255) / 256, 256, 0, ctx->stream>>>(ctx->nblocks, ctx->d_boff, ctx->d_boff10);
    SCK(cudaGetLastError());
    SCK(cudaStreamSynchronize(ctx->stream));
    return VEFEM_OK;
}

}  // namespace

extern "C" int vefem_stability_pattern(vefem_ctx *ctx, int64_t *n, int64_t *nnz, int64_t *rowptr,
                                       int32_t *colind)
{
    if (!ctx || !n || !nnz) return VEFEM_ERR_ARG;
    SCK(cudaSetDevice(ctx->device));
    if (int rc = stab_pattern(ctx)) return rc;
    *n = (int64_t)ctx->h_rowptr10.size() - 1;
    *nnz = (int64_t)ctx->h_colind10.size();
    if (rowptr) std::copy(ctx->h_rowptr10.begin(), ctx->h_rowptr10.end(), rowptr);
    if (colind) std::copy(ctx->h_colind10.begin(), ctx->h_colind10.end(), colind);
    return VEFEM_OK;
}

extern "C" int vefem_stability_assemble(vefem_ctx *ctx, const double *TLb, int nk, const double *kw,
                                        int flags, double *const *A, double *B, int on_device)
{
    if (!ctx) return VEFEM_ERR_ARG;
    const int known = VEFEM_ZERO_FIRST | VEFEM_STAB_AS_WRITTEN;
    if (flags & ~known) return sfail(ctx, VEFEM_ERR_UNSUPPORTED, "unknown flag");
    if (!TLb || nk < 0 || (nk > 0 && (!kw || !A))) return sfail(ctx, VEFEM_ERR_ARG, "NULL argument");
    for (int k = 0; k < nk; k++)
        if (!A[k]) return sfail(ctx, VEFEM_ERR_ARG, "NULL A array");
    if (ctx->prm.form != FORM_T)
        return sfail(ctx, VEFEM_ERR_UNSUPPORTED, "stability assembly: T form only");
    SCK(cudaSetDevice(ctx->device));
    if (int rc = stab_pattern(ctx)) return rc;
    cudaStream_t s = ctx->stream;
    const int64_t N10 = (int64_t)ctx->nnodes * ST_NEQ, nnz10 = (int64_t)ctx->h_colind10.size();
    if (!ctx->d_nonplanar) SCK(cudaMalloc((void **)&ctx->d_nonplanar, sizeof(int)));
    if (!ctx->d_tlb) {
        SCK(cudaMalloc((void **)&ctx->d_tlb, (size_t)N10 * sizeof(double)));
        GaussTables gt;
        gauss_tables_host(&gt);
        SCK(stab_upload_tables(gt, s));
    }
    if (nk > ctx->stab_nk) {
        cudaFree(ctx->d_kw);
        cudaFree(ctx->d_Aptr);
        SCK(cudaMalloc((void **)&ctx->d_kw, nk * sizeof(double)));
        SCK(cudaMalloc((void **)&ctx->d_Aptr, nk * sizeof(double *)));
        ctx->stab_nk = nk;
    }
    // device pointers of the outputs (host buffers: staging arrays)
    std::vector<double *> dA(nk);
    double *dB = B;
    if (!on_device) {
        if (nk > ctx->stab_nk_stage) {
            cudaFree(ctx->d_Astage);
            SCK(cudaMalloc((void **)&ctx->d_Astage, (size_t)nk * nnz10 * sizeof(double)));
            ctx->stab_nk_stage = nk;
        }
        if (B && !ctx->d_Bstage) SCK(cudaMalloc((void **)&ctx->d_Bstage, (size_t)nnz10 * sizeof(double)));
        for (int k = 0; k < nk; k++) dA[k] = ctx->d_Astage + (size_t)k * nnz10;
        dB = B ? ctx->d_Bstage : nullptr;
        SCK(cudaMemcpyAsync(ctx->d_tlb, TLb, N10 * sizeof(double), cudaMemcpyHostToDevice, s));
        if (!(flags & VEFEM_ZERO_FIRST)) {
            for (int k = 0; k < nk; k++)
                SCK(cudaMemcpyAsync(dA[k], A[k], nnz10 * sizeof(double), cudaMemcpyHostToDevice, s));
            if (B) SCK(cudaMemcpyAsync(dB, B, nnz10 * sizeof(double), cudaMemcpyHostToDevice, s));
        }
    } else {
        for (int k = 0; k < nk; k++) dA[k] = A[k];
        SCK(cudaMemcpyAsync(ctx->d_tlb, TLb, N10 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    }
    // a base state in the plane takes the sparse kernels, any other the general one
    int nonplanar = 0;
    SCK(cudaMemsetAsync(ctx->d_nonplanar, 0, sizeof(int), s));
    k_nonplanar<<<(ctx->nnodes + 255) / 256, 256, 0, s>>>(ctx->nnodes, ctx->d_tlb, ctx->d_nonplanar);
    SCK(cudaGetLastError());
    SCK(cudaMemcpyAsync(&nonplanar, ctx->d_nonplanar, sizeof(int), cudaMemcpyDeviceToHost, s));
    SCK(cudaStreamSynchronize(s));
    const bool cover = nnz10 == (int64_t)ctx->nblocks * 100;
    const bool store = (flags & VEFEM_ZERO_FIRST) && !nonplanar && cover;   // every entry written, none read
    if ((flags & VEFEM_ZERO_FIRST) && !store) {
        for (int k = 0; k < nk; k++) SCK(cudaMemsetAsync(dA[k], 0, nnz10 * sizeof(double), s));
        if (dB) SCK(cudaMemsetAsync(dB, 0, nnz10 * sizeof(double), s));
    }
    if (nk > 0) {
        SCK(cudaMemcpyAsync(ctx->d_kw, kw, nk * sizeof(double), on_device ? cudaMemcpyDeviceToDevice
                                                                          : cudaMemcpyHostToDevice, s));
        SCK(cudaMemcpyAsync(ctx->d_Aptr, dA.data(), nk * sizeof(double *), cudaMemcpyHostToDevice, s));
    }
    // element kernel
    StabArgs a;
    a.nel = ctx->nel;
    a.nnodes = ctx->nnodes;
    a.conn = ctx->d_conn;
    a.xy = ctx->d_xy;
    a.TLb = ctx->d_tlb;
    a.es = nullptr;
    a.kz = (flags & VEFEM_STAB_AS_WRITTEN) ? 0 : 1;
    GatherArgs g;
    g.nnodes = ctx->nnodes;
    g.nblocks = ctx->nblocks;
    g.nex = 0;
    g.rowptr = ctx->d_rowptr;
    g.nptr = ctx->d_nptr;
    g.ncon = ctx->d_ncon;
    g.nbptr = ctx->d_nbptr;
    g.brow = ctx->d_brow;
    g.boff = ctx->d_boff;
    g.bptr = ctx->d_bptr;
    g.bcon = ctx->d_bcon;
    g.brec = ctx->d_brec;
    ctx->launches = 1;
    const int64_t nthr = (int64_t)ctx->nblocks * 100;
    if (!nonplanar) {
        const bool fene = ctx->prm.model == FENE_CR || ctx->prm.model == FENE_P;
        const int nv = fene ? PL_NV : PL_NV0, ns = fene ? PL_NS : PL_NS0;
        const int nm = fene || ctx->prm.ReN != 0.0 ? PL_NM : PL_NM0;
        if (!ctx->d_prec) SCK(cudaMalloc((void **)&ctx->d_prec, (size_t)ctx->nel * 9 * PL_REC * sizeof(double)));
        if (!ctx->d_pes) SCK(cudaMalloc((void **)&ctx->d_pes, (size_t)ctx->nel * PL_OUT * sizeof(double)));
        PlMap map = {};
        int dep = 0;
        for (int q = 0; q < PL_NP; q++) {
            const bool on = q < PL_NV ? q < nv : (q < PL_NV + PL_NS ? q - PL_NV < ns : q - PL_NV - PL_NS < nm);
            if (!on) continue;
            const PlPair &pp = PL_PAIRS[q];
            const int k = map.n++, r = pp.e * ST_NEQ + pp.f;
            map.pair[k] = (unsigned char)q;
            map.m[k] = (unsigned char)pp.m;
            map.at[k] = (unsigned char)(pp.m >= 2 ? dep : r);
            if (pp.m >= 2) {
                map.dr[dep] = (unsigned char)r;
                map.dpw[dep++] = (unsigned char)(pp.m - 1);
            }
        }
        k_planar_coef<<<(ctx->nel + PC_EL - 1) / PC_EL, PC_THREADS, 0, s>>>(a, ctx->prm, ctx->d_prec);
        SCK(cudaGetLastError());
        const int smem = 9 * PL_REC * (int)sizeof(double);
        SCK(cudaFuncSetAttribute(k_planar_contract, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        k_planar_contract<<<ctx->nel, PK_WARPS * 32, smem, s>>>(ctx->d_prec, ctx->d_pes, nv, ns, nm);
        SCK(cudaGetLastError());
        k_planar_gather<<<ctx->nnodes, PG_THREADS, 0, s>>>(g, map, ctx->d_rowptr10, ctx->d_boff10, ctx->d_pes, nk,
                                                           ctx->d_kw, ctx->d_Aptr, dB, store);
        SCK(cudaGetLastError());
        ctx->launches += 3;
    } else {
        if (!ctx->d_ses) SCK(cudaMalloc((void **)&ctx->d_ses, (size_t)ctx->nel * 4 * ST_BLK * sizeof(double)));
        a.es = ctx->d_ses;
        const size_t smem = sizeof(double) * st_smem_doubles() + 9 * sizeof(StabBase);
        SCK(cudaFuncSetAttribute(k_stability, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int occ = 0;
        SCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_stability, ST_THREADS, smem));
        int sms = 0;
        SCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
        const int grid = std::min<int>(ctx->nel, sms * std::max(1, occ));
        if (ctx->nel > 0) {
            k_stability<<<grid, ST_THREADS, smem, s>>>(a, ctx->prm);
            SCK(cudaGetLastError());
            ctx->launches++;
        }
        if (nthr > 0) {
            k_stability_gather<<<(unsigned)((nthr + 255) / 256), 256, 0, s>>>(
                g, ctx->d_rowptr10, ctx->d_boff10, ctx->d_ses, nk, ctx->d_kw, ctx->d_Aptr, dB);
            SCK(cudaGetLastError());
            ctx->launches++;
        }
    }
    if (!on_device) {
        for (int k = 0; k < nk; k++)
            SCK(cudaMemcpyAsync(A[k], dA[k], nnz10 * sizeof(double), cudaMemcpyDeviceToHost, s));
        if (B) SCK(cudaMemcpyAsync(B, dB, nnz10 * sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    SCK(cudaStreamSynchronize(s));
    return VEFEM_OK;
}
