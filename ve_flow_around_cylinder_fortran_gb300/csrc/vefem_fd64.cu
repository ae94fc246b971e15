// FP64 element assembly kernels for sm_103a: residual and the reference's
// forward-difference Jacobian, bit-compatible with the sequential algorithm.
//
// This translation unit is compiled with -fmad=false: every multiply and add
// is a separately rounded IEEE binary64 operation, evaluated in the order the
// reference Fortran writes it, so residuals match the CPU restatement bit for
// bit and the FD Jacobian (differences divided by 1e-8) does too.  The 2-D
// Cylinder_2D problem (Ndim = 2, Neq = 6) is specialised: terms that the
// reference computes with a third dimension are exact zeros there and are
// left out, which changes no value.
//
// Kernel layout (GB300: FP64 is the scarce unit, so the work is arranged to
// spend FP64 operations only on what the algorithm needs):
//  * k_fd64: a thread per column of storeBulk's forward difference
//    (Equations_mod.F90:264-306), CTAs by the field that the columns perturb;
//    the base residual is k_res64's.  Terms that are exact zeros for Re = 0 or
//    DfN = 0 are left out by template specialisation.
//  * k_res64: residual only ('MNR'): one thread per (element, Gauss point),
//    followed by an in-order sum over the Gauss points in shared memory;
//    k_res64_wide: an element spread over a CTA, for small meshes.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "vefem_early.cuh"
#include "vefem_internal.h"
#include "vefem_physics.cuh"

namespace vefem {

__constant__ double c_w[9];
__constant__ double c_bfn[9][9];
__constant__ double c_dfdc[9][9];
__constant__ double c_dfde[9][9];
__constant__ double c_d2fdc2[9][9];
__constant__ double c_d2fde2[9][9];
__constant__ double c_d2fdce[9][9];
__constant__ double c_ew[3];
__constant__ double c_ebfn[4][3][9];
__constant__ double c_edfdc[4][3][9];
__constant__ double c_edfde[4][3][9];
__constant__ double c_ed2c[4][3][9];
__constant__ double c_ed2e[4][3][9];
__constant__ double c_ed2ce[4][3][9];

cudaError_t upload_tables(const GaussTables &t, cudaStream_t s)
{
    cudaError_t e = cudaSuccess;
#define UP(sym, src)                                                                       \
    if (e == cudaSuccess)                                                                  \
        e = cudaMemcpyToSymbolAsync(sym, src, sizeof(src), 0, cudaMemcpyHostToDevice, s);
    UP(c_w, t.w)
    UP(c_bfn, t.bfn)
    UP(c_dfdc, t.dfdc)
    UP(c_dfde, t.dfde)
    UP(c_d2fdc2, t.d2fdc2)
    UP(c_d2fde2, t.d2fde2)
    UP(c_d2fdce, t.d2fdce)
    UP(c_ew, t.ew)
    UP(c_ebfn, t.ebfn)
    UP(c_edfdc, t.edfdc)
    UP(c_edfde, t.edfde)
    UP(c_ed2c, t.ed2c)
    UP(c_ed2e, t.ed2e)
    UP(c_ed2ce, t.ed2ce)
#undef UP
    return e;
}

// ---------------------------------------------------------------------------
// FD kernel

__device__ __forceinline__ double wi_of(const ElemArgs &a, const KParams &prm)
{
    return prm.nex > 0 ? prm.Wi0 * a.EU[prm.nex - 1] : prm.WiN;
}

struct SmemView {
    const double *p;
    __device__ __forceinline__ double operator()(int pos) const { return p[pos]; }
};

// the state evaluation k sees: positions before kk are restored, kk is perturbed
struct FdView {
    const double *orig, *rest, *pert;
    int kk;
    __device__ __forceinline__ double operator()(int pos) const
    {
        const double *src = pos < kk ? rest : (pos == kk ? pert : orig);
        return src[pos];
    }
};

// Forward-difference columns by perturbed field.
//
// Column (inod, ieq) of storeBulk perturbs one unknown, and only part of the
// physics sees its field: the velocity columns keep what the stresses alone
// give (StressPart, TestStress: 22% of a test node's operations, 40% of a Gauss
// point's), the pressure columns everything but P and the momentum residual
// (45 of 154 operations at a test node), the stress columns what the velocity
// alone gives.  The kept values are computed once per element, from the same
// expressions in the same order, and every term, product and sum that follows
// is the reference's: the columns' bits are those of 54 full evaluations.  A
// CTA takes one kind of column of a run of elements:
//   27 stress columns and the arclength column x 9 elements  (252 of 256 threads)
//   18 velocity columns                        x 14 elements (252)
//    9 pressure columns                        x 28 elements (252)
// so that every lane of a warp runs the same code; 28 + 18 + 9 CTAs cover the
// same 252 elements, next to each other in the grid, so their parts of an
// element's rows meet in L2.  Meshes of up to four elements per SM take
// k_fd64_element.
// The base residual is k_res64's (launched before).
// An element with a restore residue ((x + eps) - eps differs from x, so later
// columns see a changed state) is left to the last kind of CTA, which
// evaluates it in full.
//
// Bound: the FP64 pipe.  Eight full warps per SM at 255 registers instead of
// seven; the columns' operations are 78% of full evaluations'.  Residual and
// Jacobian, SQRT form: 81.3 -> 63.6 ms on 40,000 quads, 4.95 -> 3.72 on 2,000;
// T form 50.9 -> 40.8 on 40,000.
constexpr int FS_COLS = 28, FU_COLS = 18, FP_COLS = 9;

constexpr int FD_THREADS = 256;
// elements per CTA by kind (stress, velocity, pressure, residue check)
constexpr int FD_S = 9, FD_U = 14, FD_P = 28, FD_R = 4;
constexpr int FD_RUN = 252;       // elements of a group of CTAs

struct FdStressSmem {
    double tl[FD_S][2][54];        // 0: original, 1: perturbed x + eps
    Interp<double> base[FD_S][9];
    FlowPart<double> flow[FD_S][9];
    double dotU[FD_S][9][9];
    int residue[FD_S];
};

template <int FORM>
struct FdFlowSmem {
    double tl[FD_U][2][54];
    Interp<double> base[FD_U][9];
    StressPart<double> stress[FD_U][9];
    double test[FD_U][9][9][FORM == FORM_SQRT ? 11 : 3];       // TestStress (T form: grad S . grad phi only)
    int residue[FD_U];
};

struct FdPressureSmem {
    double tl[FD_P][54];
    double pert[FD_P][9];
    GpCoef<double> g[FD_P][9];
    double keep[FD_P][9][6];       // stress + BvN G without p, div T, BvN Laplacian
    TestPressure<double> test[FD_P][9];                         // of the current Gauss point
    int residue[FD_P];
};

struct FdResidueSmem {
    double tl[FD_R][3][54];      // 0: original, 1: restored (x+eps)-eps, 2: perturbed x+eps
    int any[FD_R];
};

template <int FORM>
union FdSmem {
    FdStressSmem s;
    FdFlowSmem<FORM> u;
    FdPressureSmem p;
    FdResidueSmem r;
};

// x / y with r the rounded reciprocal of y: div_r's steps, infinities and NaN
// passed through (the quotient is the difference of two residuals over eps)
__device__ __forceinline__ double div_by(double x, double y, double r)
{
    const double q0 = x * r;
    const unsigned hi = (unsigned)__double2hiint(q0) & 0x7fffffffu;
    if (hi >= 0x7ff00000u || (hi | (unsigned)__double2loint(q0)) == 0u) return q0;
    const double e = __fma_rn(-q0, y, x);
    return __fma_rn(e, r, q0);
}

// Programmatic dependent launch: the residual kernels let the FD kernel start
// beside them, which waits for the residual only where it takes differences.
// The state, which operations before the residual kernel wrote, it reads with
// load_early (vefem_early.cuh): the same times as plain loads.  In order after
// the residual a call takes 1.2% longer on 640 and 2,000 quads in the T form.
__device__ __forceinline__ void pdl_launch_dependents()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ double early_state(const ElemArgs &a, int f, int inod, int e)
{
    return load_early(a.TL + (size_t)f * a.nnodes + a.conn[inod * a.nel + e]);
}

// Wi of the state, and of the arclength column's
__device__ __forceinline__ double early_wi(const ElemArgs &a, const KParams &prm, bool column = false)
{
    if (prm.nex == 0) return prm.WiN;
    const double eu = load_early(a.EU + prm.nex - 1);
    return prm.Wi0 * (column ? eu + prm.eps : eu);
}

// column `inod, ieq` of the element (ieq 6: the arclength column)
__device__ __forceinline__ void store_column(const ElemArgs &a, const KParams &prm, int e, int inod, int ieq,
                                             const double (&res)[54])
{
    pdl_wait();
    const double *res0 = a.rs + (size_t)e * 54;
    const double eps = prm.eps;
    const bool plain = !(eps > 1.0e-300 && eps < 1.0e300);
    const double r = plain ? 0.0 : recip_for_div(eps);
    double *dst = ieq == 6 ? a.as + (size_t)e * 54 : a.es + (size_t)e * 2916 + inod * 36 + ieq;
    const int sn = ieq == 6 ? 6 : 324, se = ieq == 6 ? 1 : 6;
#pragma unroll
    for (int jnod = 0; jnod < 9; jnod++)
#pragma unroll
        for (int jeq = 0; jeq < 6; jeq++) {
            const double d = res[jnod * 6 + jeq] - res0[jnod * 6 + jeq];
            dst[jnod * sn + jeq * se] = plain ? d / eps : div_by(d, eps, r);
        }
}

// stage the states of elements e0 .. e0 + ne, and mark those with a restore residue
template <int EL>
__device__ __forceinline__ void stage_states(const ElemArgs &a, const KParams &prm, int e0, int ne,
                                             double (*tl)[2][54], int *residue)
{
    for (int i = threadIdx.x; i < EL; i += FD_THREADS) residue[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < ne * 54; i += FD_THREADS) {
        const int el = i / 54, pos = i - 54 * el, inod = pos / 6, f = pos - 6 * inod;
        const double v = early_state(a, f, inod, e0 + el);
        const double vp = v + prm.eps, back = vp - prm.eps;
        tl[el][0][pos] = v;
        tl[el][1][pos] = vp;
        if (__double_as_longlong(back) != __double_as_longlong(v)) residue[el] = 1;
    }
    __syncthreads();
}

// the state of a column: original except position kk
struct FdCleanView {
    const double *orig, *pert;
    int kk;
    __device__ __forceinline__ double operator()(int pos) const
    {
        return pos == kk ? pert[pos] : orig[pos];
    }
};

// value and gradient of field f of the perturbed state (interpolate's sums)
__device__ __forceinline__ void perturbed(const FdCleanView &V, int f, const double *bfn, const double *dFx,
                                          const double *dFy, double &val, double &gx, double &gy)
{
    val = 0.0;
    gx = 0.0;
    gy = 0.0;
#pragma unroll
    for (int n = 0; n < 9; n++) {
        const double t = V(n * 6 + f);
        val = val + t * bfn[n];
        gx = gx + t * dFx[n];
        gy = gy + t * dFy[n];
    }
}

template <int FORM, int SPEC>
__device__ __forceinline__ void fd_stress(const ElemArgs &a, const KParams &prm, int e0, FdStressSmem &sm)
{
    static_assert(FD_S * FS_COLS <= FD_THREADS, "a thread per column");
    const int t = threadIdx.x, ne = min(FD_S, a.nel - e0);
    if (ne <= 0) return;
    stage_states<FD_S>(a, prm, e0, ne, sm.tl, sm.residue);
    for (int i = t; i < ne * 9; i += FD_THREADS) {
        const int el = i / 9, ig = i - 9 * el;
        const double *geo = a.geo + ((size_t)(e0 + el) * 9 + ig) * GEO_REC;
        SmemView V{sm.tl[el][0]};
        const Interp<double> I = interpolate(V, c_bfn[ig], geo, geo + 9, geo + 18, geo + 27);
        sm.base[el][ig] = I;
        sm.flow[el][ig] = flow_part(I, kinematics(I), geo, geo + 9, sm.dotU[el][ig]);
    }
    __syncthreads();
    const int el = t / FS_COLS, c = t - FS_COLS * el;
    const bool ac = c == 27;
    if (el >= ne || sm.residue[el] || (ac && prm.nex == 0)) return;
    const int inod = c / 3, f = 3 + c - 3 * inod, kk = ac ? -1 : inod * 6 + f, e = e0 + el;
    const double WiN = early_wi(a, prm, ac);
    double res[54];
#pragma unroll
    for (int i = 0; i < 54; i++) res[i] = 0.0;
#pragma unroll 1
    for (int ig = 0; ig < 9; ig++) {
        const double *geo = a.geo + ((size_t)e * 9 + ig) * GEO_REC, *dFx = geo, *dFy = geo + 9;
        const double H2 = geo[36], WET = geo[37];
        Interp<double> I = sm.base[el][ig];
        if (!ac) {
            FdCleanView V{sm.tl[el][0], sm.tl[el][1], kk};
            double v, gx, gy;
            perturbed(V, f, c_bfn[ig], dFx, dFy, v, gx, gy);
            I.S11 = f == 3 ? v : I.S11;
            I.dS11x = f == 3 ? gx : I.dS11x;
            I.dS11y = f == 3 ? gy : I.dS11y;
            I.S12 = f == 4 ? v : I.S12;
            I.dS12x = f == 4 ? gx : I.dS12x;
            I.dS12y = f == 4 ? gy : I.dS12y;
            I.S22 = f == 5 ? v : I.S22;
            I.dS22x = f == 5 ? gx : I.dS22x;
            I.dS22y = f == 5 ? gy : I.dS22y;
        }
        const StressPart<double> p = stress_part<FORM>(I, prm, WiN, H2);
        const GpCoef<double> g =
            combine_parts<FORM, SPEC>(I, prm, WiN, H2, p, kinematics(I), sm.flow[el][ig]);
#pragma unroll
        for (int n = 0; n < 9; n++) {
            double o[6];
            const TestStress<double> ts = test_stress<FORM>(I, p.den, p.rden, dFx[n], dFy[n]);
            test_terms<FORM, SPEC>(g, prm, ts, c_bfn[ig][n], dFx[n], dFy[n], sm.dotU[el][ig][n], WET, o);
#pragma unroll
            for (int q = 0; q < 6; q++) res[n * 6 + q] = res[n * 6 + q] + o[q];
        }
    }
    store_column(a, prm, e, inod, ac ? 6 : f, res);
}

template <int FORM, int SPEC>
__device__ __forceinline__ void fd_flow(const ElemArgs &a, const KParams &prm, int e0, FdFlowSmem<FORM> &sm)
{
    static_assert(FD_U * FU_COLS <= FD_THREADS, "a thread per column");
    const int t = threadIdx.x, ne = min(FD_U, a.nel - e0);
    if (ne <= 0) return;
    const double WiN = early_wi(a, prm);
    stage_states<FD_U>(a, prm, e0, ne, sm.tl, sm.residue);
    for (int i = t; i < ne * 9; i += FD_THREADS) {
        const int el = i / 9, ig = i - 9 * el;
        const double *geo = a.geo + ((size_t)(e0 + el) * 9 + ig) * GEO_REC;
        SmemView V{sm.tl[el][0]};
        const Interp<double> I = interpolate(V, c_bfn[ig], geo, geo + 9, geo + 18, geo + 27);
        sm.base[el][ig] = I;
        sm.stress[el][ig] = stress_part<FORM>(I, prm, WiN, geo[36]);
    }
    __syncthreads();
    for (int i = t; i < ne * 81; i += FD_THREADS) {
        const int el = i / 81, ig = (i / 9) % 9, n = i % 9;
        const double *geo = a.geo + ((size_t)(e0 + el) * 9 + ig) * GEO_REC;
        const StressPart<double> &p = sm.stress[el][ig];
        const TestStress<double> ts = test_stress<FORM>(sm.base[el][ig], p.den, p.rden, geo[n], geo[9 + n]);
        double *d = sm.test[el][ig][n];
        d[0] = ts.gd11;
        d[1] = ts.gd12;
        d[2] = ts.gd22;
        if (FORM == FORM_SQRT) {
            d[3] = ts.u11; d[4] = ts.u12; d[5] = ts.u21; d[6] = ts.u22;
            d[7] = ts.v11; d[8] = ts.v12; d[9] = ts.v21; d[10] = ts.v22;
        }
    }
    __syncthreads();
    const int el = t / FU_COLS, c = t - FU_COLS * el;
    if (el >= ne || sm.residue[el]) return;
    const int inod = c >> 1, f = c & 1, kk = inod * 6 + f, e = e0 + el;
    double res[54];
#pragma unroll
    for (int i = 0; i < 54; i++) res[i] = 0.0;
#pragma unroll 1
    for (int ig = 0; ig < 9; ig++) {
        const double *geo = a.geo + ((size_t)e * 9 + ig) * GEO_REC, *dFx = geo, *dFy = geo + 9;
        const double H2 = geo[36], WET = geo[37];
        Interp<double> I = sm.base[el][ig];
        {
            FdCleanView V{sm.tl[el][0], sm.tl[el][1], kk};
            interpolate_field(V, f, c_bfn[ig], dFx, dFy, geo + 18, geo + 27, I);
        }
        double dotU[9];
        const Kinematics<double> k = kinematics(I);
        const FlowPart<double> q = flow_part(I, k, dFx, dFy, dotU);
        const GpCoef<double> g = combine_parts<FORM, SPEC>(I, prm, WiN, H2, sm.stress[el][ig], k, q);
#pragma unroll
        for (int n = 0; n < 9; n++) {
            double o[6];
            const double *d = sm.test[el][ig][n];
            TestStress<double> ts;
            ts.gd11 = d[0];
            ts.gd12 = d[1];
            ts.gd22 = d[2];
            if (FORM == FORM_SQRT) {
                ts.u11 = d[3]; ts.u12 = d[4]; ts.u21 = d[5]; ts.u22 = d[6];
                ts.v11 = d[7]; ts.v12 = d[8]; ts.v21 = d[9]; ts.v22 = d[10];
            }
            test_terms<FORM, SPEC>(g, prm, ts, c_bfn[ig][n], dFx[n], dFy[n], dotU[n], WET, o);
#pragma unroll
            for (int w = 0; w < 6; w++) res[n * 6 + w] = res[n * 6 + w] + o[w];
        }
    }
    store_column(a, prm, e, inod, f, res);
}

template <int FORM, int SPEC>
__device__ __forceinline__ void fd_pressure(const ElemArgs &a, const KParams &prm, int e0, FdPressureSmem &sm)
{
    static_assert(FD_P * FP_COLS <= FD_THREADS, "a thread per column");
    const int t = threadIdx.x, ne = min(FD_P, a.nel - e0);
    if (ne <= 0) return;
    const double WiN = early_wi(a, prm);
    for (int i = t; i < FD_P; i += FD_THREADS) sm.residue[i] = 0;
    __syncthreads();
    for (int i = t; i < ne * 54; i += FD_THREADS) {
        const int el = i / 54, pos = i - 54 * el, inod = pos / 6, f = pos - 6 * inod;
        const double v = early_state(a, f, inod, e0 + el);
        const double vp = v + prm.eps, back = vp - prm.eps;
        sm.tl[el][pos] = v;
        if (f == 2) sm.pert[el][inod] = vp;
        if (__double_as_longlong(back) != __double_as_longlong(v)) sm.residue[el] = 1;
    }
    __syncthreads();
    for (int i = t; i < ne * 9; i += FD_THREADS) {
        const int el = i / 9, ig = i - 9 * el;
        const double *geo = a.geo + ((size_t)(e0 + el) * 9 + ig) * GEO_REC;
        SmemView V{sm.tl[el]};
        const Interp<double> I = interpolate(V, c_bfn[ig], geo, geo + 9, geo + 18, geo + 27);
        const Kinematics<double> k = kinematics(I);
        const StressPart<double> p = stress_part<FORM>(I, prm, WiN, geo[36]);
        double dotU[9];
        const FlowPart<double> q = flow_part(I, k, geo, geo + 9, dotU);
        sm.g[el][ig] = combine_parts<FORM, SPEC>(I, prm, WiN, geo[36], p, k, q);
        double *c = sm.keep[el][ig];
        c[0] = p.T11 + prm.BvN * k.Gd11;
        c[1] = p.T22 + prm.BvN * k.Gd22;
        c[2] = p.divT1;
        c[3] = p.divT2;
        c[4] = prm.BvN * I.lap1;
        c[5] = prm.BvN * I.lap2;
    }
    __syncthreads();
    const int el = t / FP_COLS, inod = t - FP_COLS * el;    // also the test node in the kept terms
    const bool staged = el < ne, live = staged && !sm.residue[el];
    const int e = e0 + el;
    double res[54];
#pragma unroll
    for (int i = 0; i < 54; i++) res[i] = 0.0;
#pragma unroll 1
    for (int ig = 0; ig < 9; ig++) {
        const double *geo = a.geo + ((size_t)(staged ? e : e0) * 9 + ig) * GEO_REC, *dFx = geo, *dFy = geo + 9;
        if (staged) {
            const GpCoef<double> &g = sm.g[el][ig];
            Interp<double> I;
            I.S11 = g.S11; I.S12 = g.S12; I.S22 = g.S22;
            I.dS11x = g.dS11x; I.dS11y = g.dS11y; I.dS12x = g.dS12x; I.dS12y = g.dS12y;
            I.dS22x = g.dS22x; I.dS22y = g.dS22y;
            const double fx = dFx[inod], fy = dFy[inod];
            const TestStress<double> ts = test_stress<FORM>(I, g.den, g.rden, fx, fy);
            sm.test[el][inod] =
                test_pressure<FORM, SPEC>(g, prm, ts, c_bfn[ig][inod], fx, fy, g.U1 * fx + g.U2 * fy);
        }
        __syncthreads();
        if (live) {
            const GpCoef<double> &g = sm.g[el][ig];
            const double *c = sm.keep[el][ig];
            double P = 0.0, dPx = 0.0, dPy = 0.0;
#pragma unroll
            for (int n = 0; n < 9; n++) {
                const double v = n == inod ? sm.pert[el][n] : sm.tl[el][n * 6 + 2];
                P = P + v * c_bfn[ig][n];
                dPx = dPx + v * dFx[n];
                dPy = dPy + v * dFy[n];
            }
            const double P11 = c[0] - P, P22 = c[1] - P;
            const double divP1 = (-dPx + c[2]) + c[4], divP2 = (-dPy + c[3]) + c[5];
            const double M1 = (SPEC & SPEC_RE0) ? -divP1 : g.rc1 - divP1;
            const double M2 = (SPEC & SPEC_RE0) ? -divP2 : g.rc2 - divP2;
            const double WET = geo[37], scale = FORM == FORM_T ? g.omb : g.WiN;
#pragma unroll
            for (int n = 0; n < 9; n++) {
                double o[6];
                const double fx = dFx[n], fy = dFy[n];
                pressure_terms<FORM, SPEC>(sm.test[el][n], P11, P22, M1, M2, g.rc1, g.rc2, g.tR, g.tlsme, scale,
                                           c_bfn[ig][n], fx, fy, (SPEC & SPEC_RE0) ? 0.0 : g.U1 * fx + g.U2 * fy, WET,
                                           o);
#pragma unroll
                for (int w = 0; w < 6; w++) res[n * 6 + w] = res[n * 6 + w] + o[w];
            }
        }
        __syncthreads();
    }
    if (live) store_column(a, prm, e, inod, 2, res);
}

// Elements with a restore residue: all 55 columns, each a full evaluation of the
// state the sequential loop would have, 4 elements on 220 lanes.  Values below
// eps that are not zero leave one, so a converged flow has them wherever a
// component vanishes: 4 elements to a CTA and not 64 in turn, SQRT form, 20,000
// quads with residues in all of them 75 -> 46.6 ms, in half 65 -> 39.8.  A CTA
// without any costs its look at the state, 2 us.
template <int FORM, int SPEC>
__device__ __forceinline__ void fd_residue(const ElemArgs &a, const KParams &prm, int e0, FdResidueSmem &sm)
{
    static_assert(FD_R * 55 <= FD_THREADS, "a thread per column");
    const int t = threadIdx.x, ne = min(FD_R, a.nel - e0);
    if (t < FD_R) sm.any[t] = 0;
    __syncthreads();
    if (t < ne * 54) {
        const int el = t / 54, k = t - 54 * el, inod = k / 6, f = k - 6 * inod;
        const double v = early_state(a, f, inod, e0 + el);
        const double vp = v + prm.eps, back = vp - prm.eps;
        sm.tl[el][0][k] = v;
        sm.tl[el][2][k] = vp;
        sm.tl[el][1][k] = back;
        if (__double_as_longlong(back) != __double_as_longlong(v)) sm.any[el] = 1;
    }
    __syncthreads();
    const int el = t / 55, k = t - 55 * el, e = e0 + el;
    const bool ac = k == 54;
    if (el >= ne || !sm.any[el] || (ac && prm.nex == 0)) return;
    FdView V;
    V.orig = sm.tl[el][0];
    V.rest = sm.tl[el][1];
    V.pert = sm.tl[el][2];
    V.kk = k;
    const double WiN = early_wi(a, prm, ac);
    double res[54];
#pragma unroll
    for (int q = 0; q < 54; q++) res[q] = 0.0;
#pragma unroll 1
    for (int ig = 0; ig < 9; ig++) {
        const double *geo = a.geo + ((size_t)e * 9 + ig) * GEO_REC, *dFx = geo, *dFy = geo + 9;
        const Interp<double> I = interpolate(V, c_bfn[ig], dFx, dFy, geo + 18, geo + 27);
        double dotU[9];
        const GpCoef<double> g = gauss_point<FORM, SPEC>(I, prm, WiN, geo[36], dFx, dFy, dotU);
#pragma unroll
        for (int n = 0; n < 9; n++) {
            double o[6];
            test_node<FORM, SPEC>(g, prm, c_bfn[ig][n], dFx[n], dFy[n], dotU[n], geo[37], o);
#pragma unroll
            for (int w = 0; w < 6; w++) res[n * 6 + w] = res[n * 6 + w] + o[w];
        }
    }
    store_column(a, prm, e, ac ? 0 : k / 6, ac ? 6 : k - 6 * (k / 6), res);
}

// All columns of an element in one CTA, for a mesh whose CTAs fit the GPU at once:
// its time is one column's chain of FP64 instructions, which keeping the other
// fields' part does not shorten (a thread first waits for it).  One element, 55
// of 64 lanes, where there are up to three to an SM: SQRT form, 300 quads, 765
// us, 850 with residues (four elements 1,255 and 1,440).  Four, 220 of 224 lanes,
// up to four to an SM, where a CTA of one would be the fourth on some of them:
// SQRT form, 460 / 500 / 606 quads, 1,240 / 1,241 / 1,244 us, with residues in half
// of the elements 1,413 / 1,415 / 1,425; T form 757 to 759 and 932 to 943.  Columns
// by field in CTAs of 64 threads took 1,220 / 1,288 / 1,289 and 1,443 / 1,626 /
// 1,819 there, in the T form 775 to 786 and 995 to 1,283.
template <int EL>
struct FdElementSmem {
    double tl[EL][3][54];        // 0: original, 1: restored (x+eps)-eps, 2: perturbed x+eps
    Interp<double> base[EL][9];
    int any[EL];
};

constexpr int FE_COLS = 55;
template <int EL> constexpr int FE_THREADS = (EL * FE_COLS + 31) / 32 * 32;

template <int FORM, int SPEC, int EL>
__global__ void __launch_bounds__(FE_THREADS<EL>, EL == 1 ? 4 : 1) k_fd64_element(const ElemArgs a, const KParams prm)
{
    __shared__ __align__(16) unsigned char raw[sizeof(FdElementSmem<EL>)];
    FdElementSmem<EL> &sm = *reinterpret_cast<FdElementSmem<EL> *>(raw);
    const int el = threadIdx.x / FE_COLS, t = threadIdx.x - FE_COLS * el, e = blockIdx.x * EL + el;
    const bool in = el < EL && e < a.nel;
    const int inod = t / 6, f = t - 6 * inod;
    if (threadIdx.x < EL) sm.any[threadIdx.x] = 0;
    __syncthreads();
    if (in && t < 54) {
        const double v = a.TL[(size_t)f * a.nnodes + a.conn[inod * a.nel + e]];
        const double vp = v + prm.eps, back = vp - prm.eps;
        sm.tl[el][0][t] = v;
        sm.tl[el][2][t] = vp;
        sm.tl[el][1][t] = back;
        if (__double_as_longlong(back) != __double_as_longlong(v)) sm.any[el] = 1;
    }
    __syncthreads();
    const bool clean = in && !sm.any[el];
    if (clean && t < 9) {
        const double *geo = a.geo + ((size_t)e * 9 + t) * GEO_REC;
        SmemView V{sm.tl[el][0]};
        sm.base[el][t] = interpolate(V, c_bfn[t], geo, geo + 9, geo + 18, geo + 27);
    }
    __syncthreads();
    const bool ac = t == 54;
    if (!in || (ac && prm.nex == 0)) return;
    double WiN = prm.WiN;
    if (prm.nex > 0) {
        const double eu = a.EU[prm.nex - 1];
        WiN = prm.Wi0 * (ac ? eu + prm.eps : eu);
    }
    double res[54];
#pragma unroll
    for (int q = 0; q < 54; q++) res[q] = 0.0;
#pragma unroll 1
    for (int ig = 0; ig < 9; ig++) {
        const double *geo = a.geo + ((size_t)e * 9 + ig) * GEO_REC, *dFx = geo, *dFy = geo + 9;
        Interp<double> I;
        if (clean) {
            I = sm.base[el][ig];
            FdCleanView V{sm.tl[el][0], sm.tl[el][2], t};
            if (!ac) interpolate_field(V, f, c_bfn[ig], dFx, dFy, geo + 18, geo + 27, I);
        } else {
            FdView V;
            V.orig = sm.tl[el][0];
            V.rest = sm.tl[el][1];
            V.pert = sm.tl[el][2];
            V.kk = t;
            I = interpolate(V, c_bfn[ig], dFx, dFy, geo + 18, geo + 27);
        }
        double dotU[9];
        const GpCoef<double> g = gauss_point<FORM, SPEC>(I, prm, WiN, geo[36], dFx, dFy, dotU);
#pragma unroll
        for (int n = 0; n < 9; n++) {
            double o[6];
            test_node<FORM, SPEC>(g, prm, c_bfn[ig][n], dFx[n], dFy[n], dotU[n], geo[37], o);
#pragma unroll
            for (int w = 0; w < 6; w++) res[n * 6 + w] = res[n * 6 + w] + o[w];
        }
    }
    store_column(a, prm, e, ac ? 0 : inod, ac ? 6 : f, res);
}

template <int FORM, int SPEC>
__global__ void __launch_bounds__(FD_THREADS, 1) k_fd64(const ElemArgs a, const KParams prm, int groups)
{
    extern __shared__ __align__(16) unsigned char fd_raw[];
    FdSmem<FORM> &sm = *reinterpret_cast<FdSmem<FORM> *>(fd_raw);
    // CTAs of each kind in a group, in this order
    constexpr int S = FD_RUN / FD_S, U = FD_RUN / FD_U, P = FD_RUN / FD_P;
    static_assert(S * FD_S == FD_RUN && U * FD_U == FD_RUN && P * FD_P == FD_RUN, "whole CTAs in a group");
    const int grp = blockIdx.x / (S + U + P);
    if (grp >= groups) {
        fd_residue<FORM, SPEC>(a, prm, (blockIdx.x - groups * (S + U + P)) * FD_R, sm.r);
        return;
    }
    const int b = blockIdx.x - grp * (S + U + P), e0 = grp * FD_RUN;
    if (b < S)
        fd_stress<FORM, SPEC>(a, prm, e0 + b * FD_S, sm.s);
    else if (b < S + U)
        fd_flow<FORM, SPEC>(a, prm, e0 + (b - S) * FD_U, sm.u);
    else
        fd_pressure<FORM, SPEC>(a, prm, e0 + (b - S - U) * FD_P, sm.p);
}

// ---------------------------------------------------------------------------
// Residual-only kernel: thread = (element, Gauss point)
//
// A CTA of RES_EPB = 7 elements is 63 of 64 lanes; 8 elements (72 threads) left
// 24 of 96 lanes idle, and an FP64 instruction holds the pipe for a whole warp
// whatever its lanes do.  The geometry of the Gauss points comes from the
// mesh's table (11% of the instructions, once per mesh instead of per call).
// The 54 terms of a Gauss point go through shared memory three test nodes at a
// time, which keeps a CTA at 31 KB, 6 or 7 of them per SM.  40,000 elements:
// 2.43 -> 1.63 ms.
constexpr int RS_EPB = RES_EPB;
constexpr int RS_THREADS = 64;
constexpr int RS_MIN_CTAS = 6;
constexpr int RS_CHUNK = 3;                 // test nodes per pass through shared memory
static_assert(RS_EPB * 9 <= RS_THREADS, "a thread per element and Gauss point");

// elements [e0, e0 + count) of one mesh, count <= RS_EPB; SPEC leaves out the
// exact-zero terms of ReN = 0 / DfN = 0 as the FD kernel does (same values)
template <int FORM, int SPEC>
__device__ __forceinline__ void res64_block(const ElemArgs &a, const KParams &prm, int e0,
                                            int count)
{
    __shared__ double s_tl[RS_EPB][54];
    __shared__ __align__(16) double s_geo[RS_EPB * 9 * GEO_REC];
    __shared__ double s_bfn[9][9];
    __shared__ double s_part[RS_EPB][9][RS_CHUNK * 6];
    const int t = threadIdx.x;
    const int el = t / 9;
    const int ig = t - el * 9;
    const int e_end = min(e0 + count, a.nel);
    const bool live = t < RS_EPB * 9 && e0 + el < e_end;
    // stage element states (54 values each, spread over the CTA) and geometry records
    for (int i = t; i < RS_EPB * 54; i += RS_THREADS) {
        const int ee = e0 + i / 54;
        const int pos = i - (i / 54) * 54;
        if (ee < e_end) {
            const int inod = pos / 6, f = pos - 6 * (pos / 6);
            s_tl[i / 54][pos] = a.TL[(size_t)f * a.nnodes + a.conn[inod * a.nel + ee]];
        }
    }
    const double2 *gsrc = reinterpret_cast<const double2 *>(a.geo + (size_t)e0 * 9 * GEO_REC);
    const int ng = (e_end - e0) * 9 * GEO_REC / 2;
    for (int i = t; i < ng; i += RS_THREADS) reinterpret_cast<double2 *>(s_geo)[i] = gsrc[i];
    for (int i = t; i < 81; i += RS_THREADS) s_bfn[i / 9][i % 9] = c_bfn[i / 9][i % 9];
    __syncthreads();
    const double *geo = s_geo + (live ? t : 0) * GEO_REC;
    const double *dFx = geo, *dFy = geo + 9, *bfn = s_bfn[ig];
    const double WET = geo[37];
    double dotU[9];
    GpCoef<double> g;
    if (live) {
        SmemView V{s_tl[el]};
        const auto I = interpolate(V, bfn, dFx, dFy, geo + 18, geo + 27);
        g = gauss_point<FORM, SPEC>(I, prm, wi_of(a, prm), geo[36], dFx, dFy, dotU);
    }
#pragma unroll
    for (int n0 = 0; n0 < 9; n0 += RS_CHUNK) {
        if (live) {
#pragma unroll
            for (int n = n0; n < n0 + RS_CHUNK; n++)
                test_node<FORM, SPEC>(g, prm, bfn[n], dFx[n], dFy[n], dotU[n], WET,
                                      &s_part[el][ig][(n - n0) * 6]);
        }
        __syncthreads();
        // in-order sum over the Gauss points (Res = Res + TERM*WET, ig = 1..9)
        for (int i = t; i < RS_EPB * RS_CHUNK * 6; i += RS_THREADS) {
            const int le = i / (RS_CHUNK * 6), pos = i - le * (RS_CHUNK * 6);
            if (e0 + le >= e_end) continue;
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < 9; q++) s = s + s_part[le][q][pos];
            a.rs[(size_t)(e0 + le) * 54 + n0 * 6 + pos] = s;
        }
        __syncthreads();
    }
}

template <int FORM, int SPEC>
__global__ void __launch_bounds__(RS_THREADS, RS_MIN_CTAS) k_res64(const ElemArgs a, const KParams prm)
{
    pdl_launch_dependents();
    res64_block<FORM, SPEC>(a, prm, blockIdx.x * RS_EPB, RS_EPB);
}

// The same residual for a mesh that leaves the GPU short of warps: the time is
// then one thread's chain of FP64 instructions, so E elements are spread over a
// CTA: a thread per interpolated sum (22 at each Gauss point), per Gauss point,
// and per (Gauss point, test node).  Every sum is the one of k_res64, in its
// order.  The Gauss points' warp differs from CTA to CTA, so that the longest
// phase of the CTAs of an SM spreads over its four FP64 pipes.
template <int FORM, int SPEC, int E, int THREADS>
__global__ void __launch_bounds__(THREADS, E == 1 ? 4 : 2) k_res64_wide(const ElemArgs a, const KParams prm)
{
    pdl_launch_dependents();
    __shared__ double s_tl[E][54];
    __shared__ __align__(16) double s_geo[E * 9 * GEO_REC];
    __shared__ double s_bfn[9][9];
    __shared__ double s_ip[E * 9][22];
    __shared__ GpCoef<double> s_g[E * 9];
    __shared__ double s_du[E * 9][9];
    __shared__ double s_part[E * 9][54];
    const int t = threadIdx.x, e0 = blockIdx.x * E, ne = min(E, a.nel - e0);
    for (int i = t; i < ne * 54; i += THREADS) {
        const int el = i / 54, pos = i - 54 * el, inod = pos / 6, f = pos - 6 * inod;
        s_tl[el][pos] = a.TL[(size_t)f * a.nnodes + a.conn[inod * a.nel + e0 + el]];
    }
    for (int i = t; i < ne * 9 * GEO_REC; i += THREADS) s_geo[i] = a.geo[(size_t)e0 * 9 * GEO_REC + i];
    for (int i = t; i < 81; i += THREADS) s_bfn[i / 9][i % 9] = c_bfn[i / 9][i % 9];
    __syncthreads();
    // sums 0..4 and 5..9: u and v against phi, dphi/dx, dphi/dy, d2x, d2y;
    // 10..21: p and the stresses against phi, dphi/dx, dphi/dy
    for (int i = t; i < ne * 9 * 22; i += THREADS) {
        const int gp = i / 22, q = i - 22 * gp;
        const int f = q < 10 ? q / 5 : 2 + (q - 10) / 3, k = q < 10 ? q % 5 : (q - 10) % 3;
        const double *w = k == 0 ? s_bfn[gp % 9] : s_geo + gp * GEO_REC + 9 * (k - 1);
        double s = 0.0;
#pragma unroll
        for (int n = 0; n < 9; n++) s = s + s_tl[gp / 9][n * 6 + f] * w[n];
        s_ip[gp][q] = s;
    }
    __syncthreads();
    const int gp = t - 32 * (blockIdx.x % (THREADS / 32));
    if (gp >= 0 && gp < ne * 9) {
        const double *q = s_ip[gp], *geo = s_geo + gp * GEO_REC;
        Interp<double> I;
        I.U1 = q[0]; I.GU11 = q[1]; I.GU21 = q[2]; I.lap1 = q[3] + q[4];
        I.U2 = q[5]; I.GU12 = q[6]; I.GU22 = q[7]; I.lap2 = q[8] + q[9];
        I.P = q[10]; I.dPx = q[11]; I.dPy = q[12];
        I.S11 = q[13]; I.dS11x = q[14]; I.dS11y = q[15];
        I.S12 = q[16]; I.dS12x = q[17]; I.dS12y = q[18];
        I.S22 = q[19]; I.dS22x = q[20]; I.dS22y = q[21];
        double dotU[9];
        s_g[gp] = gauss_point<FORM, SPEC>(I, prm, wi_of(a, prm), geo[36], geo, geo + 9, dotU);
#pragma unroll
        for (int n = 0; n < 9; n++) s_du[gp][n] = dotU[n];
    }
    __syncthreads();
    for (int i = t; i < ne * 81; i += THREADS) {
        const int ig = i / 9, n = i - 9 * ig;
        const double *geo = s_geo + ig * GEO_REC;
        test_node<FORM, SPEC>(s_g[ig], prm, s_bfn[ig % 9][n], geo[n], geo[9 + n], s_du[ig][n], geo[37],
                              &s_part[ig][n * 6]);
    }
    __syncthreads();
    for (int i = t; i < ne * 54; i += THREADS) {
        const int el = i / 54, pos = i - 54 * el;
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < 9; q++) s = s + s_part[el * 9 + q][pos];
        a.rs[(size_t)(e0 + el) * 54 + pos] = s;
    }
}

// persistent form over the work items of many meshes
template <int FORM, int SPEC>
__global__ void __launch_bounds__(RS_THREADS, RS_MIN_CTAS)
k_res64_batched(const BatchInst *__restrict__ insts, const WorkItem *__restrict__ work, int nwork)
{
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = work[w];
        const ElemArgs a = insts[it.inst].ea;
        const KParams prm = insts[it.inst].prm;
        res64_block<FORM, SPEC>(a, prm, it.e0, it.count);
        __syncthreads();
    }
}

// the kernel's specialisation for the parameters: (form, which of ReN, DfN are zero)
#define RES_DISPATCH(form, spec, LAUNCH)                                                        \
    do {                                                                                        \
        if ((form) == FORM_SQRT) {                                                              \
            switch (spec) {                                                                     \
            case 0: LAUNCH(FORM_SQRT, 0); break;                                                \
            case SPEC_RE0: LAUNCH(FORM_SQRT, SPEC_RE0); break;                                  \
            case SPEC_DF0: LAUNCH(FORM_SQRT, SPEC_DF0); break;                                  \
            default: LAUNCH(FORM_SQRT, SPEC_RE0 | SPEC_DF0); break;                             \
            }                                                                                   \
        } else {                                                                                \
            switch (spec) {                                                                     \
            case 0: LAUNCH(FORM_T, 0); break;                                                   \
            case SPEC_RE0: LAUNCH(FORM_T, SPEC_RE0); break;                                     \
            case SPEC_DF0: LAUNCH(FORM_T, SPEC_DF0); break;                                     \
            default: LAUNCH(FORM_T, SPEC_RE0 | SPEC_DF0); break;                                \
            }                                                                                   \
        }                                                                                       \
    } while (0)

static int spec_of(const KParams &p)
{
    return (p.ReN == 0.0 ? SPEC_RE0 : 0) | (p.DfN == 0.0 ? SPEC_DF0 : 0);
}

cudaError_t launch_residual64(const ElemArgs &a, const KParams &p, cudaStream_t s)
{
    if (a.nel <= 0) return cudaSuccess;
    if (a.nel <= RES_WIDE1_MAX) {
#define GO(F, SP) k_res64_wide<F, SP, 1, 96><<<a.nel, 96, 0, s>>>(a, p)
        RES_DISPATCH(p.form, spec_of(p), GO);
#undef GO
        return cudaGetLastError();
    }
    if (a.nel <= RES_WIDE3_MAX) {
#define GO(F, SP) k_res64_wide<F, SP, 3, 256><<<(a.nel + 2) / 3, 256, 0, s>>>(a, p)
        RES_DISPATCH(p.form, spec_of(p), GO);
#undef GO
        return cudaGetLastError();
    }
    const int grid = (a.nel + RS_EPB - 1) / RS_EPB;
#define GO(F, SP) k_res64<F, SP><<<grid, RS_THREADS, 0, s>>>(a, p)
    RES_DISPATCH(p.form, spec_of(p), GO);
#undef GO
    return cudaGetLastError();
}

// Geometry table of a mesh: per element and Gauss point dphi/dx, dphi/dy,
// d2phi/dx2, d2phi/dy2 of the 9 nodes, H^2 and the weight
__global__ void __launch_bounds__(128) k_geometry(int nel, int nnodes, const int32_t *__restrict__ conn,
                                                  const double *__restrict__ xy, double *__restrict__ geo)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)nel * 9) return;
    const int e = (int)(t / 9), ig = (int)(t - (int64_t)e * 9);
    double x[9], y[9], dFx[9], dFy[9], d2x[9], d2y[9];
#pragma unroll
    for (int n = 0; n < 9; n++) {
        const int gn = conn[n * nel + e];
        x[n] = xy[gn];
        y[n] = xy[nnodes + gn];
    }
    const auto go = geometry(c_bfn[ig], c_dfdc[ig], c_dfde[ig], c_d2fdc2[ig], c_d2fde2[ig], c_d2fdce[ig], c_w[ig],
                             x, y, dFx, dFy, d2x, d2y);
    double *r = geo + t * GEO_REC;
#pragma unroll
    for (int n = 0; n < 9; n++) {
        r[n] = dFx[n];
        r[9 + n] = dFy[n];
        r[18 + n] = d2x[n];
        r[27 + n] = d2y[n];
    }
    r[36] = go.H2;
    r[37] = go.WET;
}

cudaError_t launch_geometry(int nel, int nnodes, const int32_t *conn, const double *xy, double *geo, cudaStream_t s)
{
    if (nel <= 0) return cudaSuccess;
    k_geometry<<<(unsigned)(((int64_t)nel * 9 + 127) / 128), 128, 0, s>>>(nel, nnodes, conn, xy, geo);
    return cudaGetLastError();
}

cudaError_t launch_residual64_batched(const BatchInst *insts, const WorkItem *work, int nwork,
                                      int form, int spec, int grid, cudaStream_t s)
{
    if (nwork <= 0) return cudaSuccess;
#define GO(F, SP) k_res64_batched<F, SP><<<grid, RS_THREADS, 0, s>>>(insts, work, nwork)
    RES_DISPATCH(form, spec, GO);
#undef GO
    return cudaGetLastError();
}

int residual_batched_ctas_per_sm(int form, int spec)
{
    int n = 0;
#define GO(F, SP) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_res64_batched<F, SP>, RS_THREADS, 0)
    RES_DISPATCH(form, spec, GO);
#undef GO
    return n;
}

// The columns by field start beside the residual kernel; one wave of blocks does
// not: its blocks would go where the residual's leave first, four to an SM on
// some (300 quads, SQRT form, 765 us in order and 1,368 early).
template <int FORM, int SPEC>
static cudaError_t go_fd64(const ElemArgs &a, const KParams &p, cudaStream_t s)
{
    if (a.nel <= FD_ELEMENT_MAX) {
        k_fd64_element<FORM, SPEC, 1><<<a.nel, FE_THREADS<1>, 0, s>>>(a, p);
        return cudaGetLastError();
    }
    if (a.nel <= FD_FOUR_MAX) {
        k_fd64_element<FORM, SPEC, 4><<<(a.nel + 3) / 4, FE_THREADS<4>, 0, s>>>(a, p);
        return cudaGetLastError();
    }
    const int groups = (a.nel + FD_RUN - 1) / FD_RUN, residue = (a.nel + FD_R - 1) / FD_R;
    const int per = FD_RUN / FD_S + FD_RUN / FD_U + FD_RUN / FD_P, smem = (int)sizeof(FdSmem<FORM>);
    const cudaError_t e = cudaFuncSetAttribute(k_fd64<FORM, SPEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute early[1];
    early[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(groups * per + residue));
    cfg.blockDim = dim3(FD_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_fd64<FORM, SPEC>, a, p, groups);
}

bool fd64_one_wave(int nel) { return nel <= FD_FOUR_MAX; }

cudaError_t launch_fd64(const ElemArgs &a, const KParams &p, cudaStream_t s)
{
    if (a.nel <= 0) return cudaSuccess;
#define GO(F, SP) return go_fd64<F, SP>(a, p, s)
    RES_DISPATCH(p.form, spec_of(p), GO);
#undef GO
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Outlet open-BC edges (residualEdge / openBC / storeEdge, Equations_mod.F90:
// 387-554, Residuals_mod.F90:599-624, Element_Calculations_mod.F90:852-924).
// One CTA per edge, 56 threads = the 56 FD evaluations.

template <int FORM>
__global__ void __launch_bounds__(64) k_edge64(const EdgeArgs a, const KParams prm, int want_jac)
{
    __shared__ double s_tl[3][54];
    __shared__ double s_res0[54];
    const int k = threadIdx.x;
    const int ed = blockIdx.x;
    const int e = a.edge_elem[ed];
    const int side = a.edge_id[ed] - 1;
    const double eps = prm.eps;
    if (k < 54) {
        const int inod = k / 6, f = k - 6 * (k / 6);
        const double v = a.TL[(size_t)f * a.nnodes + a.conn[inod * a.nel + e]];
        const double vp = v + eps;
        s_tl[0][k] = v;
        s_tl[2][k] = vp;
        s_tl[1][k] = vp - eps;
    }
    __syncthreads();
    const bool is_ac = (k == 55);
    const bool active = (k == 0) || (want_jac && (k < 55 || (is_ac && prm.nex > 0)));
    double res[54];
#pragma unroll
    for (int i = 0; i < 54; i++) res[i] = 0.0;
    if (active) {
        FdView V;
        V.orig = s_tl[0];
        V.rest = s_tl[1];
        V.pert = s_tl[2];
        V.kk = (k == 0) ? -1 : (is_ac ? 54 : k - 1);
        double WiN = prm.WiN;
        if (prm.nex > 0) {
            const double eu = a.EU[prm.nex - 1];
            WiN = prm.Wi0 * (is_ac ? eu + eps : eu);
        }
        double x[9], y[9];
#pragma unroll
        for (int n = 0; n < 9; n++) {
            const int gn = a.conn[n * a.nel + e];
            x[n] = a.xy[gn];
            y[n] = a.xy[a.nnodes + gn];
        }
        for (int ig = 0; ig < 3; ig++) {
            double dFx[9], dFy[9], d2x[9], d2y[9];
            const double *dfdc = c_edfdc[side][ig], *dfde = c_edfde[side][ig];
            auto go = geometry(c_ebfn[side][ig], dfdc, dfde, c_ed2c[side][ig],
                                 c_ed2e[side][ig], c_ed2ce[side][ig], 0.0, x, y, dFx, dFy, d2x,
                                 d2y);
            (void)go;
            auto I = interpolate(V, c_ebfn[side][ig], dFx, dFy, d2x, d2y);
            double dotU[9];
            auto g = gauss_point<FORM>(I, prm, WiN, go.H2, dFx, dFy, dotU);
            // setEdgeQuantities: normal from the tangent of the edge
            double dxdc = 0.0, dydc = 0.0, dxde = 0.0, dyde = 0.0;
#pragma unroll
            for (int n = 0; n < 9; n++) {
                dxdc = dxdc + dfdc[n] * x[n];
                dydc = dydc + dfdc[n] * y[n];
                dxde = dxde + dfde[n] * x[n];
                dyde = dyde + dfde[n] * y[n];
            }
            double n1, n2;
            switch (side) {
            case 0: n1 = dydc; n2 = -dxdc; break;
            case 1: n1 = dyde; n2 = -dxde; break;
            case 2: n1 = -dydc; n2 = dxdc; break;
            default: n1 = -dyde; n2 = dxde; break;
            }
            const double dL = sqrt(n1 * n1 + n2 * n2);
            n1 = n1 / dL;
            n2 = n2 / dL;
            const double WET = c_ew[ig] * dL;
            // openBC: TERM(i) = -(n . (P_tot(:,i) + P I(:,i))) * bifn
            const double c1a = g.P11 + I.P, c1b = g.P12;          // column 1
            const double c2a = g.P12, c2b = g.P22 + I.P;          // column 2
            const double q1 = n1 * c1a + n2 * c1b;
            const double q2 = n1 * c2a + n2 * c2b;
#pragma unroll
            for (int n = 0; n < 9; n++) {
                const double bf = c_ebfn[side][ig][n];
                res[n * 6 + 0] = res[n * 6 + 0] + (-q1 * bf) * WET;
                res[n * 6 + 1] = res[n * 6 + 1] + (-q2 * bf) * WET;
                res[n * 6 + 2] = res[n * 6 + 2] + 0.0 * WET;
                res[n * 6 + 3] = res[n * 6 + 3] + 0.0 * WET;
                res[n * 6 + 4] = res[n * 6 + 4] + 0.0 * WET;
                res[n * 6 + 5] = res[n * 6 + 5] + 0.0 * WET;
            }
        }
    }
    if (k == 0) {
#pragma unroll
        for (int i = 0; i < 54; i++) {
            s_res0[i] = res[i];
            a.rs[(size_t)ed * 54 + i] = res[i];
        }
    }
    __syncthreads();
    if (!active || k == 0) return;
    if (is_ac) {
#pragma unroll
        for (int i = 0; i < 54; i++) a.as[(size_t)ed * 54 + i] = (res[i] - s_res0[i]) / eps;
        return;
    }
    const int inod = (k - 1) / 6, ieq = (k - 1) - 6 * ((k - 1) / 6);
    double *dst = a.es + (size_t)ed * 2916 + inod * 36 + ieq;
#pragma unroll
    for (int jnod = 0; jnod < 9; jnod++)
#pragma unroll
        for (int jeq = 0; jeq < 6; jeq++)
            dst[jnod * 324 + jeq * 6] = (res[jnod * 6 + jeq] - s_res0[jnod * 6 + jeq]) / eps;
}

cudaError_t launch_edge64(const EdgeArgs &a, const KParams &p, int want_jac, cudaStream_t s)
{
    if (a.nedge <= 0) return cudaSuccess;
    if (p.form == FORM_SQRT)
        k_edge64<FORM_SQRT><<<a.nedge, 64, 0, s>>>(a, p, want_jac);
    else
        k_edge64<FORM_T><<<a.nedge, 64, 0, s>>>(a, p, want_jac);
    return cudaGetLastError();
}

}  // namespace vefem
