// Prism element kernel: residual and 18x18 tangent of every prism, fused
// with the scatter into the block-sparse Jacobian.
//
// Maths follows the reference's element routines (paths relative to
// TissueFolding/TissueFolding/SourceCode/):
//   Prism::calculateCurrNodalForces      Prism.cpp:749-874
//   ShapeBase::calculateForces3D         ShapeBase.cpp:2184-2235
//   neo-Hookean S, D81, Cauchy stress    ShapeBase.cpp:2284-2341
//   calculateImplicitKElastic            ShapeBase.cpp:2619-2639, :2786-2890
//   calculateImplicitKViscous            ShapeBase.cpp:2641-2705, :2892-3053
//   write*ToMainKatrix / ge, gv scatter  ShapeBase.cpp:2148-2180, :2707-2758
// with exact identities that cut the work:
//   * Fe C^-1 Fe^T = I, so sigma = (mu (b - I) + lambda lnJ I) / J with
//     b = Fe Fe^T, and the 3^6 contraction of integral 1 collapses to
//     lambda a_i b_k + (mu - lambda lnJ)(delta_ik a.b + a_k b_i);
//   * with a, b two gradient vectors, s = a.b and t = a.(sigma' b) the whole 3x3
//     block (elastic + both viscous integrals) of one Gauss point is the
//     bilinear form
//       B(a, b) = u_a b^T + b w_a^T - v_b a^T + s Q + t I
//     with  u_a = c1 a + sigma_v' a,  w_a = Q^T a,  v_b = sigma_v' b,
//     Q = c2 I + P, P = 0.5 eta w dV (I/dt - grad v) (primes: times w dV);
//     without viscosity B(a, b) = c1 a b^T + c2 b a^T + (c2 s + t) I = B(b, a)^T;
//   * the gradient of node (i, layer) is D_i1 L g_1 + D_i2 L g_2 + (+-) N_i/2 g_3
//     with g_j = grad xi_j the same for all nodes, D constants, L the layer's
//     weight at the two heights and N_i = 1/6 + delta_it/2 at the three
//     in-plane points t.  So the 36 node-pair blocks are weighted sums of the nine
//     blocks B(g_j, g_l) (six without viscosity) of the Gauss points, and the
//     weights are products of a height and an in-plane factor: the sums are taken
//     one factor at a time.  That is ~74,000 FP32 operations per prism in
//     place of ~136,000 for B(dN_a, dN_b) pair by pair;
//   * dx/dxi_j depends on the height (j = 1, 2) or on the in-plane point (j = 3)
//     only: formed once per prism and component, not once per Gauss point;
//     w dV = det(dx/dxi) / 6.
//
// Precision split.  GB300 issues FP32 FMAs at about 64 times its FP64 rate.
// The Gauss-point algebra (deformation gradient, stress, gradients, forces) is
// FP64.  The vectors the tangent's blocks are built from are split into
// double-float pairs x = hi + lo (two FP32 values, 48 significant bits and
// more) and the block sums run in double-float arithmetic on the FP32 pipe:
// products by Dekker's exact product (hi*hi and its rounding error by one FMA,
// plus the cross terms), sums by Knuth's two-sum, the low parts gathered in a
// second FP32 accumulator and renormalised (Dekker, "A floating-point technique
// for extending the available precision", 1971; Knuth, TAOCP vol. 2, 4.2.2).  A
// block entry carries a relative error of ~1e-13 of its largest term, far inside
// the 1e-11 parity bound and far below what moves a Newton iterate; the forces and
// everything the residual depends on stay FP64.  The splits and the joins work
// on the bit patterns: conversion instructions and additions would take the
// scarce FP64 pipe.
//
// Layout: one CTA of 12 x NE threads handles NE prisms, consecutive threads
// consecutive prisms throughout -- loads, shared memory and the atomics of a
// warp are then neighbours (with a warp on the node pairs of one prism every
// atomic went to a sector of its own).  A thread is (slot, prism), slot 0..11:
//   1. slots 0-5: dx/dxi and dv/dxi, one component each (FP64);
//   2. slots 0-5: one Gauss point each (FP64), split to shared memory;
//   3. the double-float vectors of the blocks; the nodal forces (FP64);
//   4. the blocks B(g_j, g_l) summed over what their weights share, staged in
//      shared memory;
//   5. the in-plane and height weights;
//   6. each node pair's block joined to FP64 and scattered.
// The loops over a phase's tasks stay rolled: unrolled they overflow the
// instruction cache.
// The phases of one CTA use one pipe at a time; three CTAs on an SM overlap them
// (with the u_j and s_jl kept in shared memory two fit: 2.58 against 1.94 ms).
// FP64 pipe and issue slots are each half busy: 1,496 FP64 instructions per prism
// (3,156 before), ~120,000 thread instructions per prism in all; the rest is the barriers
// between the phases (starting the CTAs of an SM in different phases: no change; two
// threads per Gauss point: 1.77 ms with viscosity, but 1.29 without).
// 320,000 prisms: 3.61 -> 1.84 ms with viscosity, 2.16 -> 1.25 ms without.  K's error,
// against sums in extended precision and against the pairwise form's (before), relative
// 2-norm: without viscosity 1.9e-15 to 2.9e-15 over 240 sheets of three shapes, 2.29e-15
// on average (before 2.0e-15 to 2.8e-15, 2.29e-15), the largest entry's 3.2e-15 of the
// largest entry (3.9e-15); with viscosity 2.3e-15 to 3.0e-15 over 12 sheets, 2.61e-15 on
// average (2.6e-15 to 3.2e-15, 2.81e-15), the largest entry's 3.7e-15 (4.4e-15).
// The matrix assembled is A = K^T, the system the reference
// solves (Pardiso iparm[11] = 1, NewtonRaphsonSolver.cpp:639); in that
// orientation every element block (a, b) lands at block (conn[a], conn[b])
// without a transpose.  Fixed DOFs are masked here, which is calcutateFixedK
// (NewtonRaphsonSolver.cpp:237-255) without a second pass.
#include <cstring>

#include "tf_internal.cuh"

namespace tf {

namespace {

enum Mode { kAtomic = 0, kStore = 2 };

constexpr int kSlots = 12;  // threads per prism

struct ElemArgs {
    int ne;
    const int* __restrict__ conn;
    const double* __restrict__ metric;  // [11][6][ne] (k_metric)
    const double* __restrict__ gx;
    const double* __restrict__ wdet;
    const double* __restrict__ invFg;
    const double* __restrict__ lam;
    const double* __restrict__ mu;
    const double* __restrict__ eta;
    const uint8_t* __restrict__ fixed;
    const int* __restrict__ slot;
    const double* __restrict__ uk;
    const double* __restrict__ vel;
    double idt;                 // 1 / dt
    double* __restrict__ val;   // kAtomic: block values
    double* __restrict__ g;     // kAtomic: right-hand side
    double* __restrict__ eblk;  // kStore: [9][36*ne]
    double* __restrict__ ef;    // kStore: [18][ne]
    // batches: elements of instances whose Newton loop has stopped are skipped
    const int* __restrict__ elem_seg;
    const int* __restrict__ seg_active;
    int masked;
    // parity evaluation (reference orientation), element-relative
    int e0, count;
    double* __restrict__ Ke;
    double* __restrict__ Kv;
    double* __restrict__ fe;
    double* __restrict__ fv;
    // checked build
    int nn;
    int64_t nval;
    int* check;
};

// Per-Gauss-point values in registers.
struct GaussPoint {
    double dn[18];   // current shape gradients dN_c (node-major)
    double sg[6];    // sigma' = w dV sigma     (00 11 22 01 02 12)
    double c1, c2;   // w dV lambda / J, w dV (mu - lambda lnJ) / J
    double sv[6];    // sigma_v' = w dV eta sym(grad v)
    double pv[9];    // P = 0.5 eta w dV (I/dt - grad v)
    double fe[9];    // Fe (row-major), kept for the adjoint
    double wdv;      // w dV
    double sc;       // w dV / J
};

__device__ __forceinline__ void sym_apply(const double* s, double d0, double d1, double d2, double* o) {
    o[0] = fma(s[0], d0, fma(s[3], d1, s[4] * d2));
    o[1] = fma(s[3], d0, fma(s[1], d1, s[5] * d2));
    o[2] = fma(s[4], d0, fma(s[5], d1, s[2] * d2));
}

// Prism::calculateCurrNodalForces (Prism.cpp:749-874) for Gauss point gp of
// element e, in closed form.
__device__ __forceinline__ void gauss_point(const ElemArgs& A, int e, int gp, bool visc, GaussPoint& G) {
    const int ne = A.ne;
    int nd[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        nd[a] = __ldg(&A.conn[a * ne + e]);
        if (!TF_IN(A.check, nd[a], A.nn, CK_ELEM_NODE)) nd[a] = 0;
    }
    double gX[18];
    const size_t q = 6 * (size_t)e + gp;
#pragma unroll
    for (int k = 0; k < 18; ++k) gX[k] = __ldg(&A.gx[(size_t)k * (6 * (size_t)ne) + q]);
    // F = sum_a x_a (x) dN_X,a.  The gradients sum to zero, so positions are
    // taken relative to node 0, which removes the cancellation of ~|x|/h
    // between the products far from the origin (exact arithmetic: no change).
    double F[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) F[k] = 0.0;
    const double o0 = A.uk[3 * nd[0]], o1 = A.uk[3 * nd[0] + 1], o2 = A.uk[3 * nd[0] + 2];
#pragma unroll
    for (int a = 1; a < 6; ++a) {
        const double x0 = A.uk[3 * nd[a]] - o0, x1 = A.uk[3 * nd[a] + 1] - o1, x2 = A.uk[3 * nd[a] + 2] - o2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            F[j] = fma(x0, gX[3 * a + j], F[j]);
            F[3 + j] = fma(x1, gX[3 * a + j], F[3 + j]);
            F[6 + j] = fma(x2, gX[3 * a + j], F[6 + j]);
        }
    }
    double iFg[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) iFg[k] = __ldg(&A.invFg[k * ne + e]);
    double Fe[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            Fe[3 * i + j] = fma(F[3 * i], iFg[j], fma(F[3 * i + 1], iFg[3 + j], F[3 * i + 2] * iFg[6 + j]));
    // Every multiply-add below is an explicit fma, so the rounding does not
    // depend on how the compiler contracts expressions in each instantiation
    // of the kernel (the order-fixed assembly stays bitwise reproducible
    // whatever tile the autotuner picks).
    const double J = fma(Fe[0], fma(Fe[4], Fe[8], -(Fe[5] * Fe[7])),
                         fma(-Fe[1], fma(Fe[3], Fe[8], -(Fe[5] * Fe[6])), Fe[2] * fma(Fe[3], Fe[7], -(Fe[4] * Fe[6]))));
    const double lnJ = log(J);
    const double rJ = 1.0 / J;
    const double lam = __ldg(&A.lam[e]), mu = __ldg(&A.mu[e]);
    double b[6];
    b[0] = fma(Fe[0], Fe[0], fma(Fe[1], Fe[1], Fe[2] * Fe[2]));
    b[1] = fma(Fe[3], Fe[3], fma(Fe[4], Fe[4], Fe[5] * Fe[5]));
    b[2] = fma(Fe[6], Fe[6], fma(Fe[7], Fe[7], Fe[8] * Fe[8]));
    b[3] = fma(Fe[0], Fe[3], fma(Fe[1], Fe[4], Fe[2] * Fe[5]));
    b[4] = fma(Fe[0], Fe[6], fma(Fe[1], Fe[7], Fe[2] * Fe[8]));
    b[5] = fma(Fe[3], Fe[6], fma(Fe[4], Fe[7], Fe[5] * Fe[8]));
    double cf[9];  // cofactors: F^-T = cf / det F
    cf[0] = fma(F[4], F[8], -(F[5] * F[7]));
    cf[1] = fma(F[5], F[6], -(F[3] * F[8]));
    cf[2] = fma(F[3], F[7], -(F[4] * F[6]));
    cf[3] = fma(F[2], F[7], -(F[1] * F[8]));
    cf[4] = fma(F[0], F[8], -(F[2] * F[6]));
    cf[5] = fma(F[1], F[6], -(F[0] * F[7]));
    cf[6] = fma(F[1], F[5], -(F[2] * F[4]));
    cf[7] = fma(F[2], F[3], -(F[0] * F[5]));
    cf[8] = fma(F[0], F[4], -(F[1] * F[3]));
    const double detF = fma(F[0], cf[0], fma(F[1], cf[1], F[2] * cf[2]));
    const double rdF = 1.0 / detF;
    const double wdV = __ldg(&A.wdet[q]) * detF;
    G.wdv = wdV;
#pragma unroll
    for (int k = 0; k < 9; ++k) G.fe[k] = Fe[k];
    const double sc = wdV * rJ;
    G.sc = sc;
    const double dterm = fma(lam, lnJ, -mu);
    G.sg[0] = sc * fma(mu, b[0], dterm);
    G.sg[1] = sc * fma(mu, b[1], dterm);
    G.sg[2] = sc * fma(mu, b[2], dterm);
    G.sg[3] = sc * mu * b[3];
    G.sg[4] = sc * mu * b[4];
    G.sg[5] = sc * mu * b[5];
    G.c1 = sc * lam;
    G.c2 = sc * fma(-lam, lnJ, mu);
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        const double g0 = gX[3 * a], g1 = gX[3 * a + 1], g2 = gX[3 * a + 2];
        G.dn[3 * a] = rdF * fma(cf[0], g0, fma(cf[1], g1, cf[2] * g2));
        G.dn[3 * a + 1] = rdF * fma(cf[3], g0, fma(cf[4], g1, cf[5] * g2));
        G.dn[3 * a + 2] = rdF * fma(cf[6], g0, fma(cf[7], g1, cf[8] * g2));
    }
    if (visc) {
        // grad v = sum_c v_c (x) dN_c (ShapeBase.cpp:2892-2919), velocities
        // relative to node 0 for the same reason as the positions
        double L[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) L[k] = 0.0;
        const double w0 = A.vel[3 * nd[0]], w1 = A.vel[3 * nd[0] + 1], w2 = A.vel[3 * nd[0] + 2];
#pragma unroll
        for (int c = 1; c < 6; ++c) {
            const double v0 = A.vel[3 * nd[c]] - w0, v1 = A.vel[3 * nd[c] + 1] - w1, v2 = A.vel[3 * nd[c] + 2] - w2;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                L[j] = fma(v0, G.dn[3 * c + j], L[j]);
                L[3 + j] = fma(v1, G.dn[3 * c + j], L[3 + j]);
                L[6 + j] = fma(v2, G.dn[3 * c + j], L[6 + j]);
            }
        }
        const double eta = __ldg(&A.eta[e]);
        const double ew = eta * wdV;
        const double hw = 0.5 * ew;
        G.sv[0] = ew * L[0];
        G.sv[1] = ew * L[4];
        G.sv[2] = ew * L[8];
        G.sv[3] = hw * (L[1] + L[3]);
        G.sv[4] = hw * (L[2] + L[6]);
        G.sv[5] = hw * (L[5] + L[7]);
#pragma unroll
        for (int k = 0; k < 9; ++k) G.pv[k] = -hw * L[k];
        G.pv[0] = fma(hw, A.idt, G.pv[0]);
        G.pv[4] = fma(hw, A.idt, G.pv[4]);
        G.pv[8] = fma(hw, A.idt, G.pv[8]);
    }
}

// ---- double-float arithmetic (phase B) ----------------------------------
// A value is hi + lo with hi, lo FP32.  Every operation is an explicit
// rounding intrinsic, so no instantiation of the kernel contracts or
// reassociates differently (the order-fixed assembly stays bitwise
// reproducible whatever tile the autotuner picks).

// x = hi + lo on the bit pattern: hi is x rounded to 24 significant bits (half
// away from zero; the carry runs into the exponent), lo the rest as an integer
// of 29 signed bits, scaled (in two factors: 2^(exponent - 52) itself can lie below
// FP32's normal range).  Magnitudes below FP32's normal range become a signed zero, those above
// it infinity; NaN and infinity stay so.
__device__ __forceinline__ float2 df_split(double x) {
    const unsigned l = __double2loint(x), h = __double2hiint(x);
    const unsigned sgn = h & 0x80000000u;
    const int e = (int)((h >> 20) & 0x7ffu);
    const unsigned l2 = l + (1u << 28), h2 = h + (l2 < l ? 1u : 0u);
    unsigned f = sgn | ((((h2 >> 20) & 0x7ffu) - 896u) << 23) | ((h2 & 0xfffffu) << 3) | (l2 >> 29);
    f = e > 896 ? f : sgn;
    f = e > 1150 ? (sgn | 0x7f800000u | ((e == 0x7ff && (h & 0xfffffu)) ? 0x400000u : 0u)) : f;
    const float scale = __uint_as_float(sgn | ((unsigned)(e - 896) << 23));  // 2^exponent
    const float lo = __int2float_rn((int)(l2 & 0x1fffffffu) - (1 << 28)) * 0x1p-52f * scale;
    return make_float2(__uint_as_float(f), (e > 896 && e <= 1150) ? lo : 0.f);
}

// hi + lo as a double on the bit patterns; |lo| at most half an ulp of hi (after
// df_norm).  The 24 bits of hi, shifted to a double's 53, plus or minus those of
// lo at their place (bits below a double's last are cut off: an error under one
// ulp of the double, a hundredth of what the pair carries).
__device__ __forceinline__ double df_join(float hi, float lo) {
    const unsigned uh = __float_as_uint(hi), ul = __float_as_uint(lo);
    const int eh = (int)((uh >> 23) & 0xffu), el = (int)((ul >> 23) & 0xffu);
    const unsigned long long mh = (unsigned long long)((uh & 0x7fffffu) | 0x800000u) << 29;
    const unsigned long long ml = el ? (unsigned long long)((ul & 0x7fffffu) | 0x800000u) << 29 : 0ull;
    const unsigned long long t = ml >> min(eh - el, 63);
    const unsigned long long m = ((uh ^ ul) & 0x80000000u) ? mh - t : mh + t;
    // the leading bit of m adds one to the exponent; a difference may have lost it
    const bool low = m < (1ull << 52);
    const unsigned long long b = low ? ((unsigned long long)(eh + 894) << 52) + (m << 1)
                                     : ((unsigned long long)(eh + 895) << 52) + m;
    const unsigned long long sgn = (unsigned long long)(uh & 0x80000000u) << 32;
    unsigned long long r = sgn | b;
    if (eh == 0) r = sgn;
    if (eh == 0xff) r = sgn | 0x7ff0000000000000ull | ((uh & 0x7fffffu) ? 0x8000000000000ull : 0ull);
    return __longlong_as_double((long long)r);
}

// (H, L) += x * y: Dekker's product (the rounding error of hi*hi by one FMA,
// the cross terms into the low word; lo*lo is below the format's precision),
// Knuth's two-sum of the high words, the error into the low word.
__device__ __forceinline__ void df_mac(float& H, float& L, float2 x, float2 y) {
    const float p = __fmul_rn(x.x, y.x);
    float e = __fmaf_rn(x.x, y.x, -p);
    e = __fmaf_rn(x.x, y.y, e);
    e = __fmaf_rn(x.y, y.x, e);
    const float s = __fadd_rn(H, p);
    const float bb = __fsub_rn(s, H);
    const float err = __fadd_rn(__fsub_rn(H, __fsub_rn(s, bb)), __fsub_rn(p, bb));
    L = __fadd_rn(L, __fadd_rn(err, e));
    H = s;
}

// (H, L) += x
__device__ __forceinline__ void df_add(float& H, float& L, float2 x) {
    const float s = __fadd_rn(H, x.x);
    const float bb = __fsub_rn(s, H);
    const float err = __fadd_rn(__fsub_rn(H, __fsub_rn(s, bb)), __fsub_rn(x.x, bb));
    L = __fadd_rn(L, __fadd_rn(err, x.y));
    H = s;
}

// Fast two-sum: the low word brought back under half an ulp of the high word.
__device__ __forceinline__ void df_norm(float& H, float& L) {
    const float s = __fadd_rn(H, L);
    L = __fsub_rn(L, __fsub_rn(s, H));
    H = s;
}

// c x, c a double-float constant
__device__ __forceinline__ float2 df_scale(float2 c, float2 x) {
    float p = __fmul_rn(c.x, x.x);
    float e = __fmaf_rn(c.x, x.x, -p);
    e = __fmaf_rn(c.x, x.y, e);
    e = __fmaf_rn(c.y, x.x, e);
    df_norm(p, e);
    return make_float2(p, e);
}
// x + y.  FULL: both words by two-sums (the low words' rounding carried too),
// else the low words simply added.
template <bool FULL>
__device__ __forceinline__ float2 df_sum(float2 x, float2 y) {
    if constexpr (!FULL) {
        df_add(x.x, x.y, y);
        df_norm(x.x, x.y);
        return x;
    } else {
        float s = __fadd_rn(x.x, y.x);
        float bb = __fsub_rn(s, x.x);
        float e = __fadd_rn(__fsub_rn(x.x, __fsub_rn(s, bb)), __fsub_rn(y.x, bb));
        const float t = __fadd_rn(x.y, y.y);
        bb = __fsub_rn(t, x.y);
        const float ee = __fadd_rn(__fsub_rn(x.y, __fsub_rn(t, bb)), __fsub_rn(y.y, bb));
        e = __fadd_rn(e, t);
        df_norm(s, e);
        e = __fadd_rn(e, ee);
        df_norm(s, e);
        return make_float2(s, e);
    }
}
// m + c x, c a small integer (the product's error by one FMA)
__device__ __forceinline__ float2 df_muladd(float2 m, float c, float2 x) {
    df_mac(m.x, m.y, make_float2(c, 0.f), x);
    df_norm(m.x, m.y);
    return m;
}
// (H, L) += s x, s = +-1 (the products are exact).  FULL: the low words' sum by
// a two-sum too, its rounding gathered in E.
template <bool FULL>
__device__ __forceinline__ void df_addmul(float& H, float& L, float& E, float s, float2 x) {
    const float t = __fmaf_rn(s, x.x, H);
    float bb = __fsub_rn(t, H);
    const float err = __fadd_rn(__fsub_rn(H, __fsub_rn(t, bb)), __fmaf_rn(s, x.x, -bb));
    H = t;
    if constexpr (!FULL) {
        L = __fadd_rn(L, __fmaf_rn(s, x.y, err));
    } else {
        const float l = __fadd_rn(L, err);
        bb = __fsub_rn(l, L);
        E = __fadd_rn(E, __fadd_rn(__fsub_rn(L, __fsub_rn(l, bb)), __fsub_rn(err, bb)));
        L = __fmaf_rn(s, x.y, l);
        bb = __fsub_rn(L, l);
        E = __fadd_rn(E, __fadd_rn(__fsub_rn(l, __fsub_rn(L, bb)), __fmaf_rn(s, x.y, -bb)));
    }
}
// s x, s a power of two or its negative (exact)
__device__ __forceinline__ float2 df_pow2(float s, float2 x) { return make_float2(s * x.x, s * x.y); }
__device__ __forceinline__ float2 df_neg(float2 x) { return make_float2(-x.x, -x.y); }

constexpr double kSqrt3 = 1.73205080756887729353;
constexpr float df_hi(double x) { return (float)x; }
constexpr float df_lo(double x) { return (float)(x - (double)(float)x); }
#define DF_CONST(x) make_float2(df_hi(x), df_lo(x))

__device__ __forceinline__ bool element_live(const ElemArgs& A, int e) {
    return e < A.ne && (!A.masked || A.seg_active[A.elem_seg[e]] != 0);
}

// Index of (j, l) in the order 00 11 22 01 02 12.
__device__ __forceinline__ int sym_index(int j, int l) { return j == l ? j : j + l + 2; }

// Shared memory of a CTA, the prism fastest everywhere.
//   gp: double-float vectors of the Gauss points, [value][gp][NE]: the gradients
//       g_1/sqrt(3), g_2/sqrt(3), g_3/12 (G; the weights of phase 4 are then small
//       integers but for one factor; the forces' weights and the velocities carry
//       the inverse), their w_j (W) and with viscosity v_j, Q, t_jl
//       and c1 (u_j and s_jl are formed again in phase 4: their room would cost a
//       CTA per SM), without it u_j and d_jl = c2 s_jl + t_jl (U, D);
//   st: staged 3x3 blocks, [block][9][NE]: A_jl(height), j, l in {1, 2}, then
//       M_jl(layers bb, bt) in their place; B(g_j, g_3)(height, in-plane point)
//       and with viscosity B(g_3, g_l), then H(layer, node) in their place; and
//       B(g_3, g_3)(in-plane point), without viscosity per height.  M_jl(tt) and
//       W(node pair i <= k) go where gp was.
// st first holds what only the phases before need: dx/dxi and dv/dxi
// [2][7][3][NE] in FP64 (X), (sigma' + sigma_v') g_j [9][gp][NE] in FP64 for the
// forces (F), and [value][gp][NE] (C): with viscosity sigma', sigma_v', without it c1,
// c2 and sigma' g_j, formed in FP64 for the forces anyway.
template <bool VISC>
struct Lay {
    static constexpr int G = 0, W = 9, V = 18, Q = 27, T = 36, K1 = 42, U = 18, D = 27;
    static constexpr int NV = VISC ? 43 : 33;
    static constexpr int NJL = VISC ? 4 : 3;             // pairs (j, l) of {1, 2}
    static constexpr int NR = VISC ? 4 : 2;              // (1,3) (2,3) and with viscosity (3,1) (3,2)
    static constexpr int BA = 0;                         // [NJL][2]
    static constexpr int BR = 2 * NJL;                   // [NR][2][3]
    static constexpr int BB = BR + 6 * NR;               // [3], without viscosity [2][3]
    static constexpr int NB = BB + (VISC ? 3 : 6);
    static constexpr int XM = 0, XW = NJL;               // blocks in gp's place: [NJL], [6]
    static constexpr int SG = 0, SV = 6;                 // values of C with viscosity (c1 is in gp, c2 in Q)
    static constexpr int C1 = 0, C2 = 1, SF = 2;         // ... and without
    static constexpr int NC = VISC ? 12 : 11;
};
template <int NE, bool VISC>
constexpr size_t elem_smem() {
    using Y = Lay<VISC>;
    static_assert(8 * 42 + 8 * 54 + 8 * 6 * Y::NC <= 72 * Y::NB, "X, F and C fit st");
    return sizeof(float2) * NE * (Y::NV * 6 + Y::NB * 9);
}

// B(g_j, g_l) of Gauss point gp into (H, L)[9]
template <int NE, bool VISC>
__device__ __forceinline__ void gp_block(const float2* __restrict__ sg, int j, int l, int gp, int el, float (&H)[9],
                                         float (&L)[9]) {
    using Y = Lay<VISC>;
    auto at = [&](int v) { return sg[(v * 6 + gp) * NE + el]; };
    const int jl = sym_index(j, l);
    const float2 b[3] = {at(Y::G + 3 * l), at(Y::G + 3 * l + 1), at(Y::G + 3 * l + 2)};
    float2 u[3];
    if constexpr (VISC) {  // u = c1 g + sigma_v' g
        const float2 c1 = at(Y::K1);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            u[i] = at(Y::V + 3 * j + i);
            df_mac(u[i].x, u[i].y, c1, at(Y::G + 3 * j + i));
            df_norm(u[i].x, u[i].y);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) u[i] = at(Y::U + 3 * j + i);
    }
    const float2 w[3] = {at(Y::W + 3 * j), at(Y::W + 3 * j + 1), at(Y::W + 3 * j + 2)};
#pragma unroll
    for (int k = 0; k < 9; ++k) {  // u b^T: the first product needs no sum
        const float2 x = u[k / 3], y = b[k % 3];
        H[k] = __fmul_rn(x.x, y.x);
        L[k] = __fmaf_rn(x.y, y.x, __fmaf_rn(x.x, y.y, __fmaf_rn(x.x, y.x, -H[k])));
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) df_mac(H[k], L[k], b[k / 3], w[k % 3]);
    if constexpr (VISC) {
        const float2 a[3] = {at(Y::G + 3 * j), at(Y::G + 3 * j + 1), at(Y::G + 3 * j + 2)};
        const float2 v[3] = {df_neg(at(Y::V + 3 * l)), df_neg(at(Y::V + 3 * l + 1)), df_neg(at(Y::V + 3 * l + 2))};
        const float2 t = at(Y::T + jl);
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 3; ++i) df_mac(s.x, s.y, a[i], b[i]);
        df_norm(s.x, s.y);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            df_mac(H[k], L[k], v[k / 3], a[k % 3]);
            df_mac(H[k], L[k], s, at(Y::Q + k));
            if (k % 4 == 0) df_add(H[k], L[k], t);
        }
    } else {
        const float2 d = at(Y::D + jl);
#pragma unroll
        for (int k = 0; k < 9; k += 4) df_add(H[k], L[k], d);
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) df_norm(H[k], L[k]);
}

// o = s d for a symmetric s (00 11 22 01 02 12), in double-float
__device__ __forceinline__ void df_sym_apply(const float2* s, const float2* d, float2* o) {
    const int ix[9] = {0, 3, 4, 3, 1, 5, 4, 5, 2};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float H = 0.0f, L = 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) df_mac(H, L, s[ix[3 * i + j]], d[j]);
        df_norm(H, L);
        o[i] = make_float2(H, L);
    }
}

// Node pairs a <= b of the symmetric (inviscid) case.
__constant__ int8_t kPairA[21] = {0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, 2, 2, 2, 2, 3, 3, 3, 4, 4, 5};
__constant__ int8_t kPairB[21] = {0, 1, 2, 3, 4, 5, 1, 2, 3, 4, 5, 2, 3, 4, 5, 3, 4, 5, 4, 5, 5};

template <int NE, int MODE, bool VISC>
__global__ void __launch_bounds__(NE* kSlots, 48 / NE) k_element(ElemArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Y = Lay<VISC>;
    float2* sg = reinterpret_cast<float2*>(smem_raw);     // [NV][6][NE]
    float2* st = sg + Y::NV * 6 * NE;                     // [NB][9][NE]
    double* sx = reinterpret_cast<double*>(st);           // X [2][7][3][NE]
    double* hf = sx + 42 * NE;                            // F [9][6][NE]
    float2* sc0 = reinterpret_cast<float2*>(hf + 54 * NE);  // C [NC][6][NE]
    const int el = threadIdx.x % NE, slot = threadIdx.x / NE;
    const int e = blockIdx.x * NE + el;
    const bool live = element_live(A, e);
    if (!__syncthreads_or(live)) return;
    const int ne = A.ne;

    // ---- 1. dx/dxi_1, dx/dxi_2 at both heights, dx/dxi_3 at the in-plane points
    // (component slot % 3), and dv/dxi likewise times sqrt(3), sqrt(3) and 12 (the
    // gradients come divided by these): apical weight (1 + zeta)/2 = b at the first
    // height, a at the second
    constexpr double wa = 0.5 - kSqrt3 / 6.0, wb = 0.5 + kSqrt3 / 6.0;
    if (live && slot < (VISC ? 6 : 3)) {
        const int c = slot % 3;
        const double* __restrict__ src = slot < 3 ? A.uk : A.vel;
        double x[6];
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            int nd = __ldg(&A.conn[a * ne + e]);
            if (!TF_IN(A.check, nd, A.nn, CK_ELEM_NODE)) nd = 0;
            x[a] = src[3 * nd + c];
        }
        double* o = sx + (size_t)(slot / 3) * 21 * NE + c * NE + el;
        const bool vel = slot >= 3;
        const double a = vel ? kSqrt3 * wa : wa, b = vel ? kSqrt3 * wb : wb;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double lo = x[1 + j] - x[0], up = x[4 + j] - x[3];
            o[(2 * j) * 3 * NE] = fma(a, lo, b * up);
            o[(2 * j + 1) * 3 * NE] = fma(b, lo, a * up);
        }
        const double d[3] = {x[3] - x[0], x[4] - x[1], x[5] - x[2]};
        const double m = (d[0] + d[1] + d[2]) * (vel ? 1.0 : 1.0 / 12.0), q = vel ? 3.0 : 0.25;
#pragma unroll
        for (int t = 0; t < 3; ++t) o[(4 + t) * 3 * NE] = fma(q, d[t], m);
    }
    __syncthreads();

    // ---- 2. the Gauss points: Prism::calculateCurrNodalForces (Prism.cpp:749-874)
    // in closed form.  Every multiply-add is an explicit fma, so the rounding does
    // not depend on how the compiler contracts expressions in each instantiation
    // (the order-fixed assembly stays bitwise reproducible whatever tile the
    // autotuner picks).
    if (live && slot < kGauss) {
        const int gp = slot, t = gp % 3, hgt = gp / 3;
        auto col = [&](int q, int j, int i) {  // dx_i/dxi_j (q = 0), dv_i/dxi_j (1)
            const int m = j == 2 ? 4 + t : 2 * j + hgt;
            return sx[((size_t)(q * 7 + m) * 3 + i) * NE + el];
        };
        double X[9];  // X[3 j + i] = dx_i / dxi_j
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) X[3 * j + i] = col(0, j, i);
        double g[9];  // g[3 j + i]: the cofactors, then grad xi_j over sqrt(3), sqrt(3), 12
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double* p = X + 3 * ((j + 1) % 3);
            const double* q = X + 3 * ((j + 2) % 3);
            g[3 * j] = fma(p[1], q[2], -(p[2] * q[1]));
            g[3 * j + 1] = fma(p[2], q[0], -(p[0] * q[2]));
            g[3 * j + 2] = fma(p[0], q[1], -(p[1] * q[0]));
        }
        const double det = fma(X[0], g[0], fma(X[1], g[1], X[2] * g[2]));
        // Fe = X^T M, M = dxi/dX Fg^-1; b = Fe Fe^T; J = det M det X
        double Fe[9], b[6];  // b: 00 11 22 01 02 12
        const double* __restrict__ me = A.metric + (size_t)gp * ne + e;
        const size_t st6 = (size_t)6 * ne;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double a0 = __ldg(&me[k * st6]), a1 = __ldg(&me[(3 + k) * st6]), a2 = __ldg(&me[(6 + k) * st6]);
#pragma unroll
            for (int i = 0; i < 3; ++i) Fe[3 * i + k] = fma(X[i], a0, fma(X[3 + i], a1, X[6 + i] * a2));
        }
        {
            auto bij = [&](int i, int k) {
                return fma(Fe[3 * i], Fe[3 * k], fma(Fe[3 * i + 1], Fe[3 * k + 1], Fe[3 * i + 2] * Fe[3 * k + 2]));
            };
            b[0] = bij(0, 0);
            b[1] = bij(1, 1);
            b[2] = bij(2, 2);
            b[3] = bij(0, 1);
            b[4] = bij(0, 2);
            b[5] = bij(1, 2);
        }
        const double lnJ = log(det * __ldg(&me[9 * st6]));
        const double sc = __ldg(&me[10 * st6]);  // w dV / J
        const double wdV = det * (1.0 / 6.0);
        const double rd = 1.0 / det;
        float2* out = sg + gp * NE + el;
        auto put = [&](int v, double x) { out[(size_t)v * 6 * NE] = df_split(x); };
        {
            const double r1 = rd * (1.0 / kSqrt3), r3 = rd * (1.0 / 12.0);
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                g[k] *= k < 6 ? r1 : r3;
                put(Y::G + k, g[k]);
            }
        }
        const double lam = __ldg(&A.lam[e]), mu = __ldg(&A.mu[e]);
        const double dterm = fma(lam, lnJ, -mu);
        float2* outc = sc0 + gp * NE + el;
        auto putc = [&](int v, double x) { outc[(size_t)v * 6 * NE] = df_split(x); };
        // c1 = w dV lambda / J, c2 = w dV (mu - lambda lnJ) / J
        if constexpr (VISC) put(Y::K1, sc * lam);
        else putc(Y::C1, sc * lam);
        const double c2d = -sc * dterm;
        double sgm[6];  // sigma' = w dV sigma (00 11 22 01 02 12)
        const double sm = sc * mu;
#pragma unroll
        for (int k = 0; k < 3; ++k) sgm[k] = sc * fma(mu, b[k], dterm);
#pragma unroll
        for (int k = 3; k < 6; ++k) sgm[k] = sm * b[k];
        if constexpr (VISC) {
#pragma unroll
            for (int k = 0; k < 6; ++k) putc(Y::SG + k, sgm[k]);
            // grad v = sum_j dv/dxi_j (x) g_j (ShapeBase.cpp:2892-2919), the scales of
            // the two cancelling; a prism without viscosity has eta = 0 and these terms vanish
            double Lg[9];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const double v0 = col(1, 0, i), v1 = col(1, 1, i), v2 = col(1, 2, i);
#pragma unroll
                for (int k = 0; k < 3; ++k) Lg[3 * i + k] = fma(v0, g[k], fma(v1, g[3 + k], v2 * g[6 + k]));
            }
            const double eta = __ldg(&A.eta[e]);
            const double ew = eta * wdV, hw = 0.5 * ew;
            const bool visc = eta != 0.0;
            double sv[6];  // sigma_v' = w dV eta sym(grad v)
            sv[0] = ew * Lg[0];
            sv[1] = ew * Lg[4];
            sv[2] = ew * Lg[8];
            sv[3] = hw * (Lg[1] + Lg[3]);
            sv[4] = hw * (Lg[2] + Lg[6]);
            sv[5] = hw * (Lg[5] + Lg[7]);
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                sv[k] = visc ? sv[k] : 0.0;
                putc(Y::SV + k, sv[k]);
                sgm[k] += sv[k];  // one stress for the forces
            }
            // Q = c2 I + P, P = 0.5 eta w dV (I/dt - grad v)
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const double p = visc ? (k % 4 == 0 ? hw * (A.idt - Lg[k]) : -hw * Lg[k]) : 0.0;
                put(Y::Q + k, k % 4 == 0 ? c2d + p : p);
            }
        } else {
            putc(Y::C2, c2d);
        }
        double* ho = hf + gp * NE + el;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            double h3[3];
            sym_apply(sgm, g[3 * j], g[3 * j + 1], g[3 * j + 2], h3);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                ho[(size_t)(3 * j + i) * 6 * NE] = h3[i];
                if constexpr (!VISC) putc(Y::SF + 3 * j + i, h3[i]);
            }
        }
    }
    __syncthreads();

    // ---- 3. the double-float vectors of every (Gauss point, g_j): its own ones in
    // the first 18 tasks, its products with the other gradients in the last 18; then
    // the nodal forces on slots 6-8
#pragma unroll 1
    for (int task = slot; task < 36; task += kSlots) {
        const int gp = task % 6, j = (task / 6) % 3;
        auto at = [&](int v) -> float2& { return sg[(v * 6 + gp) * NE + el]; };
        auto ct = [&](int v) { return sc0[(v * 6 + gp) * NE + el]; };
        const float2 a[3] = {at(Y::G + 3 * j), at(Y::G + 3 * j + 1), at(Y::G + 3 * j + 2)};
        float2 s6[6], o[3];
        if (task < 18) {
            if constexpr (VISC) {
#pragma unroll
                for (int k = 0; k < 6; ++k) s6[k] = ct(Y::SV + k);
                df_sym_apply(s6, a, o);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    at(Y::V + 3 * j + i) = o[i];
                    float wH = 0.f, wL = 0.f;  // w = Q^T g
#pragma unroll
                    for (int k = 0; k < 3; ++k) df_mac(wH, wL, at(Y::Q + 3 * k + i), a[k]);
                    df_norm(wH, wL);
                    at(Y::W + 3 * j + i) = make_float2(wH, wL);
                }
            } else {
                const float2 c1 = ct(Y::C1), c2 = ct(Y::C2);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    at(Y::U + 3 * j + i) = df_scale(c1, a[i]);
                    at(Y::W + 3 * j + i) = df_scale(c2, a[i]);
                }
            }
        } else {
            if constexpr (VISC) {
#pragma unroll
                for (int k = 0; k < 6; ++k) s6[k] = ct(Y::SG + k);
                df_sym_apply(s6, a, o);
            } else {
#pragma unroll
                for (int i = 0; i < 3; ++i) o[i] = ct(Y::SF + 3 * j + i);
            }
#pragma unroll 1
            for (int l = j; l < 3; ++l) {
                float sH = 0.f, sL = 0.f, tH = 0.f, tL = 0.f;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float2 b = at(Y::G + 3 * l + i);
                    df_mac(tH, tL, o[i], b);
                    if constexpr (!VISC) df_mac(sH, sL, a[i], b);
                }
                if constexpr (!VISC) {
                    df_norm(sH, sL);
                    df_mac(tH, tL, ct(Y::C2), make_float2(sH, sL));
                }
                df_norm(tH, tL);
                at((VISC ? Y::T : Y::D) + sym_index(j, l)) = make_float2(tH, tL);
            }
        }
    }
    // component c of the forces: f_a = - sum_g (sigma' + sigma_v') dN_a
    // (ShapeBase.cpp:2203-2227), the weights one factor at a time
    if (live && slot >= 6 && slot < 9) {
        const int c = slot - 6;
        auto h = [&](int j, int gp) { return hf[((size_t)(3 * j + c) * 6 + gp) * NE + el]; };
        double T[2][2], z[3];  // T[j][layer]
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double s0 = h(j, 0) + h(j, 1) + h(j, 2), s1 = h(j, 3) + h(j, 4) + h(j, 5);
            T[j][0] = fma(kSqrt3 * wa, s0, (kSqrt3 * wb) * s1);
            T[j][1] = fma(kSqrt3 * wb, s0, (kSqrt3 * wa) * s1);
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) z[t] = h(2, t) + h(2, 3 + t);
        const double zs = z[0] + z[1] + z[2];
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            const int i = a % 3, up = a / 3;
            const double in = i == 0 ? -(T[0][up] + T[1][up]) : T[i - 1][up];
            const double zi = fma(3.0, z[i], zs);
            const double f = up ? -(in + zi) : zi - in;
            const int node = __ldg(&A.conn[a * ne + e]);
            if (!TF_IN(A.check, node, A.nn, CK_ELEM_NODE)) continue;
            const bool fx = A.fixed[3 * node + c] != 0;
            if (MODE == kStore) A.ef[(size_t)(3 * a + c) * ne + e] = fx ? 0.0 : f;
            else if (!fx) atomicAdd(&A.g[3 * node + c], f);
        }
    }
    __syncthreads();

    // ---- 4. the blocks B(g_j, g_l), one Gauss point after the other: a unit is
    // stored by itself or added to the units before it (A_jl over the in-plane
    // points; B(g_3, g_3) over the heights with viscosity)
    auto blk = [&](int b) { return st + (size_t)b * 9 * NE + el; };
    {
        float SH[9], SL[9];
        constexpr int kUnits = VISC ? 5 : 3;
#pragma unroll 1
        for (int u = 0; u < kUnits; ++u) {
            int j, l, gp, b;
            bool first = true, last = true;
            if (VISC && u < 2) {  // slots 0-5: (j, 3), 6-11: (3, l); both heights
                const int t = (slot / 2) % 3;
                j = slot < 6 ? slot % 2 : 2;
                l = slot < 6 ? 2 : slot % 2;
                gp = 3 * u + t;
                b = Y::BR + 6 * (slot < 6 ? slot % 2 : 2 + slot % 2) + gp;
            } else if (VISC) {
                if (slot < 8) {
                    j = slot / 4;
                    l = (slot / 2) % 2;
                    gp = 3 * (slot % 2) + u - 2;
                    b = Y::BA + slot;
                    first = u == 2;
                    last = u == 4;
                } else {
                    if (slot == 11 || u == 4) break;
                    j = l = 2;
                    gp = slot - 8 + 3 * (u - 2);
                    b = Y::BB + slot - 8;
                    first = u == 2;
                    last = u == 3;
                }
            } else if (slot < 6) {  // A_jl, pairs 11 12 22
                j = slot / 4;
                l = slot < 2 ? 0 : 1;
                gp = 3 * (slot % 2) + u;
                b = Y::BA + slot;
                first = u == 0;
                last = u == 2;
            } else if (u < 2) {
                const int q = slot - 6;
                j = q % 2;
                l = 2;
                gp = 3 * u + q / 2;
                b = Y::BR + 6 * j + gp;
            } else {
                j = l = 2;
                gp = slot - 6;
                b = Y::BB + gp;
            }
            float H[9], L[9];
            gp_block<NE, VISC>(sg, j, l, gp, el, H, L);
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                if (!first) {
                    const float2 x = df_sum<false>(make_float2(SH[k], SL[k]), make_float2(H[k], L[k]));
                    H[k] = x.x;
                    L[k] = x.y;
                }
                SH[k] = H[k];
                SL[k] = L[k];
            }
            if (last) {
                float2* o = blk(b);
#pragma unroll
                for (int k = 0; k < 9; ++k) o[k * NE] = make_float2(H[k], L[k]);
            }
        }
    }
    __syncthreads();

    // ---- 5. the weights, entry by entry -----------------------------------------
    auto xblk = [&](int b) { return sg + (size_t)b * 9 * NE + el; };
    constexpr bool kFull = !VISC;
    {
        // H(layer, k) = sum over the in-plane points and heights of N_k/2 L_layer B:
        // S + 3 (k) in the plane, sqrt(3)/2 (B0 + B1) -+ (B0 - B1)/2 over the heights
        constexpr int kGroups = kSlots / Y::NR;
        float2* r = blk(Y::BR + 6 * (slot % Y::NR));
#pragma unroll 1
        for (int k = slot / Y::NR; k < 9; k += kGroups) {
            float2 p[3], d[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float2 x = r[(9 * t + k) * NE], y = r[(9 * (3 + t) + k) * NE];
                p[t] = df_scale(DF_CONST(0.5 * kSqrt3), df_sum<kFull>(x, y));
                d[t] = df_pow2(0.5f, df_sum<kFull>(x, df_neg(y)));
            }
            const float2 ps = df_sum<kFull>(df_sum<kFull>(p[0], p[1]), p[2]);
            const float2 ds = df_sum<kFull>(df_sum<kFull>(d[0], d[1]), d[2]);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float2 x = df_muladd(ps, 3.f, p[t]), y = df_muladd(ds, 3.f, d[t]);
                r[(9 * t + k) * NE] = df_sum<kFull>(x, df_neg(y));
                r[(9 * (3 + t) + k) * NE] = df_sum<kFull>(x, y);
            }
        }
    }
    {
        // M = sum over the heights of the two layers' weights times A: with
        // p = A0 + A1 and d = sqrt(3)/2 (A0 - A1), bb p - d, bt p/2, tt p + d
        constexpr int kGroups = kSlots / Y::NJL;
        const int q = slot % Y::NJL;
        float2 *a0 = blk(Y::BA + 2 * q), *a1 = a0 + 9 * NE, *a2 = xblk(Y::XM + q);
#pragma unroll 1
        for (int k = slot / Y::NJL; k < 9; k += kGroups) {
            const float2 x = a0[k * NE], y = a1[k * NE];
            const float2 p = df_sum<kFull>(x, y);
            const float2 d = df_scale(DF_CONST(0.5 * kSqrt3), df_sum<kFull>(x, df_neg(y)));
            a0[k * NE] = df_sum<kFull>(p, df_neg(d));
            a1[k * NE] = df_pow2(0.5f, p);
            a2[k * NE] = df_sum<kFull>(p, d);
        }
    }
    {
        // W(i, k) = sum_t N_i N_k/4 B(t): S + 15 B(i), or S + 3 (B(i) + B(k))
        const int q = slot % 6;
        const int i = q < 3 ? q : (q < 5 ? 0 : 1), k2 = q < 3 ? q : (q == 3 ? 1 : 2);
        float2* o = xblk(Y::XW + q);
#pragma unroll 1
        for (int k = slot / 6; k < 9; k += 2) {
            float2 b[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                b[t] = blk(Y::BB + t)[k * NE];
                if (!VISC) b[t] = df_sum<kFull>(b[t], blk(Y::BB + 3 + t)[k * NE]);
            }
            const float2 s = df_sum<kFull>(df_sum<kFull>(b[0], b[1]), b[2]);
            const float2 bi = i == 0 ? b[0] : (i == 1 ? b[1] : b[2]), bk = k2 == 1 ? b[1] : b[2];
            o[k * NE] = i == k2 ? df_muladd(s, 15.f, bi) : df_muladd(s, 3.f, df_sum<kFull>(bi, bk));
        }
    }
    __syncthreads();
    if (!live) return;

    // ---- 6. the node pairs ------------------------------------------------------
    constexpr int kPairs = VISC ? 36 : 21;
#pragma unroll 1
    for (int pr = slot; pr < kPairs; pr += kSlots) {
        const int a = VISC ? pr / 6 : kPairA[pr];
        const int bq = VISC ? pr - 6 * (pr / 6) : kPairB[pr];
        const int i = a % 3, la = a / 3, k2 = bq % 3, lb = bq / 3;
        // node 0 has both in-plane gradients, negated; node j the j-th
        const int j0 = i == 2 ? 1 : 0, l0 = k2 == 2 ? 1 : 0, nj = i == 0 ? 2 : 1, nl = k2 == 0 ? 2 : 1;
        const float si = i == 0 ? -1.f : 1.f, sk = k2 == 0 ? -1.f : 1.f;
        const float ta = la ? 1.f : -1.f, tb = lb ? 1.f : -1.f;
        float H[9], L[9], E[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) H[k] = L[k] = E[k] = 0.f;
#pragma unroll 1
        for (int m = 0; m < 1 + nj + nl + nj * nl; ++m) {
            const float2* x;
            float s;
            bool tr = false;  // transposed (the symmetric case stores one triangle)
            if (m == 0) {
                x = xblk(Y::XW + sym_index(i, k2));
                s = ta * tb;
            } else if (m <= nj) {
                x = blk(Y::BR + 6 * (j0 + m - 1) + 3 * la + k2);
                s = si * tb;
            } else if (m <= nj + nl) {
                const int l = l0 + m - 1 - nj;
                x = blk(Y::BR + 6 * (VISC ? 2 + l : l) + 3 * lb + i);
                s = sk * ta;
                tr = !VISC;
            } else {
                const int q = m - 1 - nj - nl;
                const int j = j0 + q / nl, l = l0 + q % nl;
                const int jl = VISC ? 2 * j + l : j + l;
                x = la != lb ? blk(Y::BA + 2 * jl + 1) : (la ? xblk(Y::XM + jl) : blk(Y::BA + 2 * jl));
                s = si * sk;
                tr = !VISC && j > l;
            }
            const int s1 = tr ? 3 * NE : NE, s3 = tr ? NE : 3 * NE;
#pragma unroll
            for (int k = 0; k < 9; ++k)
                df_addmul<kFull>(H[k], L[k], E[k], s, x[(k / 3) * s3 + (k % 3) * s1]);
        }
        double acc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            if (kFull) L[k] = __fadd_rn(L[k], E[k]);
            df_norm(H[k], L[k]);
            acc[k] = df_join(H[k], L[k]);
        }
        const int na = __ldg(&A.conn[a * ne + e]);
        const int nb = __ldg(&A.conn[bq * ne + e]);
        if (!TF_IN(A.check, na, A.nn, CK_ELEM_NODE) || !TF_IN(A.check, nb, A.nn, CK_ELEM_NODE)) continue;
        bool fr[3], fc[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            fr[q] = A.fixed[3 * na + q] != 0;
            fc[q] = A.fixed[3 * nb + q] != 0;
        }
        const bool mirror = !VISC && (a != bq);
        if (MODE == kStore) {
            const size_t stride = (size_t)36 * ne;
            const size_t base = (size_t)(6 * a + bq) * ne + e;
            const size_t baseT = (size_t)(6 * bq + a) * ne + e;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double v = (fr[r] || fc[k]) ? 0.0 : acc[3 * r + k];
                    A.eblk[(3 * r + k) * stride + base] = v;
                    if (mirror) A.eblk[(3 * k + r) * stride + baseT] = v;
                }
        } else {
            const int off = __ldg(&A.slot[(6 * a + bq) * ne + e]);
            if (!TF_IN(A.check, off, A.nval - 8 * kSlice, CK_ELEM_SLOT)) continue;
            double* dst = A.val + off;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    if (!fr[r] && !fc[k]) atomicAdd(dst + kSlice * (3 * r + k), acc[3 * r + k]);
            if (mirror) {
                const int offT = __ldg(&A.slot[(6 * bq + a) * ne + e]);
                if (!TF_IN(A.check, offT, A.nval - 8 * kSlice, CK_ELEM_SLOT)) continue;
                double* dt = A.val + offT;
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (!fr[r] && !fc[k]) atomicAdd(dt + kSlice * (3 * k + r), acc[3 * r + k]);
            }
        }
    }
}

// ---- parity evaluation: separate elastic / viscous outputs ----------------

struct GpEval {
    double dn[18];
    double c1, c2;
    double sdn[18];
    double pv[9];
    double pdn[18];
    double svdn[18];
};

template <int NE>
__global__ void __launch_bounds__(NE * kGauss) k_element_eval(ElemArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GpEval* sh = reinterpret_cast<GpEval*>(smem_raw);
    const int tid = threadIdx.x;
    const int limit = A.e0 + A.count;
    {
        const int el = tid / kGauss;
        const int gp = tid - el * kGauss;
        const int e = A.e0 + blockIdx.x * NE + el;
        if (e < limit) {
            const bool visc = __ldg(&A.eta[e]) != 0.0;
            GaussPoint G;
            gauss_point(A, e, gp, visc, G);
            GpEval& S = sh[el * kGauss + gp];
            S.c1 = G.c1;
            S.c2 = G.c2;
#pragma unroll
            for (int a = 0; a < 6; ++a) {
                const double d0 = G.dn[3 * a], d1 = G.dn[3 * a + 1], d2 = G.dn[3 * a + 2];
                S.dn[3 * a] = d0;
                S.dn[3 * a + 1] = d1;
                S.dn[3 * a + 2] = d2;
                sym_apply(G.sg, d0, d1, d2, &S.sdn[3 * a]);
                if (visc) {
                    sym_apply(G.sv, d0, d1, d2, &S.svdn[3 * a]);
                    S.pdn[3 * a] = fma(G.pv[0], d0, fma(G.pv[3], d1, G.pv[6] * d2));
                    S.pdn[3 * a + 1] = fma(G.pv[1], d0, fma(G.pv[4], d1, G.pv[7] * d2));
                    S.pdn[3 * a + 2] = fma(G.pv[2], d0, fma(G.pv[5], d1, G.pv[8] * d2));
                } else {
                    S.svdn[3 * a] = S.svdn[3 * a + 1] = S.svdn[3 * a + 2] = 0.0;
                    S.pdn[3 * a] = S.pdn[3 * a + 1] = S.pdn[3 * a + 2] = 0.0;
                }
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) S.pv[k] = visc ? G.pv[k] : 0.0;
        }
    }
    __syncthreads();
    for (int task = tid; task < NE * 18; task += NE * kGauss) {
        const int el = task / 18;
        const int k = task - el * 18;
        const int e = A.e0 + blockIdx.x * NE + el;
        if (e >= limit) continue;
        double se = 0.0, sv = 0.0;
#pragma unroll
        for (int gp = 0; gp < kGauss; ++gp) {
            se -= sh[el * kGauss + gp].sdn[k];
            sv -= sh[el * kGauss + gp].svdn[k];
        }
        const int a = k / 3, d = k - 3 * (k / 3);
        const bool fx = A.fixed[3 * __ldg(&A.conn[a * A.ne + e]) + d] != 0;
        const size_t r = (size_t)(e - A.e0);
        if (A.fe) A.fe[18 * r + k] = fx ? 0.0 : se;
        if (A.fv) A.fv[18 * r + k] = fx ? 0.0 : sv;
    }
    for (int task = tid; task < NE * 36; task += NE * kGauss) {
        const int el = task / 36;
        const int pr = task - el * 36;
        const int e = A.e0 + blockIdx.x * NE + el;
        if (e >= limit) continue;
        const int a = pr / 6, bq = pr - 6 * (pr / 6);
        const bool visc = __ldg(&A.eta[e]) != 0.0;
        double ke[9], kv[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) ke[k] = kv[k] = 0.0;
#pragma unroll
        for (int gp = 0; gp < kGauss; ++gp) {
            const GpEval& S = sh[el * kGauss + gp];
            const double aa[3] = {S.dn[3 * a], S.dn[3 * a + 1], S.dn[3 * a + 2]};
            const double bb[3] = {S.dn[3 * bq], S.dn[3 * bq + 1], S.dn[3 * bq + 2]};
            const double s = fma(aa[0], bb[0], fma(aa[1], bb[1], aa[2] * bb[2]));
            const double t = fma(aa[0], S.sdn[3 * bq], fma(aa[1], S.sdn[3 * bq + 1], aa[2] * S.sdn[3 * bq + 2]));
            const double dg = fma(S.c2, s, t);
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    double v = fma(S.c1 * aa[i], bb[k], fma(S.c2 * aa[k], bb[i], ke[3 * i + k]));
                    if (i == k) v += dg;
                    ke[3 * i + k] = v;
                }
            if (visc) {
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        kv[3 * i + k] = fma(s, S.pv[3 * i + k],
                                            fma(bb[i], S.pdn[3 * a + k],
                                                fma(S.svdn[3 * a + i], bb[k], fma(-S.svdn[3 * bq + i], aa[k], kv[3 * i + k]))));
            }
        }
        // reference orientation: TriPointKe[3a+i][3b+k] = ke(i,k);
        // TriPointKv[3b+k][3a+i] = kv(i,k)  (ShapeBase.cpp:2968-2975)
        const size_t r = (size_t)(e - A.e0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (A.Ke) A.Ke[324 * r + (3 * a + i) * 18 + 3 * bq + k] = ke[3 * i + k];
                if (A.Kv) A.Kv[324 * r + (3 * bq + k) * 18 + 3 * a + i] = visc ? kv[3 * i + k] : 0.0;
            }
    }
}

// ---- adjoint contractions of one converged step --------------------------
//
// With lambda the adjoint of step n (A^T lambda = rhs) and
// Lam = sum_a lambda_a (x) dN_a per Gauss point:
//   dL/dlogE_e += sum_gp w dV <sigma, Lam>                 (forces are linear in E)
//   dL/dr_e    += n dt sum_{j=x,y} sum_gp w dV [<sigma,Lam> - (2 mu c_j.Lam c_j
//                  + lambda tr Lam) / J]                   (c_j = column j of Fe,
//                  d Fe / d ln Fg_jj = -Fe e_j e_j^T, ln Fg_jj = n r dt)
//   carry to step n-1 (velocity terms, d v / d u_{n-1} = -1/dt):
//     w_b += sum_gp 0.5 eta w dV / dt (Lam + Lam^T) dN_b
// Element-relative outputs: gr[e], ge[e] (no atomics), carry via atomics.
struct AdjArgs {
    const double* __restrict__ lamv;  // adjoint vector lambda [3N]
    double* __restrict__ carry;       // [3N] accumulates the carry to step n-1
    double* __restrict__ gr;          // [E] growth-rate gradient (accumulated)
    double* __restrict__ ge;          // [E] log E gradient (accumulated)
    double ndt;                       // n * dt
    double idt;
};

template <int NE>
__global__ void __launch_bounds__(NE * kGauss) k_adjoint_element(ElemArgs A, AdjArgs D) {
    __shared__ double s_gr[NE][kGauss], s_ge[NE][kGauss];
    __shared__ double s_w[NE][kGauss][18];
    const int el = threadIdx.x / kGauss, gp = threadIdx.x - (threadIdx.x / kGauss) * kGauss;
    const int e = blockIdx.x * NE + el;
    double tr = 0.0, te = 0.0;
    double w18[18];
#pragma unroll
    for (int k = 0; k < 18; ++k) w18[k] = 0.0;
    if (e < A.ne) {
        const bool visc = __ldg(&A.eta[e]) != 0.0;
        GaussPoint G;
        gauss_point(A, e, gp, visc, G);
        double Lm[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) Lm[k] = 0.0;
#pragma unroll
        for (int a = 0; a < 6; ++a) {
            const int nd = __ldg(&A.conn[a * A.ne + e]);
            const double l0 = D.lamv[3 * nd], l1 = D.lamv[3 * nd + 1], l2 = D.lamv[3 * nd + 2];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                Lm[j] = fma(l0, G.dn[3 * a + j], Lm[j]);
                Lm[3 + j] = fma(l1, G.dn[3 * a + j], Lm[3 + j]);
                Lm[6 + j] = fma(l2, G.dn[3 * a + j], Lm[6 + j]);
            }
        }
        // <sigma', Lam> with sigma' symmetric (00 11 22 01 02 12)
        const double sl = fma(G.sg[0], Lm[0], fma(G.sg[1], Lm[4], fma(G.sg[2], Lm[8],
                          fma(G.sg[3], Lm[1] + Lm[3], fma(G.sg[4], Lm[2] + Lm[6], G.sg[5] * (Lm[5] + Lm[7]))))));
        te = sl;
        // Fe columns, 1/J and the material, recomputed as in gauss_point
        const double lam = __ldg(&A.lam[e]), mu = __ldg(&A.mu[e]);
        const double trL = Lm[0] + Lm[4] + Lm[8];
        // w dV (2 mu c.Lam c + lambda tr Lam) / J = 2 mu sc c.Lam c + c1 tr Lam
        const double sc = G.sc;
        (void)lam;
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double c0 = G.fe[j], c1v = G.fe[3 + j], c2v = G.fe[6 + j];
            const double Lc0 = fma(Lm[0], c0, fma(Lm[1], c1v, Lm[2] * c2v));
            const double Lc1 = fma(Lm[3], c0, fma(Lm[4], c1v, Lm[5] * c2v));
            const double Lc2 = fma(Lm[6], c0, fma(Lm[7], c1v, Lm[8] * c2v));
            const double cLc = fma(c0, Lc0, fma(c1v, Lc1, c2v * Lc2));
            t += sl - fma(2.0 * mu * sc, cLc, G.c1 * trL);
        }
        tr = D.ndt * t;
        if (visc) {
            const double hw = 0.5 * __ldg(&A.eta[e]) * G.wdv * D.idt;
            double S[9];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int k = 0; k < 3; ++k) S[3 * i + k] = hw * (Lm[3 * i + k] + Lm[3 * k + i]);
#pragma unroll
            for (int b = 0; b < 6; ++b) {
                const double d0 = G.dn[3 * b], d1 = G.dn[3 * b + 1], d2 = G.dn[3 * b + 2];
                w18[3 * b] = fma(S[0], d0, fma(S[1], d1, S[2] * d2));
                w18[3 * b + 1] = fma(S[3], d0, fma(S[4], d1, S[5] * d2));
                w18[3 * b + 2] = fma(S[6], d0, fma(S[7], d1, S[8] * d2));
            }
        }
    }
    s_gr[el][gp] = tr;
    s_ge[el][gp] = te;
#pragma unroll
    for (int k = 0; k < 18; ++k) s_w[el][gp][k] = w18[k];
    __syncthreads();
    if (e < A.ne && gp == 0) {
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int q = 0; q < kGauss; ++q) {
            a += s_gr[el][q];
            b += s_ge[el][q];
        }
        D.gr[e] += a;
        D.ge[e] += b;
    }
    for (int task = threadIdx.x; task < NE * 18; task += NE * kGauss) {
        const int l = task / 18, k = task - 18 * (task / 18);
        const int ee = blockIdx.x * NE + l;
        if (ee >= A.ne || __ldg(&A.eta[ee]) == 0.0) continue;
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < kGauss; ++q) v += s_w[l][q][k];
        const int nd = __ldg(&A.conn[(k / 3) * A.ne + ee]);
        atomicAdd(&D.carry[3 * nd + (k % 3)], v);
    }
}

ElemArgs make_args(tf_handle* h) {
    const Device& d = h->d;
    ElemArgs A{};
    A.ne = d.ne;
    A.conn = d.conn;
    A.metric = d.metric;
    A.gx = d.gx;
    A.wdet = d.wdet;
    A.invFg = d.invFg;
    A.lam = d.lam;
    A.mu = d.mu;
    A.eta = d.eta;
    A.fixed = d.fixed;
    A.slot = d.slot;
    A.uk = d.uk;
    A.vel = d.vel;
    A.idt = 1.0 / h->dt;
    A.val = d.val;
    A.g = d.g;
    A.eblk = d.eblk;
    A.ef = d.ef;
    A.elem_seg = d.elem_seg;
    A.seg_active = d.seg_active;
    A.masked = d.nseg > 1 ? 1 : 0;
    A.nn = d.nn;
    A.nval = d.nval;
    A.check = d.check;
    return A;
}

template <int NE, int MODE, bool VISC>
tf_status launch_fast(tf_handle* h, const ElemArgs& A) {
    constexpr size_t smem = elem_smem<NE, VISC>();
    constexpr unsigned bit = 1u << (2 * (NE / 8) + (VISC ? 1 : 0));  // the assembly mode is the handle's
    if (!(h->elem_smem & bit)) {
        TF_CUDA(cudaFuncSetAttribute(k_element<NE, MODE, VISC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        h->elem_smem |= bit;
    }
    k_element<NE, MODE, VISC><<<cdiv(A.ne, NE), NE * kSlots, smem, h->stream>>>(A);
    TF_LAUNCH_CHECK(h);
    return TF_OK;
}

template <int NE>
tf_status launch_ne(tf_handle* h, const ElemArgs& A) {
    const bool visc = h->d.any_visc;
    if (h->opt.deterministic) return visc ? launch_fast<NE, kStore, true>(h, A) : launch_fast<NE, kStore, false>(h, A);
    return visc ? launch_fast<NE, kAtomic, true>(h, A) : launch_fast<NE, kAtomic, false>(h, A);
}

tf_status launch_with(tf_handle* h, const ElemArgs& A, int ne_per_cta) {
    switch (ne_per_cta) {
        case 8: return launch_ne<8>(h, A);
        case 32: return launch_ne<32>(h, A);
        default: return launch_ne<16>(h, A);
    }
}

}  // namespace

struct ShapeDerivatives {
    double dN[6][3][6];
};
// dN_X = InvdXde^T dN of every prism and Gauss point (Prism.cpp:705-728)
__global__ void k_shape_gradients(int ne, ShapeDerivatives S, const double* __restrict__ ginv, double* __restrict__ gx) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;  // 6 e + gp
    if (q >= 6 * ne) return;
    const int e = q / 6, gp = q - 6 * e;
    double inv[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) inv[k] = ginv[((size_t)k * 6 + gp) * ne + e];
#pragma unroll
    for (int a = 0; a < 6; ++a)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            gx[(size_t)(3 * a + k) * (6 * (size_t)ne) + q] =
                inv[k] * S.dN[gp][0][a] + inv[3 + k] * S.dN[gp][1][a] + inv[6 + k] * S.dN[gp][2][a];
}

tf_status launch_shape_gradients(tf_handle* h, const double* dN) {
    ShapeDerivatives S;
    std::memcpy(S.dN, dN, sizeof(S.dN));
    k_shape_gradients<<<cdiv(6 * (int64_t)h->d.ne, 256), 256, 0, h->stream>>>(h->d.ne, S, h->d.ginv, h->d.gx);
    TF_LAUNCH_CHECK(h);
    return TF_OK;
}

// What the element kernel needs of a Gauss point's reference and growth: M =
// dxi/dX Fg^-1 (Fe = X^T M for X = dx/dxi), det M (J = det X det M) and 1 / (6 det M)
// = w dV / J.  They change with the growth, once per time step, and take a matrix
// product, a determinant and a division out of every Gauss point of every assembly:
// a sixth of its FP64 instructions (320,000 prisms 1.37 -> 1.26 ms without
// viscosity, 1.89 -> 1.81 with; 0.15 ms per change of the growth).  C = M M^T in place of M would save
// three loads, but X^T C X loses the digits of a skewed prism's M twice.
__global__ void k_metric(int ne, const double* __restrict__ ginv, const double* __restrict__ invFg,
                         double* __restrict__ metric) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;  // gp ne + e
    if (q >= 6 * ne) return;
    const int e = q % ne;
    const size_t st6 = (size_t)6 * ne;
    double G[9], F[9], M[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        G[k] = ginv[k * st6 + q];
        F[k] = invFg[(size_t)k * ne + e];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            M[3 * j + k] = fma(G[3 * j], F[k], fma(G[3 * j + 1], F[3 + k], G[3 * j + 2] * F[6 + k]));
            metric[(3 * j + k) * st6 + q] = M[3 * j + k];
        }
    const double det = fma(M[0], fma(M[4], M[8], -(M[5] * M[7])),
                           fma(-M[1], fma(M[3], M[8], -(M[5] * M[6])), M[2] * fma(M[3], M[7], -(M[4] * M[6]))));
    metric[9 * st6 + q] = det;
    metric[10 * st6 + q] = 1.0 / (6.0 * det);
}

tf_status launch_metric(tf_handle* h) {
    const Device& d = h->d;
    if (d.ne <= 0) return TF_OK;
    k_metric<<<cdiv(6 * (int64_t)d.ne, 256), 256, 0, h->stream>>>(d.ne, d.ginv, d.invFg, d.metric);
    TF_LAUNCH_CHECK(h);
    return TF_OK;
}

tf_status launch_element(tf_handle* h) {
    const ElemArgs A = make_args(h);
    if (A.ne <= 0) return TF_OK;
    return launch_with(h, A, h->elem_cta);
}

// Picks the prisms-per-CTA tile (8, 16 or 32 prisms) by
// timing each candidate on the handle's own mesh; run once per handle before
// the first assembly.  Results do not depend on the choice.
tf_status autotune_element(tf_handle* h) {
    if (h->tuned || h->d.ne <= 0) return TF_OK;
    h->tuned = true;
    if (h->opt.autotune_off) return TF_OK;
    const ElemArgs A = make_args(h);
    const int cand[3] = {8, 16, 32};
    float best = 1e30f;
    for (int c : cand) {
        if (launch_with(h, A, c) != TF_OK) continue;  // warm-up (and smem attribute)
        TF_CUDA(cudaEventRecord(h->ev[4], h->stream));
        for (int r = 0; r < 2; ++r) {
            const tf_status s = launch_with(h, A, c);
            if (s != TF_OK) return s;
        }
        TF_CUDA(cudaEventRecord(h->ev[5], h->stream));
        TF_CUDA(cudaEventSynchronize(h->ev[5]));
        float ms = 0.f;
        TF_CUDA(cudaEventElapsedTime(&ms, h->ev[4], h->ev[5]));
        if (ms < best) {
            best = ms;
            h->elem_cta = c;
        }
    }
    return TF_OK;
}

tf_status launch_adjoint_element(tf_handle* h, const double* lamv, double* carry, double* gr, double* ge,
                                 double ndt) {
    ElemArgs A = make_args(h);
    if (A.ne <= 0) return TF_OK;
    AdjArgs D{lamv, carry, gr, ge, ndt, 1.0 / h->dt};
    constexpr int NE = 16;
    k_adjoint_element<NE><<<cdiv(A.ne, NE), NE * kGauss, 0, h->stream>>>(A, D);
    TF_LAUNCH_CHECK(h);
    return TF_OK;
}

tf_status launch_element_eval(tf_handle* h, int e0, int count, double* Ke, double* Kv, double* fe, double* fv) {
    ElemArgs A = make_args(h);
    A.e0 = e0;
    A.count = count;
    A.Ke = Ke;
    A.Kv = Kv;
    A.fe = fe;
    A.fv = fv;
    if (count <= 0) return TF_OK;
    constexpr int NE = 8;
    const size_t smem = sizeof(GpEval) * NE * kGauss;
    TF_CUDA(cudaFuncSetAttribute(k_element_eval<NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_element_eval<NE><<<cdiv(count, NE), NE * kGauss, smem, h->stream>>>(A);
    TF_LAUNCH_CHECK(h);
    return TF_OK;
}

}  // namespace tf
