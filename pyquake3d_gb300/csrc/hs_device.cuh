// Half-space terms of the triangular-dislocation Green's function: the image
// dislocation and the free-surface correction (FSC), per (receiver, source)
// pair, for unit strike and unit dip slip (assembly) or a general Burgers
// vector (point entry points).
//
// Reference behaviour reproduced (file:line in PyQuake3D):
//   total = main + FSC + image          src/TDstressFS_C.cpp:1934-2033 (TDstressHS)
//     image = full-space solution of the triangle mirrored in z = 0; when all
//     three vertices lie on the surface its xz and yz components change sign
//   FSC = sum over the sides           src/TDstressFS_C.cpp:1785-1931 (TDstress_HarFunc)
//   one side                           src/TDstressFS_C.cpp:1489-1782 (AngSetupFSC_S)
//     beta = angle of -side with e_Z; no contribution within 1e-4 of 0 or pi;
//     frame ey1 = horizontal side direction, ey3 = -e_Z, ey2 = ey3 x ey1;
//     configuration I (beta * yA_1 >= 0): evaluate at (-y1, -y2, y3) with
//     pi - beta and (-b1, -b2, b3), then flip the 13 and 23 strain components;
//     strain = (B end) - (A end), rotated to EFCS
//   harmonic displacement of one angular dislocation: the published formulas
//   (Nikkhoo & Walter 2015, after Comninou & Dundurs 1975), as stated in
//   src/DH_greenfunction.py:313-400 (AngDisDispFSC); an image point within
//   1e-12 m of the receiver contributes zero (src/TDstressFS_C.cpp:651-654).
//
// Method (stated): the reference differentiates the harmonic displacement by
// hand (AngDisStrainFSC, src/TDstressFS_C.cpp:613-1487, ~870 lines).  Here the
// displacement is evaluated once in forward mode, as a function of six
// variables: y1, y2, y3 where they appear explicitly, and rb, P = rb + y3b and
// Q = rb + z3b, on which every reciprocal depends.  Each intermediate carries
// only the partial derivatives that it has (a reciprocal one, a product of two
// the union), and the gradient in y comes from the chain rule once per result:
// the nine unit-Burgers displacements cost about half the operations of three
// dense partials carried through every product.  The displacement is linear in
// the Burgers vector, so an end point yields the strains of the three unit
// vectors, which are combined for every slip direction.  Divisions are replaced
// by a few reciprocals (1/rb, 1/P, 1/Q, and per side 1/sin beta).
#pragma once

#include "gf_device.cuh"

namespace pq3d {
namespace gf {

// ---------------------------------------------------------------------------
// forward mode with a set of partials known at compile time: value v and the
// partials d[i] of the variables i in M (the others are zero and take no
// operations)

enum SdVar { V_Y1 = 1, V_Y2 = 2, V_Y3 = 4, V_R = 8, V_P = 16, V_Q = 32 };

template <int M>
struct Sd {
    double v, d[6];
};

#define PQ3D_SD_EACH(body)                                                                  \
    { constexpr int i = 0, bit = 1; body } { constexpr int i = 1, bit = 2; body }            \
    { constexpr int i = 2, bit = 4; body } { constexpr int i = 3, bit = 8; body }            \
    { constexpr int i = 4, bit = 16; body } { constexpr int i = 5, bit = 32; body }

template <int A, int B>
__host__ __device__ __forceinline__ Sd<A | B> operator*(const Sd<A> &a, const Sd<B> &b)
{
    Sd<A | B> r;
    r.v = a.v * b.v;
    PQ3D_SD_EACH(if constexpr ((A & bit) && (B & bit)) r.d[i] = a.v * b.d[i] + b.v * a.d[i];
                 else if constexpr (A & bit) r.d[i] = b.v * a.d[i];
                 else if constexpr (B & bit) r.d[i] = a.v * b.d[i];)
    return r;
}
template <int A, int B>
__host__ __device__ __forceinline__ Sd<A | B> operator+(const Sd<A> &a, const Sd<B> &b)
{
    Sd<A | B> r;
    r.v = a.v + b.v;
    PQ3D_SD_EACH(if constexpr ((A & bit) && (B & bit)) r.d[i] = a.d[i] + b.d[i];
                 else if constexpr (A & bit) r.d[i] = a.d[i];
                 else if constexpr (B & bit) r.d[i] = b.d[i];)
    return r;
}
template <int A>
__host__ __device__ __forceinline__ Sd<A> operator-(const Sd<A> &a)
{
    Sd<A> r;
    r.v = -a.v;
    PQ3D_SD_EACH(if constexpr (A & bit) r.d[i] = -a.d[i];)
    return r;
}
template <int A, int B>
__host__ __device__ __forceinline__ Sd<A | B> operator-(const Sd<A> &a, const Sd<B> &b)
{
    Sd<A | B> r;
    r.v = a.v - b.v;
    PQ3D_SD_EACH(if constexpr ((A & bit) && (B & bit)) r.d[i] = a.d[i] - b.d[i];
                 else if constexpr (A & bit) r.d[i] = a.d[i];
                 else if constexpr (B & bit) r.d[i] = -b.d[i];)
    return r;
}
template <int A>
__host__ __device__ __forceinline__ Sd<A> operator*(double k, const Sd<A> &a)
{
    Sd<A> r;
    r.v = k * a.v;
    PQ3D_SD_EACH(if constexpr (A & bit) r.d[i] = k * a.d[i];)
    return r;
}
template <int A>
__host__ __device__ __forceinline__ Sd<A> operator+(double k, const Sd<A> &a)   // the partials stay
{
    Sd<A> r = a;
    r.v = k + a.v;
    return r;
}
template <int A>
__host__ __device__ __forceinline__ Sd<A> operator-(double k, const Sd<A> &a)
{
    Sd<A> r = -a;
    r.v = k - a.v;
    return r;
}

// ---------------------------------------------------------------------------
// per-source side table (three sides: P1->P2, P2->P3, P3->P1)

enum FscField {
    S_VALID,                       // 1: the side contributes
    S_PAX, S_PAY, S_PAZ, S_PBZ,    // start point, end-point depth
    S_C1, S_S1,                    // ey1 = (c1, s1, 0), ey2 = (s1, -c1, 0), ey3 = (0, 0, -1)
    S_YAB0, S_YAB1, S_YAB2,        // side vector in the side frame
    S_SIN2, S_COS2, S_COT2, S_CTH2,   // configuration II: sin, cos, cot of beta, cot(beta / 2)
    S_SIN1, S_COS1, S_COT1, S_CTH1,   // configuration I: the same for pi - beta
    S_BN0, S_BN1, S_BN2,           // unit tensile (normal) Burgers vector in the side frame
    S_BS0, S_BS1, S_BS2,           // unit strike
    S_BD0, S_BD1, S_BD2,           // unit dip
    S_ISIN,                        // 1 / sin beta (both configurations)
    S_COUNT
};
constexpr int kFscSurface = 3 * S_COUNT;   // 1 when all three vertices have z == 0
constexpr int kFscStride = 88;             // fields per source (>= 3 * S_COUNT + 1)
static_assert(kFscStride >= 3 * S_COUNT + 1, "side table");
constexpr int kImgStride = kSrcStride;     // image-source record: setup_source of the mirrored triangle

// Fields of side sd (P1 P2, P2 P3, P3 P1) into f[i * fstride].
__host__ __device__ inline void setup_fsc_side(const double P1[3], const double P2[3], const double P3[3], int sd,
                                               double *f, int fstride)
{
    // triangle frame (normal, strike, dip) as TDstress_HarFunc builds it
    double n[3] = {(P2[1] - P1[1]) * (P3[2] - P1[2]) - (P2[2] - P1[2]) * (P3[1] - P1[1]),
                   (P2[2] - P1[2]) * (P3[0] - P1[0]) - (P2[0] - P1[0]) * (P3[2] - P1[2]),
                   (P2[0] - P1[0]) * (P3[1] - P1[1]) - (P2[1] - P1[1]) * (P3[0] - P1[0])};
    const double nl = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (nl != 0.0) { n[0] /= nl; n[1] /= nl; n[2] /= nl; }
    double st[3] = {-n[1], n[0], 0.0};
    const double sl = sqrt(st[0] * st[0] + st[1] * st[1]);
    if (sl == 0.0) { st[0] = 0.0; st[1] = n[2]; }
    else { st[0] /= sl; st[1] /= sl; }
    const double dp[3] = {n[1] * st[2] - n[2] * st[1], n[2] * st[0] - n[0] * st[2], n[0] * st[1] - n[1] * st[0]};
    const double *PA = sd == 0 ? P1 : (sd == 1 ? P2 : P3), *PB = sd == 0 ? P2 : (sd == 1 ? P3 : P1);
    double v[S_COUNT];
    for (int i = 0; i < S_COUNT; ++i) v[i] = 0.0;
    const double sv[3] = {PB[0] - PA[0], PB[1] - PA[1], PB[2] - PA[2]};
    const double len = sqrt(sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2]);
    const double beta = acos(-sv[2] / len);
    if (!(fabs(beta) < 1e-4 || fabs(kPi - beta) < 1e-4)) {
        const double hl = sqrt(sv[0] * sv[0] + sv[1] * sv[1]);
        const double c1 = sv[0] / hl, s1 = sv[1] / hl;
        // ey1 = (c1, s1, 0), ey2 = (s1, -c1, 0), ey3 = (0, 0, -1)
        v[S_VALID] = 1.0;
        v[S_PAX] = PA[0]; v[S_PAY] = PA[1]; v[S_PAZ] = PA[2]; v[S_PBZ] = PB[2];
        v[S_C1] = c1; v[S_S1] = s1;
        v[S_YAB0] = sv[0] * c1 + sv[1] * s1;
        v[S_YAB1] = sv[0] * s1 - sv[1] * c1;
        v[S_YAB2] = -sv[2];
        // everything from sin and cos beta (tan(beta/2) without cancellation)
        const double sb = sin(beta), cb = cos(beta), th = cb >= 0.0 ? sb / (1.0 + cb) : (1.0 - cb) / sb;
        v[S_SIN2] = sb; v[S_COS2] = cb; v[S_COT2] = cb / sb; v[S_CTH2] = 1.0 / th;
        v[S_SIN1] = sb; v[S_COS1] = -cb; v[S_COT1] = -cb / sb; v[S_CTH1] = th;
        v[S_ISIN] = 1.0 / sb;
        const double *B[3] = {n, st, dp};
        for (int q = 0; q < 3; ++q) {
            v[S_BN0 + 3 * q] = B[q][0] * c1 + B[q][1] * s1;
            v[S_BN0 + 3 * q + 1] = B[q][0] * s1 - B[q][1] * c1;
            v[S_BN0 + 3 * q + 2] = -B[q][2];
        }
    }
    for (int i = 0; i < S_COUNT; ++i) f[i * fstride] = v[i];
}

__host__ __device__ inline double fsc_surface(const double P1[3], const double P2[3], const double P3[3])
{
    return (P1[2] == 0.0 && P2[2] == 0.0 && P3[2] == 0.0) ? 1.0 : 0.0;
}

__host__ __device__ inline void setup_fsc(const double P1[3], const double P2[3], const double P3[3], double *f,
                                          int fstride)
{
    for (int sd = 0; sd < 3; ++sd) setup_fsc_side(P1, P2, P3, sd, f + sd * S_COUNT * fstride, fstride);
    f[kFscSurface * fstride] = fsc_surface(P1, P2, P3);
}

// ---------------------------------------------------------------------------
// harmonic displacement of one angular dislocation and its strains

struct FscTrig {
    double s, c, ct, cth, is, k;   // sin, cos, cot beta, cot(beta / 2), 1 / sin beta, 1 - cos beta
};

// Gradient in y of a result F of the six variables.
struct FscChain {
    double y1r, y2r, y3r, s, c;   // y / rb; sin, cos beta
    template <int M>
    __device__ __forceinline__ void operator()(const Sd<M> &F, double g[3]) const
    {
        double t = 0.0;
        if constexpr (M & V_R) t = F.d[3];
        if constexpr (M & V_P) t = t + F.d[4];
        if constexpr (M & V_Q) t = t + F.d[5];
        g[0] = t * y1r;
        g[1] = t * y2r;
        g[2] = t * y3r;
        if constexpr (M & V_Y1) g[0] += F.d[0];
        if constexpr (M & V_Y2) g[1] += F.d[1];
        if constexpr (M & V_Y3) g[2] += F.d[2];
        if constexpr (M & V_P) g[2] += F.d[4];
        if constexpr (M & V_Q) {
            g[0] -= s * F.d[5];
            g[2] += c * F.d[5];
        }
    }
};

// Strains (11, 22, 33, 2 x 12, 2 x 13, 2 x 23) of the harmonic displacement at
// (y1, y2, y3) for the three unit Burgers vectors, without the common factor
// 1 / (4 pi (1 - nu)); a = depth of the vertex.  The displacement formulas are
// the published ones with 1/(rb cos beta) cot beta = 1/(rb sin beta), factors
// y2 taken out, and the terms that several components share formed once.
__device__ __forceinline__ void fsc_unit_strain(double y1v, double y2v, double y3v, const FscTrig &T, double nu,
                                                double a, double E[3][6])
{
    const double s = T.s, c = T.c, ct = T.ct, is = T.is;
    const double n1 = 1.0 - 2.0 * nu, n2 = 1.0 - nu, ct2 = ct * ct, cct = c * ct;
    const double y3bv = y3v + 2.0 * a, hv = y3v + a;
    double rv, irv;
    root_and_reciprocal(y1v * y1v + y2v * y2v + y3bv * y3bv, rv, irv);
    const double z3bv = y3bv * c - y1v * s;
    const double iPv = reciprocal(rv + y3bv), iQv = reciprocal(rv + z3bv);
    const FscChain grad{y1v * irv, y2v * irv, y3bv * irv, s, c};
    // the variables and what depends on one of them
    const Sd<V_Y1> y1{y1v, {1.0}};
    const Sd<V_Y3> y3b{y3bv, {0.0, 0.0, 1.0}}, h{hv, {0.0, 0.0, 1.0}};
    const Sd<V_R> ir{irv, {0.0, 0.0, 0.0, -irv * irv}};
    const Sd<V_P> iP{iPv, {0.0, 0.0, 0.0, 0.0, -iPv * iPv}};
    const Sd<V_Q> iQ{iQv, {0.0, 0.0, 0.0, 0.0, 0.0, -iQv * iQv}};
    const Sd<V_Y1 | V_Y3> z1b{y1v * c + y3bv * s, {c, 0.0, s}};
    const Sd<V_Y3 | V_R> W{rv * c + y3bv, {0.0, 0.0, 1.0, c}};
    const Sd<V_Y1 | V_R> rsy{rv * s - y1v, {-1.0, 0.0, 0.0, s}};
    const double y2sv = y2v * y2v;
    const Sd<V_Y2> y2s{y2sv, {0.0, y2v + y2v}};
    const Sd<V_R> ar = a * ir, car = c + ar;
    const Sd<V_R> airb2 = ar * ir;
    const Sd<V_Y3 | V_R> ay3 = y3b * airb2, hr = h * ir, hA = hr * airb2;
    const auto hP = hr * iP;
    const auto hQ = hr * iQ;
    const auto HP = h * iP;
    const auto HQ = h * iQ;
    const auto y1P = y1 * iP;
    const auto WQ = W * iQ;
    const auto K1 = ay3 + ar * WQ;           // a y3b/rb^2 + a W/(rb Q)
    const auto V1 = c * WQ + K1;             // W/Q (c + a/rb) + a y3b/rb^2
    const auto hQV = hQ * V1;
    const auto carQ = car * iQ;
    const auto iPt = iP * (2.0 * nu + ar);
    const auto iPn = iP * (nu + ar);
    const auto iP1 = iP * (1.0 + ar);
    const auto E1 = ct + is * ar;            // cot beta + a/(rb sin beta)
    const auto y1A = y1 * airb2;
    const auto y1t = y1 * iPt;
    const auto z1car = z1b * carQ;
    const auto y1hA = y1 * hA;
    const auto z1K = z1b * K1;
    // Burgers function 2 atan(-y2/(y1 - P cot(beta/2))): its gradient
    double fib[3];
    {
        const double w = y1v - (rv + y3bv) * T.cth, id = reciprocal(y2sv + w * w), q = 2.0 * y2v * id;
        const double qp = -T.cth * q;        // d/dP
        fib[0] = qp * grad.y1r + q;
        fib[1] = qp * grad.y2r - 2.0 * w * id;
        fib[2] = qp * grad.y3r + qp;
    }
    // ln P - cos beta ln Q, which comes times cot^2 beta: its gradient with the
    // cancellation of a nearly vertical side (Q -> P) taken out, Q ∂P - c P ∂Q =
    // (k r - s y1) ∂P + c P (s, 0, k) with k = 1 - cos beta (its rounding, and
    // that of the reciprocals, would otherwise come times cot^2 beta too)
    double gD[3];
    {
        const double kr = T.k - s * grad.y1r;
        gD[0] = (kr * y1v + (c * s) * (rv + y3bv)) * (iPv * iQv);
        gD[1] = (kr * y2v) * (iPv * iQv);
        gD[2] = (kr + c * T.k) * iQv;
    }
    double g[3][3] = {};   // gradients of the three displacement components
    auto add_D = [&](double f, double o[3]) {
        o[0] += f * gD[0];
        o[1] += f * gD[1];
        o[2] += f * gD[2];
    };
    auto strain = [&](int k) {
        E[k][0] = g[0][0];
        E[k][1] = g[1][1];
        E[k][2] = g[2][2];
        E[k][3] = g[0][1] + g[1][0];
        E[k][4] = g[0][2] + g[2][0];
        E[k][5] = g[1][2] + g[2][1];
    };
    // y2 times G (no explicit y2 in G), plus f times the Burgers function
    auto odd = [&](const auto &G, double f, double o[3]) {
        grad(G, o);
        o[0] = y2v * o[0] + f * fib[0];
        o[1] = y2v * o[1] + (G.v + f * fib[1]);
        o[2] = y2v * o[2] + f * fib[2];
    };
    // terms of P that the 11 and 22 parts share with opposite signs
    const auto nct = n1 * ct - ct * ar;      // (1 - 2 nu - a/rb) cot beta
    const auto A = n1 * (iP * nct - y1P * iPn) + hP * ((y1t + y1A) - Sd<0>{n1 * ct, {}}) + ct * hA;
    const auto L = y1 * nct;
    const auto iPQ = iPt + airb2;
    // b1
    odd(A + ((n1 * cct) * carQ + hQ * (cct * (WQ * (n1 * c - ar)) + (2.0 * n2 * c * c) * (rsy * iQ) - cct * ay3)),
        -2.0 * n2 * n1 * ct2, g[0]);
    {
        const Sd<V_P | V_Q> ln{0.0, {0.0, 0.0, 0.0, 0.0, -(n1 * nu) * iPv, -(n1 * n1 * c) * iQv}};
        const auto F = ln - n1 * (iP * (L + nu * y3b - Sd<0>{a, {}} + y2s * iPn)) - (n1 * ct) * z1car - ct * y1hA +
                       HP * Sd<0>{-2.0 * nu, {}} + hP * (((n1 * ct) * y1 - Sd<0>{a, {}}) + y2s * iPQ) + (c * c) * HQ +
                       hQ * (ct * (z1K - n1 * z1b) - Sd<0>{a * c, {}} - (c * c) * (y2s * iQ));
        grad(F, g[1]);
        add_D(2.0 * n2 * n1 * ct2, g[1]);
    }
    odd((2.0 * n2) * (iPt - c * carQ) + (2.0 * nu) * hP + hA + c * (n1 * hQ - hQV), 2.0 * n2 * n1 * ct, g[2]);
    strain(0);
    // b2
    {
        const auto y1s = y1 * y1;
        const Sd<V_P | V_Q> ln{0.0, {0.0, 0.0, 0.0, 0.0, (n1 * nu) * iPv, -(n1 * c) * iQv}};
        const auto F = ln + n1 * (iP * (nu * y3b - L - Sd<0>{a, {}} + y1s * iPn)) -
                       n1 * (iQ * (cct * z1b - is * (rsy * ar))) - ct * y1hA + (2.0 * nu) * HP +
                       hP * (((n1 * ct) * y1 + Sd<0>{a, {}}) - y1s * iPQ) - (c * c) * HQ +
                       hQ * (is * (y1 * ay3) + rsy * ((2.0 * n2 * cct) - WQ * E1));
        grad(F, g[0]);
        add_D(2.0 * n2 * n1 * ct2, g[0]);
    }
    odd(hQ * ((WQ * E1 + is * ay3) - Sd<0>{2.0 * n2 * cct, {}}) - n1 * (iQ * E1) - A, 2.0 * n2 * n1 * ct2, g[1]);
    {
        const auto F = (2.0 * n2) * (z1car - y1t) + hr * (n1 * ct - ((2.0 * nu) * y1P + y1A)) - (c * s) * HQ -
                       hQ * (ct * (W * (2.0 * n2 * c - WQ)) + Sd<0>{a * s, {}} - z1K);
        grad(F, g[2]);
        add_D(-2.0 * n2 * n1 * ct, g[2]);
    }
    strain(1);
    // b3
    odd(n1 * (iP1 - c * carQ) - hA - hP + c * hQV, 0.0, g[0]);
    {
        const Sd<V_Q> ln{0.0, {0.0, 0.0, 0.0, 0.0, 0.0, -n1 * s * iQv}};
        const auto F = ln + n1 * (z1car - y1 * iP1) + y1hA + y1 * hP - (s * c) * HQ +
                       hQ * ((c * s) * (y2s * iQ) - z1b - z1K + Sd<0>{a * s, {}});
        grad(F, g[1]);
    }
    odd(s * (2.0 * n2 * carQ + hQ + hQV), 2.0 * n2, g[2]);
    strain(2);
}

// The strains of one end point (side frame, unit Burgers vectors), added with
// weight sgn.  Configuration I evaluates at (-y1, -y2, y3) with (-b1, -b2, b3);
// fsc_side maps the signs back.  A called function, not inlined: the
// intermediates of one end point then take the register file alone.
static __device__ PQ3D_NOINLINE void fsc_endpoint(const double y[3], bool confI, const FscTrig &T, double nu, double a,
                                           double sgn, double E[3][6])
{
    const double yb3 = y[2] + 2.0 * a;
    if (y[0] * y[0] + y[1] * y[1] + yb3 * yb3 < 1e-24) return;
    double e[3][6];
    fsc_unit_strain(confI ? -y[0] : y[0], confI ? -y[1] : y[1], y[2], T, nu, a, e);
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 6; ++i) E[k][i] += sgn * e[k][i];
}

// The strains (11, 22, 33, 2 x 12, 2 x 13, 2 x 23, side frame, times
// 4 pi (1 - nu)) of one side for the three unit Burgers vectors of its frame;
// false for a side that contributes none.
template <class Fs>
__device__ __forceinline__ bool fsc_side_strains(const Fs &G, double X, double Y, double Z, double nu, double E[3][6])
{
    if (G(S_VALID) == 0.0) return false;
    const double c1 = G(S_C1), s1 = G(S_S1);
    const double dx = X - G(S_PAX), dy = Y - G(S_PAY), dz = Z - G(S_PAZ);
    const double yA[3] = {dx * c1 + dy * s1, dx * s1 - dy * c1, -dz};
    const double yB[3] = {yA[0] - G(S_YAB0), yA[1] - G(S_YAB1), yA[2] - G(S_YAB2)};
    const bool confI = yA[0] >= 0.0;   // beta * yA_1 >= 0 with 0 < beta < pi
    FscTrig T;
    if (confI) { T.s = G(S_SIN1); T.c = G(S_COS1); T.ct = G(S_COT1); T.cth = G(S_CTH1); }
    else { T.s = G(S_SIN2); T.c = G(S_COS2); T.ct = G(S_COT2); T.cth = G(S_CTH2); }
    T.is = G(S_ISIN);
    T.k = T.s * (confI ? G(S_CTH2) : G(S_CTH1));   // sin times the tangent of the half angle
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 6; ++i) E[k][i] = 0.0;
    fsc_endpoint(yB, confI, T, nu, -G(S_PBZ), 1.0, E);
    fsc_endpoint(yA, confI, T, nu, -G(S_PAZ), -1.0, E);
    if (confI) {
        // y1, y2 and b1, b2 change sign: so do the 13 and 23 strains, and all of b1, b2
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int i = 0; i < 6; ++i)
                if ((k < 2) != (i > 3)) E[k][i] = -E[k][i];
    }
    return true;
}

template <class Fs>
struct FscSideOf {   // the fields of one side of a source
    const Fs &G;
    int o;
    __device__ __forceinline__ double operator()(int f) const { return G(o + f); }
};

// FSC strain (EFCS, xx yy zz xy xz yz) of one side at (X, Y, Z) for NB
// Burgers vectors given in the side frame, added to E[q].
template <int NB, class Fs>
__device__ __forceinline__ void fsc_side(const Fs &F, double X, double Y, double Z, double nu, const double b[NB][3],
                                         double E[NB][6])
{
    double U[3][6];
    if (!fsc_side_strains(F, X, Y, Z, nu, U)) return;
    const double c1 = F(S_C1), s1 = F(S_S1);
    const double K = 1.0 / (4.0 * kPi * (1.0 - nu));
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        double e[6];
#pragma unroll
        for (int i = 0; i < 6; ++i)
            e[i] = (i < 3 ? K : 0.5 * K) * (b[q][0] * U[0][i] + b[q][1] * U[1][i] + b[q][2] * U[2][i]);
        // local strain, then EFCS: E = A e A^T with A = [[c1, s1, 0], [s1, -c1, 0], [0, 0, -1]]
        const double cc = c1 * c1, ss = s1 * s1, cs = c1 * s1;
        E[q][0] += cc * e[0] + 2.0 * cs * e[3] + ss * e[1];
        E[q][1] += ss * e[0] - 2.0 * cs * e[3] + cc * e[1];
        E[q][2] += e[2];
        E[q][3] += cs * (e[0] - e[1]) + (ss - cc) * e[3];
        E[q][4] += -(c1 * e[4] + s1 * e[5]);
        E[q][5] += -(s1 * e[4] - c1 * e[5]);
    }
}

// The correction of one side as a matrix like an edge's (row c = traction component c of
// the receiver record R, column = Burgers component in the receiver's frame, in units of
// mu/(4 pi)), added to M.
template <class Fs>
__device__ __forceinline__ void fsc_matrix(const Fs &F, const double *R, double nu, double two_mu, double lam,
                                           double M[9])
{
    double U[3][6];
    if (!fsc_side_strains(F, R[0], R[1], R[2], nu, U)) return;
    const double c1 = F(S_C1), s1 = F(S_S1);
    // in units of mu/(4 pi): the strains' factor 1/(4 pi (1 - nu)) times 2 mu, lambda
    const double c2 = 2.0 / (1.0 - nu), cl = c2 * lam / two_mu;
    double r[3][3];   // the receiver's axes in the side's frame
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double *e = R + 3 + 3 * a;
        r[a][0] = e[0] * c1 + e[1] * s1;
        r[a][1] = e[0] * s1 - e[1] * c1;
        r[a][2] = -e[2];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double *e = U[k];
        const double h3 = 0.5 * e[3], h4 = 0.5 * e[4], h5 = 0.5 * e[5];
        const double u0 = e[0] * r[2][0] + h3 * r[2][1] + h4 * r[2][2];
        const double u1 = h3 * r[2][0] + e[1] * r[2][1] + h5 * r[2][2];
        const double u2 = h4 * r[2][0] + h5 * r[2][1] + e[2] * r[2][2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double t = c2 * (r[c][0] * u0 + r[c][1] * u1 + r[c][2] * u2);
            if (c == 2) t += cl * (e[0] + e[1] + e[2]);
#pragma unroll
            for (int a = 0; a < 3; ++a) M[3 * c + a] += t * r[a][k];
        }
    }
}

// Tractions (e1, e2, n of the receiver record R) of an EFCS strain.
__device__ __forceinline__ void tractions_efcs(const double E[6], const double *R, double two_mu, double lam,
                                                        double out[3])
{
    const double *n = R + 9;
    const double u0 = E[0] * n[0] + E[3] * n[1] + E[4] * n[2];
    const double u1 = E[3] * n[0] + E[1] * n[1] + E[5] * n[2];
    const double u2 = E[4] * n[0] + E[5] * n[1] + E[2] * n[2];
    const double tr = E[0] + E[1] + E[2];
    out[0] = two_mu * (R[3] * u0 + R[4] * u1 + R[5] * u2);
    out[1] = two_mu * (R[6] * u0 + R[7] * u1 + R[8] * u2);
    out[2] = two_mu * (n[0] * u0 + n[1] * u1 + n[2] * u2) + lam * tr;
}

// Half-space tractions of one pair (unit strike ts, unit dip td): main
// dislocation F, image Fi (mirrored triangle), side table G.
template <class Src, class Fs>
__device__ __forceinline__ void pair_tractions_hs(const Src &F, const Src &Fi, const Fs &G, const double *R,
                                                  double nu, double k, double two_mu, double lam, double ts[3],
                                                  double td[3])
{
    pair_tractions(F, R, nu, k, two_mu, lam, ts, td);
    double is[3], id[3];
    if (G(kFscSurface) != 0.0) {
        // surface triangle: the image equals the main strain with xz, yz
        // negated, i.e. the main strain seen through receiver axes reflected in z
        double Rr[kRecvStride];
#pragma unroll
        for (int q = 0; q < kRecvStride; ++q) Rr[q] = R[q];
        Rr[5] = -R[5]; Rr[8] = -R[8]; Rr[11] = -R[11];
        pair_tractions(F, Rr, nu, k, two_mu, lam, is, id);
    } else {
        pair_tractions(Fi, R, nu, k, two_mu, lam, is, id);
    }
    double E[2][6];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int i = 0; i < 6; ++i) E[q][i] = 0.0;
    for (int sd = 0; sd < 3; ++sd) {
        const FscSideOf<Fs> S{G, sd * S_COUNT};
        const double b[2][3] = {{S(S_BS0), S(S_BS1), S(S_BS2)}, {S(S_BD0), S(S_BD1), S(S_BD2)}};
        fsc_side<2>(S, R[0], R[1], R[2], nu, b, E);
    }
    double fs[3], fd[3];
    tractions_efcs(E[0], R, two_mu, lam, fs);
    tractions_efcs(E[1], R, two_mu, lam, fd);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ts[c] += fs[c] + is[c];
        td[c] += fd[c] + id[c];
    }
}

// Half-space strain (EFCS) at a point for the Burgers vector (bx, by, bz) =
// (tensile, strike, dip), in its four parts: one side of the free-surface
// correction, and the main and the image dislocation.
template <class Fs>
__device__ __forceinline__ void point_strain_side(const Fs &S, double X, double Y, double Z, double bx, double by,
                                                  double bz, double nu, double e[6])
{
    double E[1][6] = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}};
    double b[1][3];
    for (int c = 0; c < 3; ++c) b[0][c] = bx * S(S_BN0 + c) + by * S(S_BS0 + c) + bz * S(S_BD0 + c);
    fsc_side<1>(S, X, Y, Z, nu, b, E);
    for (int i = 0; i < 6; ++i) e[i] = E[0][i];
}

template <class Src>
__device__ __forceinline__ void point_strain_full(const Src &F, double X, double Y, double Z, double bx, double by,
                                                  double bz, double nu, double k, double e[6])
{
    double x, y, z, E[6];
    tdcs_point(F, X, Y, Z, x, y, z);
    tdcs_strain_general(F, x, y, z, bx, by, bz, nu, k, E);
    tdcs_to_efcs(F, E, e);
}

// surface: the triangle lies on the surface (kFscSurface)
__device__ __forceinline__ void image_signs(double surface, double e[6])
{
    if (surface != 0.0) { e[4] = -e[4]; e[5] = -e[5]; }
}

// All parts by one thread: for the host check (the kernels share them over warps).
template <class Src, class Fs>
__device__ __forceinline__ void point_strain_hs(const Src &F, const Src &Fi, const Fs &G, double X, double Y,
                                                double Z, double bx, double by, double bz, double nu, double k,
                                                double e[6])
{
    double ei[6], f[6], sum[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    point_strain_full(F, X, Y, Z, bx, by, bz, nu, k, e);
    point_strain_full(Fi, X, Y, Z, bx, by, bz, nu, k, ei);
    image_signs(G(kFscSurface), ei);
    for (int sd = 0; sd < 3; ++sd) {
        point_strain_side(FscSideOf<Fs>{G, sd * S_COUNT}, X, Y, Z, bx, by, bz, nu, f);
        for (int i = 0; i < 6; ++i) sum[i] += f[i];
    }
    for (int i = 0; i < 6; ++i) e[i] += sum[i] + ei[i];
}

}  // namespace gf
}  // namespace pq3d
