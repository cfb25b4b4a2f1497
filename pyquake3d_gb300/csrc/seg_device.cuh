// Full-space tractions of a triangular dislocation as a sum over its three
// edges: the closed-loop line integral of the elastic Green's function
// (Peach and Koehler 1950; Mura 1987, eq. 37.4; straight segments as in Hirth
// and Lothe 1982), written as one 3 x 3 matrix per (receiver, edge).
//
// With R the vector from a point of the edge to the receiver, t the edge's
// direction, w = R.t, d = R - t w, c = b x t and integrals over the edge
//   I30 = int 1/|R|^3, I31 = int w/|R|^3, J5q = 3 int w^q/|R|^5 (q = 0, 1, 2),
// the traction on the receiver's plane n is mu/(4 pi) M b, summed over the
// edges, with G = d I30 + t I31, u = t x d, kap = -1/(1 - nu) and
//   M b = (G x b)(t.n) + t ((G x b).n)
//       + kap [ -c (G.n) - G (c.n) + (n I30 + 3 int R (R.n)/|R|^5) (b.u) ].
// All vectors are in the receiver's frame (e1, e2, n), where n = (0, 0, 1):
// every product with n is a component, and the rows of M are the traction
// components the operator stores.
//
// Against the three angular dislocations of tdcs_strain_sd2k (the published
// expressions of the same field):
//   * the two infinite legs of each angular dislocation, which cancel between
//     neighbouring vertices, never appear: the field of an edge is that of a
//     finite segment, and the antiderivatives are taken on the side of the
//     edge on which they do not cancel (w >= 0 at the edge's far end).  Errors
//     against 80-bit arithmetic are smaller everywhere (random receivers,
//     relative to the pair's largest traction, median: 2e-15 against 4e-15 to
//     2e-14 at a third of an edge length, 2e-15 against 2e-14 beyond an edge's
//     end, 3e-13 against 8e-10 a thousandth of an edge from a vertex);
//   * an edge's matrix does not depend on the triangle it belongs to, so the
//     assembly forms it once for both triangles of an edge, and a vertex's
//     distance once for all its edges.
// A receiver closer to an edge than 1e-6 of its length (between the edge's
// end points) gets a NaN matrix, as do vanishing or non-finite distances: the
// caller evaluates such a pair by pair_tractions, whose configuration test
// also decides the pairs on an edge.
#pragma once

#include "gf_device.cuh"

namespace pq3d {
namespace gf {

// Per-edge constants: length, its reciprocal, and the square of the distance
// below which a receiver beside the edge counts as on it.
struct SegEdge {
    double L, iL;
    float near2;
};

__host__ __device__ inline SegEdge seg_edge_record(const double A[3], const double B[3])
{
    const double x = A[0] - B[0], y = A[1] - B[1], z = A[2] - B[2];
    const double L = sqrt(x * x + y * y + z * z);
    return SegEdge{L, 1.0 / L, (float)(1e-12 * (L * L))};
}

// A vertex seen from a receiver: the vector to the receiver in its frame,
// the distance, 1/distance and 1/distance^3.
struct SegVert {
    double x, y, z, r, ir, ir3;
};

// Material factors of the edge sum: kap = -1/(1 - nu); with lambda and nu the
// caller's own pair (the reference takes nu = 1/(1 + lambda/mu)/2 and applies
// Hooke's law with lambda), the normal traction carries lambda - 2 mu nu/(1 -
// 2 nu) times the dilatation, which is the same integral as the I30 term:
// ci = 1 + (1 - 2 nu) lambda/mu - 2 nu (1 for lambda = mu).
struct SegMat {
    double kap, ci, scale;   // scale = mu/(4 pi)
};

__host__ __device__ inline SegMat seg_material(double nu, double two_mu, double lam)
{
    return SegMat{-1.0 / (1.0 - nu), 1.0 + (1.0 - 2.0 * nu) * (2.0 * lam / two_mu) - 2.0 * nu, two_mu / (8.0 * kPi)};
}

#ifdef __CUDACC__
__device__ __forceinline__ double flip_sign(double v, unsigned s)   // v with its sign bit xor s
{
    return __hiloint2double((int)((unsigned)__double2hiint(v) ^ s), __double2loint(v));
}
__device__ __forceinline__ unsigned sign_bit(double v) { return (unsigned)__double2hiint(v) & 0x80000000u; }
__device__ __forceinline__ double seg_nan() { return __hiloint2double(0x7ff80000, 0); }
__device__ __forceinline__ float seg_small(double v) { return (float)seed_f32(v); }
#else
inline double flip_sign(double v, unsigned s) { return s ? -v : v; }
inline unsigned sign_bit(double v) { return std::signbit(v) ? 0x80000000u : 0u; }
inline double seg_nan() { return NAN; }
inline float seg_small(double v) { return (float)v; }
inline double seg_rcp(double p) { return 1.0 / p; }
inline void seg_rsqrt(double q, double &r, double &ir) { r = sqrt(q); ir = 1.0 / r; }
#endif

// R: receiver record (centroid, e1, e2, n).
__device__ __forceinline__ SegVert seg_vertex(const double *R, double vx, double vy, double vz)
{
    const double dx = R[0] - vx, dy = R[1] - vy, dz = R[2] - vz;
    SegVert v;
    v.x = R[3] * dx + R[4] * dy + R[5] * dz;
    v.y = R[6] * dx + R[7] * dy + R[8] * dz;
    v.z = R[9] * dx + R[10] * dy + R[11] * dz;
    seg_rsqrt(v.x * v.x + v.y * v.y + v.z * v.z, v.r, v.ir);
    v.ir3 = v.ir * v.ir * v.ir;
    return v;
}

// The edge integrals and vectors of one (receiver, edge A -> B).  The edge is
// walked in the direction in which the receiver lies ahead of its middle:
// reversing the edge changes the signs of t and w and of the whole field, so
// t and w take the sign and the differences B - A stay.
struct SegTerms {
    double tx, ty, tz, gx, gy, gz;   // t, G
    double dx, dy, dz;               // d
    double i30, al, be;              // I30; the factors of d and t in 3 int R (R.n)/|R|^5
    double ux, uy, uz;               // kap t x d
    bool on;                         // the receiver is on the edge (to 1e-6 of its length)
};

__device__ __forceinline__ SegTerms seg_terms(const SegVert &A, const SegVert &B, double L, double iL, float near2,
                                              double kap)
{
    SegTerms s;
    double tx = (A.x - B.x) * iL, ty = (A.y - B.y) * iL, tz = (A.z - B.z) * iL;
    double wA = tx * A.x + ty * A.y + tz * A.z;
    double wB = wA - L;
    s.dx = A.x - tx * wA;
    s.dy = A.y - ty * wA;
    s.dz = A.z - tz * wA;
    const bool between = sign_bit(wA) != sign_bit(wB);
    const unsigned sg = sign_bit(wA + wB);
    s.tx = tx = flip_sign(tx, sg);
    s.ty = ty = flip_sign(ty, sg);
    s.tz = tz = flip_sign(tz, sg);
    wA = flip_sign(wA, sg);
    wB = flip_sign(wB, sg);
    const double d2 = s.dx * s.dx + s.dy * s.dy + s.dz * s.dz;
    s.on = between && !(seg_small(d2) > near2);
    // antiderivatives: int w^-3-type terms by q = 1/(r (r + w)); both
    // reciprocals from one
    const double pA = A.r + wA, pB = B.r + wB, ip = seg_rcp(pA * pB);
    const double qA = A.ir * (ip * pB), qB = B.ir * (ip * pA);
    const double i31 = B.ir - A.ir, j51 = B.ir3 - A.ir3;
    s.i30 = qB - qA;
    const double j50 = qB * qB * fma(pB, B.ir, 1.0) - qA * qA * fma(pA, A.ir, 1.0);
    const double j52 = fma(-d2, j50, 3.0 * s.i30);
    s.gx = s.dx * s.i30 + tx * i31;
    s.gy = s.dy * s.i30 + ty * i31;
    s.gz = s.dz * s.i30 + tz * i31;
    s.al = s.dz * j50 + tz * j51;
    s.be = s.dz * j51 + tz * j52;
    const double kx = kap * tx, ky = kap * ty, kz = kap * tz;
    s.ux = ky * s.dz - kz * s.dy;
    s.uy = kz * s.dx - kx * s.dz;
    s.uz = kx * s.dy - ky * s.dx;
    return s;
}

// M (row c = traction component c, column = Burgers component in the
// receiver's frame) of one edge.
__device__ __forceinline__ void seg_matrix(const SegTerms &s, double kap, double ci, double M[9])
{
    const double qx = s.dx * s.al + s.tx * s.be, qy = s.dy * s.al + s.ty * s.be;
    const double qz = s.dz * s.al + (s.tz * s.be + ci * s.i30);
    const double hx = kap * s.gx, hy = kap * s.gy, hz = kap * s.gz;
    const double g1 = s.gx + hx, g2 = s.gy + hy, g3 = s.gz + hz;
    const double m02 = s.tz * s.gy + s.ty * hz, m12 = s.tz * s.gx + s.tx * hz, zz = s.tz * g3;
    M[0] = qx * s.ux - (s.tx * s.gy + s.ty * hx);
    M[1] = qx * s.uy + (s.tx * g1 - zz);
    M[2] = qx * s.uz + m02;
    M[3] = qy * s.ux + (zz - s.ty * g2);
    M[4] = qy * s.uy + (s.ty * s.gx + s.tx * hy);
    M[5] = qy * s.uz - m12;
    M[6] = qz * s.ux - 2.0 * m02;
    M[7] = qz * s.uy + 2.0 * m12;
    M[8] = qz * s.uz;
    if (s.on) M[0] = seg_nan();
}

// A traction that is not finite: the pair goes to pair_tractions.
__device__ __forceinline__ bool seg_bad(double t)
{
#ifdef __CUDACC__
    return ((unsigned)__double2hiint(t) & 0x7ff00000u) == 0x7ff00000u;
#else
    return !std::isfinite(t);
#endif
}

}  // namespace gf
}  // namespace pq3d
