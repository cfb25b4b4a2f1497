// Host build of the tiled assemblies' device math (pyquake3d_gb300/csrc/seg_device.cuh
// and the side matrix of hs_device.cuh) for the CPU tests: the tractions of a
// (receiver, source) pair from the matrices of the source's three edges, as
// assemble_seg_kernel and assemble_hs_kernel form and add them.  Test infrastructure
// only.
//
// stdin: "n lam_over_mu" then n lines "P1(3) P2(3) P3(3) X(3) e1(3) e2(3) n(3) rev"
//   (bit q of rev: edge q is kept in the tile from its second vertex to its first)
// stdout: per case 12 numbers: full-space ts(3) td(3), half-space ts(3) td(3)
#include <cmath>
#include <cstdio>

#include "../pyquake3d_gb300/csrc/hs_device.cuh"
#include "../pyquake3d_gb300/csrc/seg_device.cuh"

using namespace pq3d::gf;

struct Arr {
    const double *f;
    double operator()(int i) const { return f[i]; }
};

// the sums of one triangle: M[q] the matrix of edge q, rev[q] walked backwards
static void add_triangle(const double M[3][9], const unsigned rev[3], const double *f, const double *R, double scale,
                         double ts[3], double td[3])
{
    double vs[3], vd[3];
    for (int a = 0; a < 3; ++a) {
        vs[a] = scale * (R[3 + 3 * a] * f[F_SX] + R[4 + 3 * a] * f[F_SY]);
        vd[a] = scale * (R[3 + 3 * a] * f[F_DX] + R[4 + 3 * a] * f[F_DY] + R[5 + 3 * a] * f[F_DZ]);
    }
    for (int c = 0; c < 3; ++c)
        for (int a = 0; a < 3; ++a) {
            double m = 0.0;
            for (int q = 0; q < 3; ++q) m += flip_sign(M[q][3 * c + a], rev[q]);
            ts[c] += m * vs[a];
            td[c] += m * vd[a];
        }
}

static void edge(const double *A, const double *B, double sz, const double *R, const SegMat &mat, double M[9])
{
    const SegEdge e = seg_edge_record(A, B);
    seg_matrix(seg_terms(seg_vertex(R, A[0], A[1], sz * A[2]), seg_vertex(R, B[0], B[1], sz * B[2]), e.L, e.iL, e.near2,
                         mat.kap), mat.kap, mat.ci, M);
}

int main()
{
    int n;
    double ratio;
    if (scanf("%d %lf", &n, &ratio) != 2) return 1;
    const double mu = 32038120320.0, lam = ratio * mu;
    const double nu = 1.0 / (1.0 + lam / mu) / 2.0;
    const SegMat mat = seg_material(nu, 2.0 * mu, lam);
    for (int c = 0; c < n; ++c) {
        double v[21];
        unsigned bits;
        for (int i = 0; i < 21; ++i)
            if (scanf("%lf", &v[i]) != 1) return 1;
        if (scanf("%u", &bits) != 1) return 1;
        const double *P[3] = {v, v + 3, v + 6}, *R = v + 9;
        double src[kSrcStride], img[kSrcStride];
        const double Q[3][3] = {{v[0], v[1], -v[2]}, {v[3], v[4], -v[5]}, {v[6], v[7], -v[8]}};
        setup_source(P[0], P[1], P[2], src, 1);
        setup_source(Q[0], Q[1], Q[2], img, 1);
        double M[3][9], Mi[3][9], Mh[3][9];
        unsigned rev[3];
        for (int q = 0; q < 3; ++q) {
            rev[q] = (bits >> q) & 1u ? 0x80000000u : 0u;
            const double *A = P[rev[q] ? (q + 1) % 3 : q], *B = P[rev[q] ? q : (q + 1) % 3];
            edge(A, B, 1.0, R, mat, M[q]);
            edge(A, B, -1.0, R, mat, Mi[q]);
            double f[S_COUNT];
            setup_fsc_side(A, B, P[(q + 2) % 3], 0, f, 1);
            for (int i = 0; i < 9; ++i) Mh[q][i] = M[q][i];
            fsc_matrix(Arr{f}, R, nu, 2.0 * mu, lam, Mh[q]);
        }
        double t[4][3] = {};
        add_triangle(M, rev, src, R, mat.scale, t[0], t[1]);
        add_triangle(Mh, rev, src, R, mat.scale, t[2], t[3]);
        add_triangle(Mi, rev, img, R, mat.scale, t[2], t[3]);
        for (int q = 0; q < 4; ++q)
            for (int i = 0; i < 3; ++i) printf("%.17g ", t[q][i]);
        printf("\n");
    }
    return 0;
}
