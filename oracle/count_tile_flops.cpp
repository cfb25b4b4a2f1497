// Operation count of the tiled dense assemblies -- test infrastructure.  Compiles the
// device math of pyquake3d_gb300/csrc (seg_device.cuh, hs_device.cuh, gf_device.cuh) with
// every `double` replaced by a counting scalar type, counts one vertex, one edge (full
// space; half space: its matrix, its image's and its free-surface correction) and one
// pair, and adds them with the vertices and edges that the tiles of a mesh hold.  The
// mesh comes on stdin: "half N" (half: 0 or 1) then N lines of 9 vertex coordinates; the
// triangles are put in the assembly's spatial order where their own leaves more than 1.66
// edges a triangle.  The sums of the three edge matrices and their products with the slip
// vectors (the kernels' own lines) are restated here.  Convention as the other counts:
// add, sub, mul, div and sqrt count one each (a fused multiply-add is a mul and an add);
// comparisons, negations and loads are free.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <map>
#include <numeric>
#include <set>
#include <vector>

struct Ops { long long add = 0, mul = 0, div = 0, sqrt_ = 0, trans = 0; };
static Ops g_ops;

struct Q64 {
    double v;
    constexpr Q64() : v(0) {}
    constexpr Q64(double x) : v(x) {}
    explicit operator int() const { return (int)v; }
    explicit operator float() const { return (float)v; }
};
inline Q64 operator+(Q64 a, Q64 b) { ++g_ops.add; return Q64(a.v + b.v); }
inline Q64 operator-(Q64 a, Q64 b) { ++g_ops.add; return Q64(a.v - b.v); }
inline Q64 operator*(Q64 a, Q64 b) { ++g_ops.mul; return Q64(a.v * b.v); }
inline Q64 operator/(Q64 a, Q64 b) { ++g_ops.div; return Q64(a.v / b.v); }
inline Q64 operator-(Q64 a) { return Q64(-a.v); }
inline Q64 &operator+=(Q64 &a, Q64 b) { ++g_ops.add; a.v += b.v; return a; }
inline Q64 &operator-=(Q64 &a, Q64 b) { ++g_ops.add; a.v -= b.v; return a; }
inline Q64 &operator*=(Q64 &a, Q64 b) { ++g_ops.mul; a.v *= b.v; return a; }
inline Q64 &operator/=(Q64 &a, Q64 b) { ++g_ops.div; a.v /= b.v; return a; }
inline bool operator<(Q64 a, Q64 b) { return a.v < b.v; }
inline bool operator>(Q64 a, Q64 b) { return a.v > b.v; }
inline bool operator<=(Q64 a, Q64 b) { return a.v <= b.v; }
inline bool operator>=(Q64 a, Q64 b) { return a.v >= b.v; }
inline bool operator==(Q64 a, Q64 b) { return a.v == b.v; }
inline bool operator!=(Q64 a, Q64 b) { return a.v != b.v; }
inline Q64 fma(Q64 a, Q64 b, Q64 c) { ++g_ops.mul; ++g_ops.add; return Q64(a.v * b.v + c.v); }
inline Q64 sqrt(Q64 a) { ++g_ops.sqrt_; return Q64(std::sqrt(a.v)); }
inline Q64 fabs(Q64 a) { return Q64(std::fabs(a.v)); }
inline Q64 sin(Q64 a) { ++g_ops.trans; return Q64(std::sin(a.v)); }
inline Q64 cos(Q64 a) { ++g_ops.trans; return Q64(std::cos(a.v)); }
inline Q64 acos(Q64 a) { ++g_ops.trans; return Q64(std::acos(a.v)); }
namespace std {
inline bool isfinite(Q64 a) { return std::isfinite(a.v); }
inline bool signbit(Q64 a) { return std::signbit(a.v); }
}

#define PQ3D_OPCOUNT
#define double Q64
#include "../pyquake3d_gb300/csrc/hs_device.cuh"
#include "../pyquake3d_gb300/csrc/seg_device.cuh"
#undef double

using namespace pq3d::gf;

struct Arr {
    const Q64 *f;
    Q64 operator()(int i) const { return f[i]; }
};

static long long take()   // operations since the last call
{
    const long long n = g_ops.add + g_ops.mul + g_ops.div + g_ops.sqrt_;
    g_ops = Ops();
    return n;
}

typedef std::array<double, 3> Vec;
typedef std::array<Vec, 3> Tri;

// distinct vertices and edges of the tiles of ts triangles each, in the given order
static void tile_items(const std::vector<Tri> &tri, const std::vector<int> &order, int ts, long long *nv, long long *ne)
{
    *nv = *ne = 0;
    for (size_t t = 0; t < order.size(); t += ts) {
        std::set<Vec> v;
        std::set<std::pair<Vec, Vec>> e;
        for (size_t i = t; i < std::min(order.size(), t + ts); ++i)
            for (int q = 0; q < 3; ++q) {
                const Vec &a = tri[order[i]][q], &b = tri[order[i]][(q + 1) % 3];
                v.insert(a);
                e.insert(std::minmax(a, b));
            }
        *nv += (long long)v.size();
        *ne += (long long)e.size();
    }
}

int main()
{
    int half;
    long long N;
    if (scanf("%d %lld", &half, &N) != 2) return 1;
    std::vector<Tri> tri(N);
    for (auto &t : tri)
        for (auto &v : t)
            for (double &c : v)
                if (scanf("%lf", &c) != 1) return 1;
    // tiles: as many as needed of at most 256 (half space 240) triangles, all alike
    const long long most = half ? 240 : 256, tiles = (N + most - 1) / most, ts = (N + tiles - 1) / tiles;
    std::vector<int> order(N);
    std::iota(order.begin(), order.end(), 0);
    long long nv, ne;
    tile_items(tri, order, (int)ts, &nv, &ne);
    const bool sorted = 100 * ne > 166 * N;
    if (sorted) {   // by the centroids' Morton codes
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, ext = 0.f;
        std::vector<std::array<float, 3>> g(N);
        for (long long j = 0; j < N; ++j)
            for (int c = 0; c < 3; ++c) {
                g[j][c] = (float)((tri[j][0][c] + tri[j][1][c] + tri[j][2][c]) / 3.0);
                lo[c] = std::min(lo[c], g[j][c]);
                hi[c] = std::max(hi[c], g[j][c]);
            }
        for (int c = 0; c < 3; ++c) ext = std::max(ext, hi[c] - lo[c]);
        const float scale = ext > 0.f ? 1023.f / ext : 0.f;
        std::vector<unsigned> key(N, 0u);
        for (long long j = 0; j < N; ++j)
            for (int c = 0; c < 3; ++c) {
                const unsigned v = (unsigned)std::min(std::max((g[j][c] - lo[c]) * scale, 0.f), 1023.f);
                for (int b = 0; b < 10; ++b) key[j] |= ((v >> b) & 1u) << (3 * b + c);
            }
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key[a] < key[b]; });
        tile_items(tri, order, (int)ts, &nv, &ne);
    }
    // one vertex, edge and pair of the mesh: the counts are the same for all
    Q64 P[3][3], R[kRecvStride], src[kSrcStride];
    for (int q = 0; q < 3; ++q)
        for (int c = 0; c < 3; ++c) P[q][c] = tri[0][q][c];
    Q64 far[3][3];
    for (int q = 0; q < 3; ++q)
        for (int c = 0; c < 3; ++c) far[q][c] = tri[N - 1][q][c];
    setup_receiver(far[0], far[1], far[2], R);
    setup_source(P[0], P[1], P[2], src, 1);
    const double mu = 32038120320.0, nu = 0.25;
    const SegMat mat = seg_material(Q64(nu), Q64(2.0 * mu), Q64(mu));
    const SegEdge e = seg_edge_record(P[0], P[1]);
    take();
    const SegVert A = seg_vertex(R, P[0][0], P[0][1], P[0][2]);
    const long long vertex = take();
    const SegVert B = seg_vertex(R, P[1][0], P[1][1], P[1][2]);
    take();
    const SegTerms s = seg_terms(A, B, e.L, e.iL, e.near2, mat.kap);
    const long long terms = take();
    Q64 M[9];
    seg_matrix(s, mat.kap, mat.ci, M);
    const long long matrix = take();
    // a triangle's sums: the slip vectors in the receiver's frame, three matrices, six products
    Q64 ts3[3], td3[3], vs[3], vd[3];
    const Q64 zero(0.0);
    take();
    for (int a = 0; a < 3; ++a) {
        vs[a] = R[3 + 3 * a] * src[F_SX] + R[4 + 3 * a] * src[F_SY];
        vd[a] = R[3 + 3 * a] * src[F_DX] + R[4 + 3 * a] * src[F_DY] + R[5 + 3 * a] * src[F_DZ];
    }
    for (int c = 0; c < 3; ++c) {
        Q64 m[3];
        for (int a = 0; a < 3; ++a) m[a] = (M[3 * c + a] + M[3 * c + a]) + M[3 * c + a];
        ts3[c] = m[0] * vs[0] + m[1] * vs[1] + m[2] * vs[2];
        td3[c] = m[0] * vd[0] + m[1] * vd[1] + m[2] * vd[2];
    }
    const long long sums = take();
    long long edge = terms + matrix, pair = sums, ends = 0, contraction = 0;
    double per_pair;
    const double vt = (double)nv / N, et = (double)ne / N;
    if (half) {
        // the same for the edges and for their images, with the slip vectors scaled (6
        // products) and the products added to the sum so far (6 additions)
        pair = 2 * (sums + 6 + 6);
        // the correction of a side that contributes one
        Q64 f[S_COUNT], U[3][6];
        bool found = false;
        for (int q = 0; q < 3 && !found; ++q) {
            setup_fsc_side(P[q], P[(q + 1) % 3], P[(q + 2) % 3], 0, f, 1);
            found = f[S_VALID].v != 0.0;
        }
        if (!found) return 1;
        take();
        fsc_side_strains(Arr{f}, R[0], R[1], R[2], Q64(nu), U);
        ends = take();
        for (Q64 &m : M) m = zero;
        fsc_matrix(Arr{f}, R, Q64(nu), Q64(2.0 * mu), Q64(mu), M);
        contraction = take() - ends;
        edge = 2 * (terms + matrix) + 4 * vertex + ends + contraction;   // its end points by itself
        per_pair = et * edge + pair;
    } else {
        per_pair = vt * vertex + et * edge + pair;
    }
    printf("{\"half\": %d, \"N\": %lld, \"spatial_order\": %s, \"vertices_per_triangle\": %.4f, \"edges_per_triangle\": %.4f, "
           "\"vertex\": %lld, \"edge_terms\": %lld, \"edge_matrix\": %lld, \"side_end_points\": %lld, "
           "\"side_contraction\": %lld, \"edge\": %lld, \"pair\": %lld, \"flops_per_pair\": %.1f}\n",
           half, N, sorted ? "true" : "false", vt, et, vertex, terms, matrix, ends, contraction, edge, pair, per_pair);
    return 0;
}
