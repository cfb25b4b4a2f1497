// Green's-function kernels and the reference-compatible C-ABI.
//
//   setup_sources / setup_receivers   once per mesh: per-source record (frame,
//                                     angles, side vectors) and per-receiver
//                                     record (centroid, frame)
//   setup_tiles                       once per mesh: the vertices and edges that
//                                     the triangles of a tile share
//   assemble_seg                      full space: per (tile of sources,
//                                     receiver) every vertex distance and edge
//                                     matrix once, then one (receiver, source)
//                                     pair per thread, both unit slips, 6
//                                     tractions -> FP64 K (+ FP32 copy) with
//                                     16-byte stores
//   assemble_hs                       half space: the same, with the edge's image
//                                     and its free-surface correction
//   points_full / points_hs           the two host-pointer entry points of the
//                                     reference TDstressFS_C.so
//   half-space (jud_halfspace / halfspace != 0): per-source image record and
//   free-surface side table (setup_hs) for single pairs (pair_tractions_hs,
//   hs_device.cuh), per-edge records (setup_tiles) for the assembly
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "gf_device.cuh"
#include "hs_device.cuh"
#include "seg_device.cuh"

namespace pq3d {
namespace gf {

struct SoaSrc {   // field f of one source in a structure-of-arrays table
    const double *base;
    int stride;
    __device__ __forceinline__ double operator()(int f) const { return base[f * stride]; }
};

struct ValSrc {   // fields held in a small array
    const double *f;
    __device__ __forceinline__ double operator()(int i) const { return f[i]; }
};

struct SrcVal { double f[kSrcStride]; };
struct FscVal { double f[kFscStride]; };

__device__ __forceinline__ void load_triangle(const double *__restrict__ nodes, const int64_t *__restrict__ tris,
                                              int64_t j, double a[3], double b[3], double c[3])
{
    const double *A = nodes + 3 * (tris[3 * j] - 1), *B = nodes + 3 * (tris[3 * j + 1] - 1),
                 *C = nodes + 3 * (tris[3 * j + 2] - 1);
    for (int q = 0; q < 3; ++q) { a[q] = A[q]; b[q] = B[q]; c[q] = C[q]; }
}

// Source and receiver records of element j, in one launch: blocks [0, nb) the
// sources, [nb, 2 nb) the receivers (both are short chains of FP64 latency).
__global__ void setup_elements_kernel(const double *__restrict__ nodes, const int64_t *__restrict__ tris, int64_t N,
                                      unsigned nb, double *__restrict__ src, double *__restrict__ recv)
{
    const bool source = blockIdx.x < nb;
    const int64_t j = (blockIdx.x - (source ? 0u : nb)) * (int64_t)blockDim.x + threadIdx.x;
    if (j >= N) return;
    double a[3], b[3], c[3];
    load_triangle(nodes, tris, j, a, b, c);
    if (source) setup_source(a, b, c, src + j, (int)N);
    else setup_receiver(a, b, c, recv + kRecvStride * j);
}

// ---------------------------------------------------------------------------
// tiles of sources: ts triangles next to one another (in the mesh's order or in
// order_tiles_kernel's) and the distinct vertices and edges they use

constexpr int kTileMax = 256;   // triangles of a tile at most
constexpr int kTileItems = 3 * kTileMax;

struct __align__(8) TileEdge {   // local edge: from vertex a to vertex b (the smaller node id first)
    double L, iL;
    float near2;
    uint16_t a, b;
};
struct __align__(8) TileTri {    // local edges of P1 P2, P2 P3, P3 P1; bit 15: walked from b to a
    uint16_t e[3], pad;
};
struct Tile {
    int32_t nv, ne, pad[2];
    double vert[kTileItems][3];
    TileEdge edge[kTileItems];
    TileTri tri[kTileMax];
    int32_t id[kTileMax];   // the triangles' numbers in the mesh
};
constexpr int kSegDoubles = (int)(sizeof(Tile) / sizeof(double));
static_assert(sizeof(Tile) % 16 == 0, "tiles start 16-byte aligned");
// Half space: the geometric fields of the edges' free-surface record (those of
// setup_fsc_side before the Burgers vectors, and 1 / sin beta), one row a field.
constexpr int kHsFields = S_BN0 + 1;
struct TileHs {
    double f[kHsFields][kTileItems];
};
constexpr int kHsDoubles = (int)(sizeof(TileHs) / sizeof(double));
struct TileSide {   // the record of one edge
    const double *f;
    __device__ __forceinline__ double operator()(int i) const
    {
        return __ldg(f + (i == S_ISIN ? kHsFields - 1 : i) * kTileItems);
    }
};

// (half space: 240 triangles, so that the matrices of 720 edges that none
// share leave room for two blocks per SM)
constexpr int kTileMaxHs = 240;
inline int64_t tile_count(int64_t N, bool half = false)
{
    const int most = half ? kTileMaxHs : kTileMax;
    return (N + most - 1) / most;
}
// equal tiles: the last one of N = 1,600 would hold 64 of 256 triangles, and
// its blocks would idle while the others finish
inline int tile_size(int64_t N, bool half = false)
{
    return (int)((N + tile_count(N, half) - 1) / tile_count(N, half));
}

// One block per tile: the node ids and the node pairs go into hash tables in
// shared memory; the thread that places a key takes the next local index.
// (The numbering depends on the order of arrival; no value computed from the
// tables does.)
constexpr int kHash = 2048;
__global__ void __launch_bounds__(kTileMax)
setup_tiles_kernel(const double *__restrict__ nodes, const int64_t *__restrict__ tris, int64_t N, int ts,
                   const int32_t *__restrict__ order, Tile *__restrict__ tiles, TileHs *__restrict__ hs)
{
    if (order && order[N] == 0) return;   // the tiles stand as they are
    __shared__ unsigned long long vkey[kHash], ekey[kHash];
    __shared__ uint16_t vidx[kHash], eidx[kHash];
    __shared__ int nv, ne;
    const int t = threadIdx.x;
    for (int i = t; i < kHash; i += kTileMax) vkey[i] = ekey[i] = ~0ull;
    if (t == 0) nv = ne = 0;
    __syncthreads();
    Tile &T = tiles[blockIdx.x];
    const int64_t pos = (int64_t)blockIdx.x * ts + t;
    const bool on = t < ts && pos < N;
    const int64_t j = on && order ? order[pos] : pos;
    int vs[3], es[3];
    bool vown[3], eown[3];
    int64_t id[3];
    // at most 768 keys in 2,048 places: the probe ends
    auto place = [](unsigned long long *key, uint16_t *idx, int *count, unsigned long long k, int &slot) {
        slot = (int)((k * 0x9E3779B97F4A7C15ull) >> 53);
        for (int probe = 0; probe < kHash; ++probe, slot = (slot + 1) & (kHash - 1)) {
            const unsigned long long old = atomicCAS(&key[slot], ~0ull, k);
            if (old == ~0ull) {
                idx[slot] = (uint16_t)atomicAdd(count, 1);
                return true;
            }
            if (old == k) return false;
        }
        return false;
    };
    if (on) {
#pragma unroll
        for (int q = 0; q < 3; ++q) id[q] = tris[3 * j + q];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const unsigned long long p = (unsigned long long)id[q], r = (unsigned long long)id[(q + 1) % 3];
            vown[q] = place(vkey, vidx, &nv, p, vs[q]);
            eown[q] = place(ekey, eidx, &ne, p < r ? (p << 32 | r) : (r << 32 | p), es[q]);
        }
    }
    __syncthreads();
    if (on) {
        TileTri tri;
        tri.pad = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int n = (q + 1) % 3;
            const bool rev = id[q] > id[n];
            if (vown[q])
                for (int c = 0; c < 3; ++c) T.vert[vidx[vs[q]]][c] = nodes[3 * (id[q] - 1) + c];
            const int e = eidx[es[q]];
            if (eown[q]) {
                const SegEdge r = seg_edge_record(nodes + 3 * (id[q] - 1), nodes + 3 * (id[n] - 1));
                T.edge[e] = TileEdge{r.L, r.iL, r.near2, vidx[vs[rev ? n : q]], vidx[vs[rev ? q : n]]};
                if (hs) {
                    const double *A = nodes + 3 * (id[rev ? n : q] - 1), *B = nodes + 3 * (id[rev ? q : n] - 1);
                    double f[S_COUNT];
                    setup_fsc_side(A, B, nodes + 3 * (id[(q + 2) % 3] - 1), 0, f, 1);
                    f[kHsFields - 1] = f[S_ISIN];
                    for (int i = 0; i < kHsFields; ++i) hs[blockIdx.x].f[i][e] = f[i];
                }
            }
            tri.e[q] = (uint16_t)(e | (rev ? 0x8000 : 0));
        }
        T.tri[t] = tri;
        T.id[t] = (int32_t)j;
    }
    if (t == 0) { T.nv = nv; T.ne = ne; }
}

// A spatial order of the triangles for meshes whose own order leaves tiles of
// many edges: the stable sort of the centroids' Morton codes (10 bits an axis),
// by one block, into order[0 .. N); order[N] = 1, or 0 where the tiles are kept.
// `tiles` is scratch from there on (12 bytes a triangle; they are set up anew).
//
// A tile of consecutive triangles is a strip of a structured mesh (1.75 edges a
// triangle at 163 columns of 62 squares) and anything up to 3 in an unordered
// one.  N = 20,000, FP64 output: in column order 167.7 -> 161.5 ms, shuffled 286.6
// -> 162.0 ms; half space, N = 2,500, shuffled 61.3 -> 36.5 ms.
// The lines: below 2^24 pairs (7 ms; half space 2^20, 6 ms) the two launches and
// the sort (40 us at N = 4,200, 130 us at 20,000) are a visible part of the call;
// at 1.66 edges a triangle there is little left to gain.  Full space into host
// memory keeps the mesh's order: neighbouring lanes' triangles are not neighbours in
// a row, and the link takes isolated 16- and 8-byte stores at a third of the rate
// (N = 20,040, shuffled, FP64 / with the FP32 copy: 436 / 903 ms sorted, 288 / 290 ms
// as it is; in column order 181 / 319 and 168 / 170 ms).  The half space is slow
// enough for the link either way (N = 3,600, shuffled: 77 ms sorted).
constexpr int64_t kOrderPairs = 1 << 24, kOrderPairsHs = 1 << 20;
constexpr int kOrderEdges = 166;   // per 100 triangles
constexpr int kOrderThreads = 1024;

__global__ void __launch_bounds__(kOrderThreads)
order_tiles_kernel(const double *__restrict__ recv, int64_t N, int64_t ntiles, Tile *tiles, int32_t *order)
{
    constexpr int kW = kOrderThreads / 32;
    __shared__ int hist[256][kW + 1];
    __shared__ float lo[3][kW], hi[3][kW];
    __shared__ int total;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    if (t == 0) total = 0;
    __syncthreads();
    for (int64_t q = t; q < ntiles; q += kOrderThreads) atomicAdd(&total, tiles[q].ne);
    __syncthreads();
    const bool sort = 100 * (int64_t)total > kOrderEdges * N;
    if (t == 0) order[N] = sort;
    if (!sort) return;
    // the centroids' box (fminf and fmaxf pass over NaN)
    float a[3] = {INFINITY, INFINITY, INFINITY}, b[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int64_t j = t; j < N; j += kOrderThreads)
        for (int c = 0; c < 3; ++c) {
            const float x = (float)recv[j * kRecvStride + c];
            a[c] = fminf(a[c], x);
            b[c] = fmaxf(b[c], x);
        }
    float ext = 0.f;
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            a[c] = fminf(a[c], __shfl_xor_sync(0xffffffffu, a[c], o));
            b[c] = fmaxf(b[c], __shfl_xor_sync(0xffffffffu, b[c], o));
        }
        if (lane == 0) { lo[c][w] = a[c]; hi[c][w] = b[c]; }
    }
    __syncthreads();
    for (int c = 0; c < 3; ++c) {
        for (int q = 0; q < kW; ++q) { a[c] = fminf(a[c], lo[c][q]); b[c] = fmaxf(b[c], hi[c][q]); }
        ext = fmaxf(ext, b[c] - a[c]);
    }
    const float scale = ext > 0.f ? 1023.f / ext : 0.f;
    uint32_t *key[2] = {(uint32_t *)tiles, (uint32_t *)tiles + N};
    int32_t *idx[2] = {order, (int32_t *)tiles + 2 * N};
    for (int64_t j = t; j < N; j += kOrderThreads) {
        uint32_t k = 0;
        for (int c = 0; c < 3; ++c) {
            const float x = ((float)recv[j * kRecvStride + c] - a[c]) * scale;
            uint32_t v = (uint32_t)(int)fminf(fmaxf(x, 0.f), 1023.f);
            v = (v | v << 16) & 0x030000ffu;
            v = (v | v << 8) & 0x0300f00fu;
            v = (v | v << 4) & 0x030c30c3u;
            v = (v | v << 2) & 0x09249249u;
            k |= v << c;
        }
        key[0][j] = k;
        idx[0][j] = (int32_t)j;
    }
    // four passes of 8 bits, a warp a contiguous part of the list
    const int64_t part = (N + kOrderThreads - 1) / kOrderThreads * 32;
    const int64_t j0 = w * part, j1 = j0 + part < N ? j0 + part : N;
    for (int pass = 0; pass < 4; ++pass) {
        const uint32_t *ki = key[pass & 1];
        const int32_t *ii = idx[pass & 1];
        uint32_t *ko = key[1 - (pass & 1)];
        int32_t *io = idx[1 - (pass & 1)];
        __syncthreads();   // the last pass's lists are in
        for (int q = t; q < 256 * (kW + 1); q += kOrderThreads) (&hist[0][0])[q] = 0;
        __syncthreads();
        for (int64_t j = j0 + lane; j < j1; j += 32) atomicAdd(&hist[(ki[j] >> (8 * pass)) & 255][w], 1);
        __syncthreads();
        // exclusive sums over (digit, warp): a warp takes 8 digits
        int sum = 0;
        for (int d = 8 * w; d < 8 * w + 8; ++d) {
            int v = hist[d][lane], x = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            hist[d][lane] = sum + x - v;
            sum += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) hist[w][kW] = sum;
        __syncthreads();
        int before = 0;
        for (int q = 0; q < w; ++q) before += hist[q][kW];
        for (int d = 8 * w; d < 8 * w + 8; ++d) hist[d][lane] += before;
        __syncthreads();
        for (int64_t jb = j0; jb < j1; jb += 32) {
            const int64_t j = jb + lane;
            const bool on = j < j1;
            const uint32_t k = on ? ki[j] : 0u;
            const int32_t i = on ? ii[j] : 0;
            const int d = on ? (int)((k >> (8 * pass)) & 255) : 256;
            const unsigned same = __match_any_sync(0xffffffffu, d);
            const int rank = __popc(same & ((1u << lane) - 1u));
            int at = 0;
            if (on) at = hist[d][w] + rank;
            __syncwarp();
            if (on && rank == 0) hist[d][w] += __popc(same);
            __syncwarp();
            if (on) { ko[at] = k; io[at] = i; }
        }
    }
}

// Half-space records of source j: the mirrored triangle's source record
// (img, stride N) and the free-surface side table (fsc, stride N).
__global__ void setup_hs_kernel(const double *__restrict__ nodes, const int64_t *__restrict__ tris, int64_t N,
                                double *__restrict__ img, double *__restrict__ fsc)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= N) return;
    const double *P1 = nodes + 3 * (tris[3 * j] - 1);
    const double *P2 = nodes + 3 * (tris[3 * j + 1] - 1);
    const double *P3 = nodes + 3 * (tris[3 * j + 2] - 1);
    double a[3] = {P1[0], P1[1], P1[2]}, b[3] = {P2[0], P2[1], P2[2]}, c[3] = {P3[0], P3[1], P3[2]};
    double am[3] = {a[0], a[1], -a[2]}, bm[3] = {b[0], b[1], -b[2]}, cm[3] = {c[0], c[1], -c[2]};
    setup_source(am, bm, cm, img + j, (int)N);
    setup_fsc(a, b, c, fsc + j, (int)N);
}

// ---------------------------------------------------------------------------
// Full-space dense assembly from the tiles.  Per batch of receivers: (1) every
// vertex of the tile from every receiver, (2) every edge's matrix, both items
// spread evenly over the block, (3) a thread per triangle adds its three edge
// matrices and applies them to its two slip directions.
//
// Bound: the FP64 pipe (2 lanes per clock and SM).  About 21 FP64 operations
// per vertex, 95 per edge and 54 per pair; on a structured mesh a tile of 256
// triangles has 0.6 vertices and 1.63 edges per triangle, so a pair takes ~220
// (520 as three angular dislocations per pair).  256 triangles per tile: 128
// have 1.9 edges per triangle; more would leave one block per SM.
constexpr int kSegThreads = 256;
constexpr int kSegRecv = 64;              // receivers of a block at most
constexpr int kSegSmem = 104 * 1024;      // two blocks per SM; holds the 768 vertices and edges of a tile
                                          // that shares none for one receiver (90 KB)
constexpr int kVertD = 6, kMatD = 9;
static_assert((kVertD + kMatD) * kTileItems * sizeof(double) <= kSegSmem, "one receiver of any tile fits");

// The pair by its angular dislocations (receivers on an edge of the source).
__device__ __noinline__ void pair_angular(const double *src, int64_t N, const double *R, double nu, double k,
                                          double two_mu, double lam, double ts[3], double td[3])
{
    const SoaSrc F{src, (int)N};
    pair_tractions(F, R, nu, k, two_mu, lam, ts, td);
}

// K64 / K32 point at row 3*row0; leading dimension 2N; nr receivers per block.
template <bool kWrite32>
__global__ void __launch_bounds__(kSegThreads, 2)
assemble_seg_kernel(const Tile *__restrict__ tiles, int ts, const double *__restrict__ src,
                    const double *__restrict__ recv, int64_t N, int64_t row0, int64_t row1, int nr, SegMat mat,
                    double nu, double k, double two_mu, double lam, double *__restrict__ K64, float *__restrict__ K32)
{
    extern __shared__ double s_buf[];
    __shared__ double s_rcv[kSegRecv * kRecvStride];
    const int t = threadIdx.x;
    const Tile &T = tiles[blockIdx.x];
    const int nv = T.nv, ne = T.ne;
    const int64_t i0 = row0 + (int64_t)blockIdx.y * nr;
    const int nrec = (int)((row1 - i0) < nr ? (row1 - i0) : nr);
    for (int q = t; q < nrec * kRecvStride; q += kSegThreads) s_rcv[q] = recv[i0 * kRecvStride + q];
    const int batch = min(nrec, kSegSmem / (int)sizeof(double) / (nv * kVertD + ne * kMatD));
    double *sv = s_buf, *sm = s_buf + (size_t)batch * nv * kVertD;
    // this thread's triangle: edges, and its slip directions times mu/(4 pi)
    const bool on = t < ts && (int64_t)blockIdx.x * ts + t < N;
    const int64_t j = on ? T.id[t] : 0;
    int e[3];
    unsigned sg[3];
    double bs[2], bd[3];
    if (on) {
        const TileTri tri = T.tri[t];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            e[q] = (tri.e[q] & 0x7fff) * kMatD;
            sg[q] = (unsigned)(tri.e[q] & 0x8000) << 16;
            if (q < 2) bs[q] = mat.scale * src[(F_SX + q) * N + j];
            bd[q] = mat.scale * src[(F_DX + q) * N + j];
        }
    }
    const int64_t ld = 2 * N;
    for (int b0 = 0; b0 < nrec; b0 += batch) {
        const int nb = min(batch, nrec - b0);
        __syncthreads();   // the receivers are in; the last batch's readers are done
        for (int q = t; q < nb * nv; q += kSegThreads) {
            const int r = q / nv, v = q - r * nv;
            const SegVert p = seg_vertex(s_rcv + (b0 + r) * kRecvStride, T.vert[v][0], T.vert[v][1], T.vert[v][2]);
            double *o = sv + q * kVertD;
            reinterpret_cast<double2 *>(o)[0] = make_double2(p.x, p.y);
            reinterpret_cast<double2 *>(o)[1] = make_double2(p.z, p.r);
            reinterpret_cast<double2 *>(o)[2] = make_double2(p.ir, p.ir3);
        }
        __syncthreads();
        for (int q = t; q < nb * ne; q += kSegThreads) {
            const int r = q / ne;
            const TileEdge ed = T.edge[q - r * ne];
            auto vert = [&](int v) {
                const double2 *o = reinterpret_cast<const double2 *>(sv + (r * nv + v) * kVertD);
                return SegVert{o[0].x, o[0].y, o[1].x, o[1].y, o[2].x, o[2].y};
            };
            double M[9];
            seg_matrix(seg_terms(vert(ed.a), vert(ed.b), ed.L, ed.iL, ed.near2, mat.kap), mat.kap, mat.ci, M);
#pragma unroll
            for (int c = 0; c < 9; ++c) sm[q * kMatD + c] = M[c];
        }
        __syncthreads();
        if (!on) continue;
        for (int r = 0; r < nb; ++r) {
            const double *R = s_rcv + (b0 + r) * kRecvStride, *Mr = sm + r * ne * kMatD;
            double vs[3], vd[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                vs[a] = R[3 + 3 * a] * bs[0] + R[4 + 3 * a] * bs[1];   // the strike axis is horizontal
                vd[a] = R[3 + 3 * a] * bd[0] + R[4 + 3 * a] * bd[1] + R[5 + 3 * a] * bd[2];
            }
            double ts3[3], td3[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double m[3];
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    m[a] = (flip_sign(Mr[e[0] + 3 * c + a], sg[0]) + flip_sign(Mr[e[1] + 3 * c + a], sg[1])) +
                           flip_sign(Mr[e[2] + 3 * c + a], sg[2]);
                ts3[c] = m[0] * vs[0] + m[1] * vs[1] + m[2] * vs[2];
                td3[c] = m[0] * vd[0] + m[1] * vd[1] + m[2] * vd[2];
            }
            if (seg_bad(ts3[0])) pair_angular(src + j, N, R, nu, k, two_mu, lam, ts3, td3);
            const int64_t row = 3 * (i0 + b0 + r - row0);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                *reinterpret_cast<double2 *>(K64 + (row + c) * ld + 2 * j) = make_double2(ts3[c], td3[c]);
                if (kWrite32)
                    *reinterpret_cast<float2 *>(K32 + (row + c) * ld + 2 * j) =
                        make_float2(d2f_rn_bits(ts3[c]), d2f_rn_bits(td3[c]));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Half-space dense assembly from the tiles: per receiver (1) every edge's
// matrices -- that of the edge with its free-surface correction, and that of
// its mirror image, whose triangles slip along axes of their own -- and (2) the
// triangles' sums.  The correction of an edge walked the other way is its
// negative, so that it too serves both triangles of an edge.
//
// Bound: the FP64 pipe, with the correction's two end points 85 % of an edge's
// ~1,700 operations; an edge per item instead of three sides per pair is 1.7
// instead of 3 of them on a structured mesh (N = 2,500: 67.8 ms with a thread
// per pair, 35.3 ms; 102 ms with the derivatives in nine variables, a thread per pair).
constexpr int kHsThreads = 128;   // 255 registers, two blocks per SM
constexpr int kHsRecv = 16;       // receivers of a block at most
constexpr int kHsMatD = 18;
constexpr int kHsSmem = 3 * kTileMaxHs * kHsMatD * (int)sizeof(double);

// The pair by its angular dislocations (receivers on an edge of the source or
// of its image; sources in the surface).
__device__ __noinline__ void pair_angular_hs(const double *src, const double *img, const double *fsc, int64_t N,
                                             const double *R, double nu, double k, double two_mu, double lam,
                                             double ts[3], double td[3])
{
    const SoaSrc F{src, (int)N}, Fi{img, (int)N}, G{fsc, (int)N};
    pair_tractions_hs(F, Fi, G, R, nu, k, two_mu, lam, ts, td);
}

template <bool kWrite32>
__global__ void __launch_bounds__(kHsThreads, 2)
assemble_hs_kernel(const Tile *__restrict__ tiles, const TileHs *__restrict__ hs, int ts,
                   const double *__restrict__ src, const double *__restrict__ recv, const double *__restrict__ img,
                   const double *__restrict__ fsc, int64_t N, int64_t row0, int64_t row1, int nr, SegMat mat, double nu,
                   double k, double two_mu, double lam, double *__restrict__ K64, float *__restrict__ K32)
{
    extern __shared__ double s_buf[];
    __shared__ double s_rcv[kHsRecv * kRecvStride];
    const int t = threadIdx.x;
    const Tile &T = tiles[blockIdx.x];
    const int ne = T.ne;
    const int64_t i0 = row0 + (int64_t)blockIdx.y * nr;
    const int nrec = (int)((row1 - i0) < nr ? (row1 - i0) : nr);
    for (int q = t; q < nrec * kRecvStride; q += kHsThreads) s_rcv[q] = recv[i0 * kRecvStride + q];
    const int batch = min(nrec, kHsSmem / (int)sizeof(double) / (ne * kHsMatD));
    const int64_t j0 = (int64_t)blockIdx.x * ts, ld = 2 * N;
    const int nt = (int)((N - j0) < ts ? (N - j0) : ts);
    for (int b0 = 0; b0 < nrec; b0 += batch) {
        const int nb = min(batch, nrec - b0);
        __syncthreads();   // the receivers are in; the last batch's readers are done
        for (int q = t; q < nb * ne; q += kHsThreads) {
            const int r = q / ne, e = q - r * ne;
            const double *R = s_rcv + (b0 + r) * kRecvStride;
            const TileEdge ed = T.edge[e];
            const double *A = T.vert[ed.a], *B = T.vert[ed.b];
            double *o = s_buf + q * kHsMatD;
            double M[9];
            seg_matrix(seg_terms(seg_vertex(R, A[0], A[1], -A[2]), seg_vertex(R, B[0], B[1], -B[2]), ed.L, ed.iL,
                                 ed.near2, mat.kap), mat.kap, mat.ci, M);
#pragma unroll
            for (int c = 0; c < 9; ++c) o[9 + c] = M[c];
            seg_matrix(seg_terms(seg_vertex(R, A[0], A[1], A[2]), seg_vertex(R, B[0], B[1], B[2]), ed.L, ed.iL,
                                 ed.near2, mat.kap), mat.kap, mat.ci, M);
            fsc_matrix(TileSide{&hs[blockIdx.x].f[0][e]}, R, nu, two_mu, lam, M);
#pragma unroll
            for (int c = 0; c < 9; ++c) o[c] = M[c];
        }
        __syncthreads();
        for (int q = t; q < nt; q += kHsThreads) {
            const int64_t j = T.id[q];
            const TileTri tri = T.tri[q];
            const bool surface = fsc[kFscSurface * N + j] != 0.0;
            for (int r = 0; r < nb; ++r) {
                const double *R = s_rcv + (b0 + r) * kRecvStride, *Mr = s_buf + r * ne * kHsMatD;
                double ts3[3] = {0.0, 0.0, 0.0}, td3[3] = {0.0, 0.0, 0.0};
#pragma unroll
                for (int p = 0; p < 2; ++p) {   // the edges with the correction, the image
                    const double *tab = p ? img : src;
                    double vs[3], vd[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        vs[a] = mat.scale * (R[3 + 3 * a] * tab[F_SX * N + j] + R[4 + 3 * a] * tab[F_SY * N + j]);
                        vd[a] = mat.scale * (R[3 + 3 * a] * tab[F_DX * N + j] + R[4 + 3 * a] * tab[F_DY * N + j] +
                                             R[5 + 3 * a] * tab[F_DZ * N + j]);
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int a = 0; a < 3; ++a) {
                            double m = 0.0;
#pragma unroll
                            for (int v = 0; v < 3; ++v)
                                m += flip_sign(Mr[(tri.e[v] & 0x7fff) * kHsMatD + 9 * p + 3 * c + a],
                                               (unsigned)(tri.e[v] & 0x8000) << 16);
                            ts3[c] += m * vs[a];
                            td3[c] += m * vd[a];
                        }
                }
                if (surface || seg_bad(ts3[0]))
                    pair_angular_hs(src + j, img + j, fsc + j, N, R, nu, k, two_mu, lam, ts3, td3);
                const int64_t row = 3 * (i0 + b0 + r - row0);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    *reinterpret_cast<double2 *>(K64 + (row + c) * ld + 2 * j) = make_double2(ts3[c], td3[c]);
                    if (kWrite32)
                        *reinterpret_cast<float2 *>(K32 + (row + c) * ld + 2 * j) =
                            make_float2(d2f_rn_bits(ts3[c]), d2f_rn_bits(td3[c]));
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Point kernels (host-pointer calls): strain and stress of n pairs -- one
// source at n receivers (kMany = false, records by value), or n sources at one
// receiver (kMany = true, the thread sets its source up).  The calls are short:
// what counts is the chain of FP64 latency of one pair (a half-space pair by
// one thread: ~200 us), so a pair's parts are shared out over the warps of a
// block of 32 pairs: half space -- three warps with a side of the free-surface
// correction each, a fourth with the main and the image dislocation; full space
// -- a warp per angular dislocation.  The parts are added in order through
// shared memory, and the 12 results per pair stored as one contiguous piece.
struct PointArgs {
    const double *A, *B, *C;      // receivers X, Y, Z, or the sources' vertices [n][3]
    double X, Y, Z;               // the one receiver (kMany)
    int64_t n;
    double bx, by, bz, mu, lam, nu, k;
    double *stress, *strain;      // [n][6]
};
constexpr int kPointPairs = 32;

template <bool kMany>
struct PointPair {
    double a[3], b[3], c[3], x, y, z;
    __device__ PointPair(const PointArgs &P, int64_t i)
    {
        if (kMany) {
            for (int q = 0; q < 3; ++q) { a[q] = P.A[3 * i + q]; b[q] = P.B[3 * i + q]; c[q] = P.C[3 * i + q]; }
            x = P.X; y = P.Y; z = P.Z;
        } else {
            x = P.A[i]; y = P.B[i]; z = P.C[i];
        }
    }
};

// The parts' sum e of pair t (thread t of the first warp) to the outputs; all
// threads of the block.
__device__ __forceinline__ void store_points(const PointArgs &P, int64_t i0, const double e[6], double (*out)[kPointPairs][6])
{
    const int t = threadIdx.x;
    if (t < kPointPairs) {
        double s[6];
        hooke(e, P.mu, P.lam, s);
        for (int q = 0; q < 6; ++q) { out[0][t][q] = s[q]; out[1][t][q] = e[q]; }
    }
    __syncthreads();
    const int n = 6 * (int)min((int64_t)kPointPairs, P.n - i0);
    for (int q = t; q < n; q += blockDim.x) {
        P.stress[6 * i0 + q] = (&out[0][0][0])[q];
        P.strain[6 * i0 + q] = (&out[1][0][0])[q];
    }
}

template <bool kMany>
__global__ void __launch_bounds__(128) points_hs_kernel(SrcVal s, SrcVal si, FscVal g, PointArgs P)
{
    __shared__ double part[5][kPointPairs][6], out[2][kPointPairs][6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * kPointPairs, i = i0 + lane;
    if (i < P.n) {
        const PointPair<kMany> p(P, i);
        if (w < 3) {
            double f[S_COUNT];
            if (kMany) setup_fsc_side(p.a, p.b, p.c, w, f, 1);
            point_strain_side(ValSrc{kMany ? f : g.f + w * S_COUNT}, p.x, p.y, p.z, P.bx, P.by, P.bz, P.nu, part[w][lane]);
        } else {
            for (int q = 0; q < 2; ++q) {
                double f[kSrcStride];
                const double sg = q ? -1.0 : 1.0;
                if (kMany) {
                    const double a[3] = {p.a[0], p.a[1], sg * p.a[2]}, b[3] = {p.b[0], p.b[1], sg * p.b[2]},
                                 c[3] = {p.c[0], p.c[1], sg * p.c[2]};
                    setup_source<false>(a, b, c, f, 1);
                }
                point_strain_full(ValSrc{kMany ? f : (q ? si.f : s.f)}, p.x, p.y, p.z, P.bx, P.by, P.bz, P.nu, P.k,
                                  part[3 + q][lane]);
            }
            image_signs(kMany ? fsc_surface(p.a, p.b, p.c) : g.f[kFscSurface], part[4][lane]);
        }
    }
    __syncthreads();
    double e[6];
    if (threadIdx.x < kPointPairs && i < P.n)
        for (int q = 0; q < 6; ++q)
            e[q] = part[3][lane][q] + ((part[0][lane][q] + part[1][lane][q] + part[2][lane][q]) + part[4][lane][q]);
    store_points(P, i0, e, out);
}

// W warps per 32 pairs: 3 (a vertex each) or 1.
template <bool kMany, int W>
__global__ void __launch_bounds__(32 * W) points_full_kernel(SrcVal s, PointArgs P)
{
    __shared__ double part[W][kPointPairs][6], out[2][kPointPairs][6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * kPointPairs, i = i0 + lane;
    double f[kSrcStride];
    const ValSrc F{kMany ? f : s.f};
    double E[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    if (i < P.n) {
        const PointPair<kMany> p(P, i);
        if (kMany) setup_source<false>(p.a, p.b, p.c, f, 1);
        double x, y, z;
        tdcs_point(F, p.x, p.y, p.z, x, y, z);
        const int m = tdcs_mode(F, x, y, z);
        if (m != 0)
            for (int v = W > 1 ? w : 0; v < (W > 1 ? w + 1 : 3); ++v)
                tdcs_vertex_general(F, m, v, x, y, z, P.bx, P.by, P.bz, P.nu, P.k, E);
        for (int q = 0; q < 6; ++q) part[w][lane][q] = E[q];
    }
    __syncthreads();
    double e[6];
    if (threadIdx.x < kPointPairs && i < P.n) {
        for (int q = 0; q < 6; ++q) {
            E[q] = part[0][lane][q];
            for (int v = 1; v < W; ++v) E[q] += part[v][lane][q];
        }
        tdcs_to_efcs(F, E, e);
    }
    store_points(P, i0, e, out);
}

// A source per thread costs its set-up once more for every warp that shares
// the pair: beyond this many pairs (the SMs hold their warps) one warp takes
// all three vertices (40,000 sources: 282 us by three warps, 184 us by one).
constexpr size_t kPointShare = 4096;

template <bool kMany>
static void launch_points_full(const SrcVal &s, const PointArgs &P, size_t n, cudaStream_t st)
{
    const unsigned blocks = (unsigned)((n + kPointPairs - 1) / kPointPairs);
    if constexpr (kMany) {
        if (n > kPointShare) {
            points_full_kernel<true, 1><<<blocks, 32, 0, st>>>(s, P);
            return;
        }
    }
    points_full_kernel<kMany, 3><<<blocks, 96, 0, st>>>(s, P);
}

static inline double poisson(double mu, double lam) { return 1.0 / (1.0 + lam / mu) / 2.0; }
static inline double kfac(double nu) { return 1.0 / (8.0 * kPi * (1.0 - nu)); }

// ---------------------------------------------------------------------------
// host-pointer context: one stream, one growing device buffer and one bounded
// page-locked buffer per host thread, given back when the thread ends
struct HostCtx {
    int device = -1;
    cudaStream_t stream = nullptr;
    double *buf = nullptr;
    size_t cap = 0;   // doubles
    double *pin = nullptr, *pin_dev = nullptr;   // host and device address
    void drop()
    {
        if (device < 0) return;
        if (stream) cudaStreamDestroy(stream);
        if (buf) cudaFree(buf);
        if (pin) cudaFreeHost(pin);
        (void)cudaGetLastError();
        device = -1;
        stream = nullptr;
        buf = pin = pin_dev = nullptr;
        cap = 0;
    }
    ~HostCtx() { drop(); }
};
static thread_local HostCtx g_ctx;

// Calls of up to kPinDoubles doubles in and out go through page-locked memory
// that the kernel reads and writes itself: one launch and one wait, where five
// copies of a few KB each cost more than the kernel (64 points: 61 -> 44 us a
// call, 4,000: 128 -> 106 us; 12,000 sources: 295 -> 351 us).  Above, the copies' own rate counts.
constexpr size_t kPinDoubles = 1 << 16;

static int host_ctx(size_t need_doubles, bool *pinned, HostCtx **out)
{
    int dev = 0;
    PQ3D_CUDA_TRY(cudaGetDevice(&dev));
    HostCtx &c = g_ctx;
    if (c.device != dev) {
        c.drop();
        PQ3D_CUDA_TRY(cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking));
        c.device = dev;
    }
    *out = &c;
    *pinned = need_doubles <= kPinDoubles;
    if (*pinned) {
        if (!c.pin) {
            PQ3D_CUDA_TRY(cudaHostAlloc(&c.pin, kPinDoubles * sizeof(double), cudaHostAllocMapped));
            void *d = nullptr;
            PQ3D_CUDA_TRY(cudaHostGetDevicePointer(&d, c.pin, 0));
            c.pin_dev = (double *)d;
        }
        return PQ3D_OK;
    }
    if (c.cap < need_doubles) {
        if (c.buf) cudaFree(c.buf);
        c.buf = nullptr;
        c.cap = 0;
        size_t cap = std::max<size_t>(need_doubles, 1 << 16);
        PQ3D_CUDA_TRY(cudaMalloc(&c.buf, cap * sizeof(double)));
        c.cap = cap;
    }
    return PQ3D_OK;
}

// n doubles into the call's buffer at offset `at` (doubles); the address the kernel reads
static int put(HostCtx *c, bool pinned, size_t at, const double *src, size_t n)
{
    if (pinned) memcpy(c->pin + at, src, n * sizeof(double));
    else PQ3D_CUDA_TRY(cudaMemcpyAsync(c->buf + at, src, n * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    return PQ3D_OK;
}

// the two results of n doubles each from offset `at`, once the kernel is done
static int take(HostCtx *c, bool pinned, size_t at, size_t n, double *stress, double *strain)
{
    if (!pinned) {
        PQ3D_CUDA_TRY(cudaMemcpyAsync(stress, c->buf + at, n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        PQ3D_CUDA_TRY(cudaMemcpyAsync(strain, c->buf + at + n, n * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    }
    PQ3D_CUDA_TRY(cudaStreamSynchronize(c->stream));
    if (pinned) {
        memcpy(stress, c->pin + at, n * sizeof(double));
        memcpy(strain, c->pin + at + n, n * sizeof(double));
    }
    return PQ3D_OK;
}

static void nan_fill(double *p, size_t n)
{
    if (!p) return;
    for (size_t i = 0; i < n; ++i) p[i] = NAN;
}

// The reference prints this and carries on (src/TDstressFS_C.cpp:1949-1953).
static void warn_halfspace_z(const double *X, const double *Y, const double *Z, size_t n, const double *P1,
                             const double *P2, const double *P3)
{
    (void)X; (void)Y;
    bool bad = (P1 && P1[2] > 0.0) || (P2 && P2[2] > 0.0) || (P3 && P3[2] > 0.0);
    for (size_t i = 0; i < n && !bad; ++i) bad = Z[i] > 0.0;
    if (bad) fprintf(stdout, "Half-space solution: Z coordinates must be negative!\n");
}

static int points_one_source(const double *X, const double *Y, const double *Z, size_t n, const double *P1,
                             const double *P2, const double *P3, double Ss, double Ds, double Ts, double mu,
                             double lam, bool half, double *stress, double *strain)
{
    clear_error();
    if (n == 0) return PQ3D_OK;
    PQ3D_REQUIRE(X && Y && Z && P1 && P2 && P3 && stress && strain, "TDstressFS_C: null pointer");
    if (half) warn_halfspace_z(X, Y, Z, n, P1, P2, P3);
    HostCtx *c;
    bool pinned;
    int rc = host_ctx(15 * n, &pinned, &c);
    const double *in[3] = {X, Y, Z};
    for (int q = 0; q < 3 && !rc; ++q) rc = put(c, pinned, q * n, in[q], n);
    if (rc) return rc;
    double *dX = pinned ? c->pin_dev : c->buf, *dY = dX + n, *dZ = dY + n, *dS = dZ + n, *dE = dS + 6 * n;
    SrcVal s, si;
    FscVal g;
    double a[3] = {P1[0], P1[1], P1[2]}, b[3] = {P2[0], P2[1], P2[2]}, cc[3] = {P3[0], P3[1], P3[2]};
    setup_source(a, b, cc, s.f, 1);
    const double nu = poisson(mu, lam);
    const PointArgs P{dX, dY, dZ, 0.0, 0.0, 0.0, (int64_t)n, Ts, Ss, Ds, mu, lam, nu, kfac(nu), dS, dE};
    const unsigned blocks = (unsigned)((n + kPointPairs - 1) / kPointPairs);
    if (half) {
        double am[3] = {a[0], a[1], -a[2]}, bm[3] = {b[0], b[1], -b[2]}, cm[3] = {cc[0], cc[1], -cc[2]};
        setup_source(am, bm, cm, si.f, 1);
        setup_fsc(a, b, cc, g.f, 1);
        points_hs_kernel<false><<<blocks, 128, 0, c->stream>>>(s, si, g, P);
    } else {
        launch_points_full<false>(s, P, n, c->stream);
    }
    PQ3D_CUDA_TRY(cudaGetLastError());
    return take(c, pinned, 3 * n, 6 * n, stress, strain);
}

static int point_many_sources(double x, double y, double z, const double *P1, const double *P2, const double *P3,
                              size_t ns, double Ss, double Ds, double Ts, double mu, double lam, bool half,
                              double *stress, double *strain)
{
    clear_error();
    if (ns == 0) return PQ3D_OK;
    PQ3D_REQUIRE(P1 && P2 && P3 && stress && strain, "TDstressEachSourceAtReceiver_C: null pointer");
    if (half) warn_halfspace_z(&x, &y, &z, 1, nullptr, nullptr, nullptr);
    HostCtx *c;
    bool pinned;
    int rc = host_ctx(21 * ns, &pinned, &c);
    const double *in[3] = {P1, P2, P3};
    for (int q = 0; q < 3 && !rc; ++q) rc = put(c, pinned, 3 * q * ns, in[q], 3 * ns);
    if (rc) return rc;
    double *d1 = pinned ? c->pin_dev : c->buf, *d2 = d1 + 3 * ns, *d3 = d2 + 3 * ns, *dS = d3 + 3 * ns, *dE = dS + 6 * ns;
    const double nu = poisson(mu, lam);
    const PointArgs P{d1, d2, d3, x, y, z, (int64_t)ns, Ts, Ss, Ds, mu, lam, nu, kfac(nu), dS, dE};
    const unsigned blocks = (unsigned)((ns + kPointPairs - 1) / kPointPairs);
    if (half) points_hs_kernel<true><<<blocks, 128, 0, c->stream>>>(SrcVal(), SrcVal(), FscVal(), P);
    else launch_points_full<true>(SrcVal(), P, ns, c->stream);
    PQ3D_CUDA_TRY(cudaGetLastError());
    return take(c, pinned, 9 * ns, 6 * ns, stress, strain);
}

// Workspace: source table [kSrcStride][N], receiver table [N][kRecvStride],
// for the half space the image table [kImgStride][N] and the side table
// [kFscStride][N], then (from an even offset) the tiles, and for the half space
// their edges' surface records, last the triangles' order (N + 1 integers).
static size_t tables_doubles(int64_t N, bool half)
{
    return (size_t)N * (kSrcStride + kRecvStride + (half ? kImgStride + kFscStride : 0));
}
static size_t tiles_offset(int64_t N, bool half) { return (tables_doubles(N, half) + 1) & ~(size_t)1; }
static size_t order_offset(int64_t N, bool half)
{
    return tiles_offset(N, half) + (size_t)tile_count(N, half) * (kSegDoubles + (half ? kHsDoubles : 0));
}
static size_t ws_bytes(int64_t N, bool half)
{
    return order_offset(N, half) * sizeof(double) + ((size_t)N / 2 + 1) * sizeof(double);
}

static void setup_elements(const double *nodes, const int64_t *tris, int64_t N, double *src, double *recv,
                           cudaStream_t st)
{
    const unsigned nb = (unsigned)((N + 127) / 128);
    setup_elements_kernel<<<2 * nb, 128, 0, st>>>(nodes, tris, N, nb, src, recv);
}

// Receivers per block: the grid's tail costs up to one block's time, so the
// count with the fewest receivers on a slot's path wins (one receiver a block on
// the smallest meshes); one extra receiver stands for a block's start.
static int seg_receivers(int most, int64_t tiles, int64_t rows, int64_t slots)
{
    int best = most;
    int64_t cost = INT64_MAX;
    for (int nr = most; nr >= 1; --nr) {
        const int64_t waves = (tiles * ((rows + nr - 1) / nr) + slots - 1) / slots;
        const int64_t c = waves * (nr + 1);
        if (c < cost) { cost = c; best = nr; }
    }
    return best;
}

static int assemble_rows(const double *nodes, const int64_t *tris, int64_t N, int64_t row0, int64_t row1, double mu,
                         double lam, double *K64, float *K32, double *ws, bool do_setup, cudaStream_t st,
                         bool half = false, bool to_host = false)
{
    double *src = ws, *recv = src + (size_t)kSrcStride * N;
    double *img = recv + (size_t)kRecvStride * N, *fsc = img + (size_t)kImgStride * N;
    Tile *tiles = (Tile *)(ws + tiles_offset(N, half));
    TileHs *hs = half ? (TileHs *)(tiles + tile_count(N, true)) : nullptr;
    const int ts = tile_size(N, half);
    const int64_t nt = (N + ts - 1) / ts;
    if (do_setup) {
        const int th = 128;
        setup_elements(nodes, tris, N, src, recv, st);
        if (half) setup_hs_kernel<<<(unsigned)((N + th - 1) / th), th, 0, st>>>(nodes, tris, N, img, fsc);
        setup_tiles_kernel<<<(unsigned)nt, kTileMax, 0, st>>>(nodes, tris, N, ts, nullptr, tiles, hs);
        const int64_t rows = row1 > row0 ? row1 - row0 : N;   // no rows: they follow, all of them
        if (rows * N >= (half ? kOrderPairsHs : kOrderPairs) && (half || !to_host)) {
            int32_t *order = (int32_t *)(ws + order_offset(N, half));
            order_tiles_kernel<<<1, kOrderThreads, 0, st>>>(recv, N, nt, tiles, order);
            setup_tiles_kernel<<<(unsigned)nt, kTileMax, 0, st>>>(nodes, tris, N, ts, order, tiles, hs);
        }
        PQ3D_CUDA_TRY(cudaGetLastError());
    }
    if (row0 == row1) return PQ3D_OK;
    int dev, sms;
    PQ3D_CUDA_TRY(cudaGetDevice(&dev));
    PQ3D_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const double nu = poisson(mu, lam);
    const SegMat mat = seg_material(nu, 2.0 * mu, lam);
    const int nr = seg_receivers(half ? kHsRecv : kSegRecv, nt, row1 - row0, 2 * (int64_t)sms);
    const dim3 grid((unsigned)nt, (unsigned)((row1 - row0 + nr - 1) / nr));
    if (half) {
        const auto kernel = K32 ? assemble_hs_kernel<true> : assemble_hs_kernel<false>;
        PQ3D_CUDA_TRY(allow_smem(kernel, kHsSmem));
        kernel<<<grid, kHsThreads, kHsSmem, st>>>(tiles, hs, ts, src, recv, img, fsc, N, row0, row1, nr, mat, nu,
                                                  kfac(nu), 2.0 * mu, lam, K64, K32);
    } else {
        const auto kernel = K32 ? assemble_seg_kernel<true> : assemble_seg_kernel<false>;
        PQ3D_CUDA_TRY(allow_smem(kernel, kSegSmem));
        kernel<<<grid, kSegThreads, kSegSmem, st>>>(tiles, ts, src, recv, N, row0, row1, nr, mat, nu, kfac(nu), 2.0 * mu,
                                                    lam, K64, K32);
    }
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}

// ---------------------------------------------------------------------------
// Fixed scratch for pq3d_assemble_dense_noalloc: the source and receiver
// tables, the tiles and their order of one call for up to kNoAllocMaxN elements, 19.4 MB
// held by every GPU that loads this library.
constexpr int64_t kNoAllocMaxN = 32768;
static __device__ __align__(256) double g_noalloc_scratch[(size_t)(kSrcStride + kRecvStride) * kNoAllocMaxN +
                                                          (size_t)(kNoAllocMaxN / kTileMax) * kSegDoubles +
                                                          (size_t)kNoAllocMaxN / 2 + 1];

// Device address of the fixed scratch on the current device, looked up with
// that device current on every call (cheap): a cached address would go stale
// if the device were reset or its primary context recreated between calls.
static int noalloc_scratch(double **out)
{
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p)
        return set_error(PQ3D_ERR_CUDA, "pq3d_assemble_dense_noalloc: cudaGetSymbolAddress failed: %s",
                         cudaGetErrorString(e));
    *out = (double *)p;
    return PQ3D_OK;
}

}  // namespace gf
}  // namespace pq3d

using namespace pq3d;
using namespace pq3d::gf;

extern "C" void TDstressFS_C(const double *X, const double *Y, const double *Z, size_t n, const double *P1,
                             const double *P2, const double *P3, double Ss, double Ds, double Ts, double mu,
                             double lambda_, bool jud_halfspace, double *stress, double *strain)
{
    int rc = points_one_source(X, Y, Z, n, P1, P2, P3, Ss, Ds, Ts, mu, lambda_, jud_halfspace, stress, strain);
    if (rc != PQ3D_OK) {
        fprintf(stderr, "pq3d: %s\n", pq3d_last_error());
        nan_fill(stress, 6 * n);
        nan_fill(strain, 6 * n);
    }
}

extern "C" void TDstressEachSourceAtReceiver_C(double x, double y, double z, const double *P1_flat,
                                               const double *P2_flat, const double *P3_flat, size_t n_sources,
                                               double Ss, double Ds, double Ts, double mu, double lambda_,
                                               bool jud_halfspace, double *stress_out, double *strain_out)
{
    int rc = point_many_sources(x, y, z, P1_flat, P2_flat, P3_flat, n_sources, Ss, Ds, Ts, mu, lambda_,
                                jud_halfspace, stress_out, strain_out);
    if (rc != PQ3D_OK) {
        fprintf(stderr, "pq3d: %s\n", pq3d_last_error());
        nan_fill(stress_out, 6 * n_sources);
        nan_fill(strain_out, 6 * n_sources);
    }
}

extern "C" void TDstressFS_C1(const double *X, const double *Y, const double *Z, size_t n, const double *P1,
                              const double *P2, const double *P3, double Ss, double Ds, double Ts, double mu,
                              double lambda_, double *Sxx, double *Syy, double *Szz, double *Sxy, double *Sxz,
                              double *Syz, double *Exx, double *Eyy, double *Ezz, double *Exy, double *Exz,
                              double *Eyz)
{
    std::vector<double> s(6 * n), e(6 * n);
    int rc = points_one_source(X, Y, Z, n, P1, P2, P3, Ss, Ds, Ts, mu, lambda_, false, s.data(), e.data());
    if (rc != PQ3D_OK) {
        fprintf(stderr, "pq3d: %s\n", pq3d_last_error());
        std::fill(s.begin(), s.end(), NAN);
        std::fill(e.begin(), e.end(), NAN);
    }
    double *S[6] = {Sxx, Syy, Szz, Sxy, Sxz, Syz}, *E[6] = {Exx, Eyy, Ezz, Exy, Exz, Eyz};
    for (size_t i = 0; i < n; ++i)
        for (int c = 0; c < 6; ++c) {
            S[c][i] = s[6 * i + c];
            E[c][i] = e[6 * i + c];
        }
}

// the size that serves both full- and half-space assemblies
extern "C" size_t pq3d_gf_workspace_bytes(int64_t N)
{
    return N > 0 ? std::max(ws_bytes(N, true), ws_bytes(N, false)) : 0;
}

extern "C" int pq3d_assemble_dense(const double *nodes, const int64_t *tris, int64_t N, int64_t row0, int64_t row1,
                                   double mu, double lambda_, int halfspace, double *K64, float *K32, void *workspace,
                                   size_t workspace_bytes, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(N > 0 && row0 >= 0 && row1 <= N && row0 <= row1, "pq3d_assemble_dense: bad sizes");
    PQ3D_REQUIRE(nodes && tris && K64 && workspace, "pq3d_assemble_dense: null pointer");
    PQ3D_REQUIRE(aligned16(K64) && (!K32 || ((uintptr_t)K32 & 7u) == 0) && aligned16(workspace),
                 "pq3d_assemble_dense: K64/workspace must be 16-byte aligned, K32 8-byte aligned");
    PQ3D_REQUIRE(workspace_bytes >= ws_bytes(N, halfspace != 0), "pq3d_assemble_dense: workspace too small (%zu < %zu)",
                 workspace_bytes, ws_bytes(N, halfspace != 0));
    if (row0 == row1) return PQ3D_OK;
    return assemble_rows(nodes, tris, N, row0, row1, mu, lambda_, K64, K32, (double *)workspace, true,
                         (cudaStream_t)stream, halfspace != 0);
}

// Device address of page-locked host memory mapped into the device address
// space (cudaHostAlloc / cudaHostRegister under unified addressing), else NULL.
static void *mapped_device_ptr(void *host)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return (a.type == cudaMemoryTypeHost) ? a.devicePointer : nullptr;
}

// Output already in mapped page-locked host memory: the assembly kernel stores
// straight into it, one launch over all rows, no staging buffers and no separate
// copies.  In the mesh's own order a warp's stores are 512 contiguous bytes, which
// the host link takes as fast as they come (N = 20,040: 168 ms, 115 GB/s; 170 ms,
// 170 GB/s, with the FP32 copy).
static int assemble_host_direct(const double *nodes_host, int64_t n_nodes, const int64_t *tris_host, int64_t N,
                                double mu, double lambda_, bool half, double *dK64, float *dK32)
{
    double *d_nodes = nullptr, *d_ws = nullptr;
    int64_t *d_tris = nullptr;
    cudaStream_t st = nullptr;
    int rc = PQ3D_OK;
#define PQ3D_D_TRY(call)                                                                              \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) {                                                                      \
            rc = set_error(PQ3D_ERR_CUDA, "pq3d_assemble_dense_host: %s: %s", #call, cudaGetErrorString(e_)); \
            goto done;                                                                                \
        }                                                                                             \
    } while (0)
    PQ3D_D_TRY(cudaMalloc(&d_nodes, 3 * n_nodes * sizeof(double)));
    PQ3D_D_TRY(cudaMalloc(&d_tris, 3 * N * sizeof(int64_t)));
    PQ3D_D_TRY(cudaMalloc(&d_ws, ws_bytes(N, half)));
    PQ3D_D_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    PQ3D_D_TRY(cudaMemcpyAsync(d_nodes, nodes_host, 3 * n_nodes * sizeof(double), cudaMemcpyHostToDevice, st));
    PQ3D_D_TRY(cudaMemcpyAsync(d_tris, tris_host, 3 * N * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    rc = assemble_rows(d_nodes, d_tris, N, 0, N, mu, lambda_, dK64, dK32, d_ws, true, st, half, true);
    if (rc) goto done;
    PQ3D_D_TRY(cudaStreamSynchronize(st));
done:
#undef PQ3D_D_TRY
    if (st) { cudaStreamSynchronize(st); cudaStreamDestroy(st); }
    cudaFree(d_nodes);
    cudaFree(d_tris);
    cudaFree(d_ws);
    return rc;
}

extern "C" int pq3d_assemble_dense_host(const double *nodes_host, int64_t n_nodes, const int64_t *tris_host,
                                        int64_t N, double mu, double lambda_, int halfspace, double *K64_host,
                                        float *K32_host)
{
    clear_error();
    PQ3D_REQUIRE(N > 0 && n_nodes > 0 && nodes_host && tris_host && K64_host, "pq3d_assemble_dense_host: bad args");
    const bool half = halfspace != 0;
    {
        double *dK64 = (double *)mapped_device_ptr(K64_host);
        float *dK32 = K32_host ? (float *)mapped_device_ptr(K32_host) : nullptr;
        if (dK64 && aligned16(dK64) && (!K32_host || (dK32 && ((uintptr_t)dK32 & 7u) == 0)))
            return assemble_host_direct(nodes_host, n_nodes, tris_host, N, mu, lambda_, half, dK64, dK32);
    }
    const size_t ld = 2 * (size_t)N;
    // rows per block: about 256 MB of FP64 output per block
    int64_t rb = std::max<int64_t>(kSegRecv,
                                   ((int64_t)(256u << 20) / (int64_t)(3 * ld * sizeof(double))) / kSegRecv * kSegRecv);
    rb = std::min<int64_t>(rb, N);
    double *d_nodes = nullptr, *d_ws = nullptr, *d_K64[2] = {nullptr, nullptr};
    float *d_K32[2] = {nullptr, nullptr};
    int64_t *d_tris = nullptr;
    cudaStream_t st[2] = {nullptr, nullptr};
    cudaEvent_t setup_done = nullptr;
    int rc = PQ3D_OK;
#define PQ3D_H_TRY(call)                                                                              \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) {                                                                      \
            rc = set_error(PQ3D_ERR_CUDA, "pq3d_assemble_dense_host: %s: %s", #call, cudaGetErrorString(e_)); \
            goto done;                                                                                \
        }                                                                                             \
    } while (0)
    PQ3D_H_TRY(cudaMalloc(&d_nodes, 3 * n_nodes * sizeof(double)));
    PQ3D_H_TRY(cudaMalloc(&d_tris, 3 * N * sizeof(int64_t)));
    PQ3D_H_TRY(cudaMalloc(&d_ws, ws_bytes(N, half)));
    for (int b = 0; b < 2; ++b) {
        PQ3D_H_TRY(cudaMalloc(&d_K64[b], 3 * rb * ld * sizeof(double)));
        if (K32_host) PQ3D_H_TRY(cudaMalloc(&d_K32[b], 3 * rb * ld * sizeof(float)));
        PQ3D_H_TRY(cudaStreamCreateWithFlags(&st[b], cudaStreamNonBlocking));
    }
    PQ3D_H_TRY(cudaEventCreateWithFlags(&setup_done, cudaEventDisableTiming));
    PQ3D_H_TRY(cudaMemcpyAsync(d_nodes, nodes_host, 3 * n_nodes * sizeof(double), cudaMemcpyHostToDevice, st[0]));
    PQ3D_H_TRY(cudaMemcpyAsync(d_tris, tris_host, 3 * N * sizeof(int64_t), cudaMemcpyHostToDevice, st[0]));
    {
        // the tables, with no rows assembled yet
        rc = assemble_rows(d_nodes, d_tris, N, 0, 0, mu, lambda_, nullptr, nullptr, d_ws, true, st[0], half);
        if (rc) goto done;
        PQ3D_H_TRY(cudaEventRecord(setup_done, st[0]));
        PQ3D_H_TRY(cudaStreamWaitEvent(st[1], setup_done, 0));
        int blk = 0;
        for (int64_t r0 = 0; r0 < N; r0 += rb, ++blk) {
            const int b = blk & 1;
            const int64_t r1 = std::min<int64_t>(N, r0 + rb);
            rc = assemble_rows(d_nodes, d_tris, N, r0, r1, mu, lambda_, d_K64[b], d_K32[b], d_ws, false, st[b], half);
            if (rc) goto done;
            PQ3D_H_TRY(cudaMemcpyAsync(K64_host + 3 * r0 * ld, d_K64[b], 3 * (r1 - r0) * ld * sizeof(double),
                                       cudaMemcpyDeviceToHost, st[b]));
            if (K32_host)
                PQ3D_H_TRY(cudaMemcpyAsync(K32_host + 3 * r0 * ld, d_K32[b], 3 * (r1 - r0) * ld * sizeof(float),
                                           cudaMemcpyDeviceToHost, st[b]));
        }
        PQ3D_H_TRY(cudaStreamSynchronize(st[0]));
        PQ3D_H_TRY(cudaStreamSynchronize(st[1]));
    }
done:
#undef PQ3D_H_TRY
    for (int b = 0; b < 2; ++b) {
        if (st[b]) { cudaStreamSynchronize(st[b]); cudaStreamDestroy(st[b]); }
        cudaFree(d_K64[b]);
        cudaFree(d_K32[b]);
    }
    if (setup_done) cudaEventDestroy(setup_done);
    cudaFree(d_nodes);
    cudaFree(d_tris);
    cudaFree(d_ws);
    return rc;
}

extern "C" int pq3d_assemble_dense_noalloc(const double *nodes, const int64_t *tris, int64_t N, int64_t row0,
                                           int64_t row1, double mu, double lambda_, int halfspace, double *K64,
                                           float *K32, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(N > 0 && row0 >= 0 && row1 <= N && row0 <= row1, "pq3d_assemble_dense_noalloc: bad sizes");
    PQ3D_REQUIRE(N <= kNoAllocMaxN, "pq3d_assemble_dense_noalloc: N = %lld exceeds the fixed scratch limit of %lld "
                 "elements (use pq3d_assemble_dense with a caller-provided workspace)", (long long)N,
                 (long long)kNoAllocMaxN);
    PQ3D_REQUIRE(nodes && tris && K64, "pq3d_assemble_dense_noalloc: null pointer");
    PQ3D_REQUIRE(aligned16(K64) && (!K32 || ((uintptr_t)K32 & 7u) == 0),
                 "pq3d_assemble_dense_noalloc: K64 must be 16-byte aligned, K32 8-byte aligned");
    if (halfspace)
        return set_error(PQ3D_ERR_UNSUPPORTED, "pq3d_assemble_dense_noalloc: the fixed scratch holds the full-space "
                         "tables only; use pq3d_assemble_dense for the half-space");
    double *scratch = nullptr;
    int rc = noalloc_scratch(&scratch);
    if (rc) return rc;
    if (row0 == row1) return PQ3D_OK;
    // every table entry the assembly reads is rewritten by this call's set-up
    // kernels, so nothing has to be cleared between calls
    return assemble_rows(nodes, tris, N, row0, row1, mu, lambda_, K64, K32, scratch, true, (cudaStream_t)stream);
}

extern "C" size_t pq3d_gf_setup_bytes(int64_t N, int halfspace)
{
    return N > 0 ? tables_doubles(N, halfspace != 0) * sizeof(double) : 0;
}

extern "C" int pq3d_gf_setup(const double *nodes, const int64_t *tris, int64_t N, int halfspace, void *workspace,
                             size_t workspace_bytes, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(nodes && tris && workspace && N > 0, "pq3d_gf_setup: bad arguments");
    PQ3D_REQUIRE(workspace_bytes >= pq3d_gf_setup_bytes(N, halfspace) && aligned16(workspace),
                 "pq3d_gf_setup: workspace too small");
    double *src = (double *)workspace;
    double *recv = src + (size_t)kSrcStride * N;
    setup_elements(nodes, tris, N, src, recv, (cudaStream_t)stream);
    if (halfspace) {
        double *img = recv + (size_t)kRecvStride * N;
        setup_hs_kernel<<<(unsigned)((N + 127) / 128), 128, 0, (cudaStream_t)stream>>>(nodes, tris, N, img,
                                                                                     img + (size_t)kImgStride * N);
    }
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}
