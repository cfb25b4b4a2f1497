// H-matrix of the traction operator on the GPU: ACA compression of the
// admissible blocks, dense near-field blocks, and the product with B
// right-hand sides.
//
// Reference: src/Hmatrix.py -- partition 68-192 and 2077-2196 (restated on the
// host in pyquake3d_gb300/hmatrix.py), ACA 661-1344, product 1773-1866.
//
// Differences in method (stated):
//   * one ACA per block on the combined (3m x 2n) block of K (rows = receiver x
//     traction component, columns = source x slip direction), i.e. all six
//     reference operators at once, with partial pivoting and the relative
//     Frobenius stopping rule |u_k| |v_k| <= tol |S_k|_F (the reference runs one
//     ACA+ per slip direction, pivoting on the first component only, with an
//     absolute step tolerance and an unseeded random start);
//   * rows and columns are generated on the fly by the GF device math
//     (no host round trip per row), the first pivot row is row 0, ties in
//     argmax go to the smallest index -- deterministic;
//   * a block that has not converged at its rank cap is stored dense;
//   * factors and dense blocks are stored in FP32; products use FP32 FMAs
//     with the right-hand side split into FP32 hi + lo pieces (2 FMAs per
//     entry, FP32 sums over one block segment, FP64 beyond), accumulated per
//     output row in a fixed order (no atomics, the same result for a run alone
//     or in a batch).  The ACA tolerance (1e-4) dominates this rounding by
//     orders of magnitude.
//   * several right-hand sides share every loaded entry in groups of up to 8
//     runs (leaf_rows_runs_kernel, lowrank_T_runs_kernel); with few leaves they
//     go run by run.
// Index space: elements are renumbered so that every cluster is a contiguous
// range (perm[p] = element at position p); a block is a pair of ranges.
#include <math.h>

#include "common.cuh"
#include "gf_device.cuh"
#include "hs_device.cuh"

namespace pq3d {
namespace hm {

using namespace ::pq3d::gf;

struct GSrc {   // source fields from the global structure-of-arrays table
    const double *base;
    int64_t stride;
    __device__ __forceinline__ double operator()(int f) const { return __ldg(base + f * stride); }
};

constexpr int kThreads = 256;

// The six tractions of pair (receiver record R, source element j): full
// space, or half space (image record and free-surface side table).
template <bool kHalf>
struct PairGen {
    const double *src, *img, *fsc;
    int64_t N;
    double nu, kf, two_mu, lam;
    __device__ __forceinline__ void operator()(int64_t j, const double *R, double ts[3], double td[3]) const
    {
        if (kHalf)
            pair_tractions_hs(GSrc{src + j, N}, GSrc{img + j, N}, GSrc{fsc + j, N}, R, nu, kf, two_mu, lam, ts, td);
        else
            pair_tractions(GSrc{src + j, N}, R, nu, kf, two_mu, lam, ts, td);
    }
};

// ---------------------------------------------------------------------------
// ACA.  A block is worked on by a group of kAcaSmall threads (a quarter of a
// CTA), by a CTA, or by a cluster of kAcaCluster CTAs; each kind only meets at
// its own barriers.  The clusters are one launch, the rest another beside it
// (clusters alone leave the SMs of a GPC that make no eighth idle), let in once
// every cluster is on the chip: eight free SMs of a GPC hardly come about while
// single CTAs take them (beside one another from the start, N = 900, 198 blocks of up
// to 450 elements: 7.55 ms, 5.57 so; N = 12,100: 35.9 and 30.6 ms; 30,000, without
// clusters: 106 ms).
//
// Bound: the FP64 pipe -- per iteration n + m pair evaluations of 520
// operations, 2 k (M + Nc) multiply-adds for the residual row and column and
// as many for the k cross products.  One 256-thread CTA per block in block
// order kept the pipe 76 % busy while an SM had a block, but 49 % over the
// launch (N = 20,000: 83 ms): most threads idled at the pivot searches of the
// many blocks of 64 x 64 pairs, and the few largest blocks, a sixth of all
// pairs, ran on one SM each long after the others.  Hence the three kinds, the
// largest blocks first, 16 warps per SM and four barriers an iteration (the
// residual, its norm and its pivot in the loop that evaluates the pairs).
constexpr int kAcaThreads = 256;
constexpr int kAcaSmall = 64;     // (the barrier counts of AcaGroup::sync)
constexpr int kAcaGroups = kAcaThreads / kAcaSmall;
constexpr int kAcaCluster = 8;
constexpr int kAcaWarps = kAcaCluster * kAcaThreads / 32;
// A block with more elements (m + n) than the average share of a CTA per SM would
// end last on one CTA: it gets a cluster, from 256 elements on -- unless the blocks
// are few (three an SM) and the clusters more than the chip holds at once, so that
// their second round ends last (156 blocks, 24 of them of more than 256 elements:
// 5.0 ms with clusters, 3.4 ms on a CTA each; 426: 6.4 and 4.3).
// A small group is for blocks of at most kAcaSmallSide elements a side (four rounds
// of the group) and of at most the share of a group's slot: with few blocks (N =
// 3,600: 216) the SMs would idle while groups of 64 threads walk 256-element sides.
// (The group's width is the order of the norms' sums: the factors' values do not
// depend on it, their number only where the stopping rule is a matter of rounding.)
constexpr int kAcaSmallSide = 256;
constexpr int kAcaHugeMin = 256;

struct __align__(16) AcaSlot {
    long long v;    // bits of the largest |value| (signed order: -1.0, no candidate, lies below all)
    double s;
    int i, pad[3];
};

struct AcaGroup {
    int t, size, id;      // thread and threads of the group; barrier: 0 the cluster's, 1 .. 4 of the CTA
    AcaSlot *slot;        // [2][warps of the group], in turn: one barrier per reduction
    int turn;
    __device__ __forceinline__ void sync() const
    {
        // literal barrier ids: a register id makes the CTA hold all 16 barriers
        __syncwarp();
        if (id == 0)
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        else if (id == 1) asm volatile("barrier.sync 1, %0;" ::"r"(size) : "memory");
        else if (id == 2) asm volatile("barrier.sync 2, 64;" ::: "memory");
        else if (id == 3) asm volatile("barrier.sync 3, 64;" ::: "memory");
        else asm volatile("barrier.sync 4, 64;" ::: "memory");
    }
    static __device__ __forceinline__ void pick(long long &v, int &idx, long long ov, int oi)
    {
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    // the largest v >= 0 (or -1.0) with the smallest index on ties, and the
    // sum of s; every thread of the group gets both, in the same order of
    // operations.  The comparisons are integer ones (FP64 compares run on the
    // FP64 pipe).
    __device__ __forceinline__ void reduce(double value, int idx, double s, double &best, int &bidx, double &sum)
    {
        long long v = __double_as_longlong(value);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            s += __shfl_xor_sync(0xffffffffu, s, o);
            pick(v, idx, ov, oi);
        }
        const int w = t >> 5, lane = t & 31, nw = size >> 5;
        AcaSlot *buf = slot + (turn & 1) * nw;
        turn ^= 1;
        if (id != 0) {
            if (lane == 0) buf[w] = AcaSlot{v, s, idx, {0, 0, 0}};
        } else if (lane < kAcaCluster) {   // into this warp's slot of every CTA of the cluster
            uint32_t at = (uint32_t)__cvta_generic_to_shared(&buf[w]);
            asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(at) : "r"(lane));
            asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(at), "l"(v), "l"(__double_as_longlong(s))
                         : "memory");
            asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(at + 16), "r"(idx) : "memory");
        }
        sync();
        v = __double_as_longlong(-1.0);
        idx = 0x7fffffff;
        s = 0.0;
        for (int q = lane; q < nw; q += 32) {
            pick(v, idx, buf[q].v, buf[q].i);
            s += buf[q].s;
        }
        for (int o = min(nw, 32) >> 1; o > 0; o >>= 1) {
            const long long ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            s += __shfl_xor_sync(0xffffffffu, s, o);
            pick(v, idx, ov, oi);
        }
        best = __longlong_as_double(__shfl_sync(0xffffffffu, v, 0));
        bidx = __shfl_sync(0xffffffffu, idx, 0);
        sum = __shfl_sync(0xffffffffu, s, 0);
    }
};

// Work order: huge, large and small blocks, each kind by size class, the
// largest first (a counting sort over half octaves of m + n in one CTA; the
// order within a class does not matter).  split = {huge blocks, large blocks}.
constexpr int kAcaClasses = 64;
__global__ void __launch_bounds__(1024)
aca_order_kernel(const int64_t *__restrict__ blk, int nblocks, int sms, int32_t *__restrict__ order,
                 int32_t *__restrict__ split)
{
    __shared__ int count[3 * kAcaClasses], nhuge;
    __shared__ unsigned long long total;
    const int t = threadIdx.x;
    if (t < 3 * kAcaClasses) count[t] = 0;
    if (t == 0) { total = 0; nhuge = 0; }
    __syncthreads();
    auto side_m = [&](int b) { return blk[4 * b + 1] - blk[4 * b]; };
    auto side_n = [&](int b) { return blk[4 * b + 3] - blk[4 * b + 2]; };
    unsigned long long mine = 0;
    for (int b = t; b < nblocks; b += blockDim.x) mine += (unsigned long long)(side_m(b) + side_n(b));
    atomicAdd(&total, mine);
    __syncthreads();
    int64_t huge = max((int64_t)kAcaHugeMin, (int64_t)(total / (unsigned)sms));
    const int64_t small = (int64_t)(total / (unsigned)(sms * kAcaGroups));
    if (nblocks <= 3 * sms) {
        for (int b = t; b < nblocks; b += blockDim.x)
            if (side_m(b) + side_n(b) > huge) atomicAdd(&nhuge, 1);
        __syncthreads();
        if (nhuge > sms / kAcaCluster) huge = INT64_MAX;
    }
    auto cls = [&](int b) {
        const int64_t m = side_m(b), n = side_n(b);
        const int kind = m + n > huge ? 0 : (max(m, n) > kAcaSmallSide || m + n > small ? 1 : 2);
        return kind * kAcaClasses + kAcaClasses - 1 - min(kAcaClasses - 1, (int)(2.0f * log2f((float)(m + n))));
    };
    for (int b = t; b < nblocks; b += blockDim.x) atomicAdd(&count[cls(b)], 1);
    __syncthreads();
    if (t == 0) {
        int s = 0;
        for (int c = 0; c < 3 * kAcaClasses; ++c) {
            if (c == kAcaClasses) split[0] = s;
            if (c == 2 * kAcaClasses) split[1] = s - split[0];
            const int n = count[c];
            count[c] = s;
            s += n;
        }
    }
    __syncthreads();
    for (int b = t; b < nblocks; b += blockDim.x) order[atomicAdd(&count[cls(b)], 1)] = b;
}

// U: kcap x M (row l = u_l), V: kcap x Nc.  One CTA per SM: at 128 registers for
// two, the compiler contracts the pair's products differently, and the last
// terms of a block, 1e-4 of its size, carry such a change of 1e-16 into 1e-11 of
// the product (two CTAs: 102 instead of 110 ms at N = 30,000).
// clusters: this launch is one of clusters, for the huge blocks.
template <bool kHalf>
__global__ void __launch_bounds__(kAcaThreads, 1)
aca_kernel(bool clusters, PairGen<kHalf> gen, const double *__restrict__ recv, const int64_t *__restrict__ perm,
           const int64_t *__restrict__ blk, const int32_t *__restrict__ order, const int32_t *__restrict__ split,
           int nblocks, const int32_t *__restrict__ kcap, double tol, double *__restrict__ UV,
           const int64_t *__restrict__ uv_off, uint8_t *__restrict__ used_ws, const int64_t *__restrict__ used_off,
           int32_t *__restrict__ rank_out, int32_t *__restrict__ status_out)
{
    __shared__ AcaSlot slots[2 * kAcaWarps];
    if (clusters) chain_release();
    // one CTA of the second launch, with a block to work on or without, ends after the clusters
    const bool last = !clusters && blockIdx.x == gridDim.x - 1;
    const int nh = split[0], nl = split[1];
    AcaGroup g;
    g.turn = 0;
    g.slot = slots;
    int pos = blockIdx.x, end;
    if (clusters) {
        g.t = (pos % kAcaCluster) * kAcaThreads + threadIdx.x;
        g.size = kAcaCluster * kAcaThreads;
        g.id = 0;
        pos /= kAcaCluster;
        end = nh;
    } else if (pos < nl) {
        g.t = threadIdx.x;
        g.size = kAcaThreads;
        g.id = 1;
        pos += nh;
        end = nh + nl;
    } else {
        const int q = threadIdx.x / kAcaSmall;
        g.t = threadIdx.x % kAcaSmall;
        g.size = kAcaSmall;
        g.id = 1 + q;
        g.slot = slots + 2 * q * (kAcaSmall / 32);
        pos = nh + nl + (pos - nl) * kAcaGroups + q;
        end = nblocks;
    }
    if (pos >= end) {   // whole groups (and whole clusters) leave
        if (last) chain_wait();
        return;
    }
    if (g.id == 0) g.sync();  // every CTA of the cluster runs before its shared memory is written to
    const int b = order[pos];
    const int64_t r0 = blk[4 * b], r1 = blk[4 * b + 1], c0 = blk[4 * b + 2], c1 = blk[4 * b + 3];
    const int m = (int)(r1 - r0), n = (int)(c1 - c0);
    const int M = 3 * m, Nc = 2 * n;
    const int K = kcap[b];
    double *U = UV + uv_off[b];
    double *V = U + (int64_t)K * M;
    uint8_t *used = used_ws + used_off[b];
    const int t = g.t;
    double frob2 = 0.0;
    int k = 0, istar = 0, status = 1;
    int guard = 0;
    while (k < K && guard < M + K) {
        ++guard;
        if (t == 0) used[istar] = 1;
        // residual row istar (receiver p, component c) over all columns
        const int pr = istar / 3, cr = istar % 3;
        const double *R = recv + kRecvStride * perm[r0 + pr];
        double *v = V + (int64_t)k * Nc;
        double mv = -1.0, sum = 0.0;
        int mi = 0x7fffffff;
        for (int q = t; q < n; q += g.size) {
            double ts[3], td[3];
            gen(perm[c0 + q], R, ts, td);
            v[2 * q] = ts[cr];
            v[2 * q + 1] = td[cr];
        }
        for (int q = t; q < n; q += g.size) {   // this thread's own columns: no barrier
            double xs = v[2 * q], xd = v[2 * q + 1];
            const double *Uc = U + istar, *Vc = V + 2 * q;
#pragma unroll 8
            for (int l = 0; l < k; ++l) {
                const double f = Uc[(int64_t)l * M];
                xs -= f * Vc[(int64_t)l * Nc];
                xd -= f * Vc[(int64_t)l * Nc + 1];
            }
            v[2 * q] = xs;
            v[2 * q + 1] = xd;
            sum += xs * xs + xd * xd;
            const double as = fabs(xs), ad = fabs(xd);
            if (as > mv) { mv = as; mi = 2 * q; }
            if (ad > mv) { mv = ad; mi = 2 * q + 1; }
        }
        double best, nv2;
        int jstar;
        g.reduce(mv, mi, sum, best, jstar, nv2);
        if (!(best > 0.0) || !isfinite(best)) {
            // row represented exactly (or not finite): next unused row, no new term
            if (!isfinite(best)) { status = 2; break; }
            int nxt = -1;
            for (int r = 0; r < M; ++r)
                if (!used[r]) { nxt = r; break; }
            if (nxt < 0) { status = 0; break; }
            istar = nxt;
            g.sync();   // every thread has looked before the row is marked
            continue;
        }
        const double pivot = v[jstar];
        // residual column jstar (source q, slip s) over all rows, scaled by the pivot
        const int qc = jstar / 2, sc = jstar % 2;
        const int64_t jb = perm[c0 + qc];
        double *u = U + (int64_t)k * M;
        mv = -1.0;
        mi = 0x7fffffff;
        double nu2 = 0.0;
        for (int p = t; p < m; p += g.size) {
            double ts[3], td[3];
            gen(jb, recv + kRecvStride * perm[r0 + p], ts, td);
            const double *tt = sc ? td : ts;
            u[3 * p] = tt[0];
            u[3 * p + 1] = tt[1];
            u[3 * p + 2] = tt[2];
        }
        for (int p = t; p < m; p += g.size) {   // this thread's own rows
            double x[3] = {u[3 * p], u[3 * p + 1], u[3 * p + 2]};
            const double *Uc = U + 3 * p, *Vc = V + jstar;
#pragma unroll 8
            for (int l = 0; l < k; ++l) {
                const double f = Vc[(int64_t)l * Nc];
                x[0] -= f * Uc[(int64_t)l * M];
                x[1] -= f * Uc[(int64_t)l * M + 1];
                x[2] -= f * Uc[(int64_t)l * M + 2];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double y = x[c] / pivot, ay = fabs(y);
                u[3 * p + c] = y;
                nu2 += y * y;
                if (ay > mv && !used[3 * p + c]) { mv = ay; mi = 3 * p + c; }   // largest |u| among unused rows
            }
        }
        g.sync();
        // |S_k|^2 = |S_{k-1}|^2 + 2 sum_l (u.u_l)(v.v_l) + |u|^2 |v|^2: the k
        // cross products one warp per term l, the sum with the others' reduction
        double cross_w = 0.0;
        {
            const int lane = t & 31;
            for (int l = t >> 5; l < k; l += g.size >> 5) {
                double du = 0.0, dv = 0.0;
                const double *Ul = U + (int64_t)l * M, *Vl = V + (int64_t)l * Nc;
#pragma unroll 4
                for (int row = lane; row < M; row += 32) du += u[row] * Ul[row];
#pragma unroll 4
                for (int col = lane; col < Nc; col += 32) dv += v[col] * Vl[col];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    du += __shfl_xor_sync(0xffffffffu, du, o);
                    dv += __shfl_xor_sync(0xffffffffu, dv, o);
                }
                cross_w += du * dv;
            }
        }
        double bv, cross, skip;
        int bi, sbi;
        g.reduce(mv, mi, nu2, bv, bi, nu2);
        g.reduce(-1.0, 0, (t & 31) == 0 ? cross_w : 0.0, skip, sbi, cross);
        frob2 += 2.0 * cross + nu2 * nv2;
        ++k;
        if (sqrt(nu2 * nv2) <= tol * sqrt(fmax(frob2, 0.0))) { status = 0; break; }
        if (bv < 0.0) { status = 0; break; }   // every row used: exact
        istar = bi;   // the next pivot row
    }
    if (t == 0) {
        rank_out[b] = k;
        status_out[b] = status;
    }
    if (last) chain_wait();
}

// Storage of block b at data + off[b] (FP32, column-major so that the lanes
// of a warp read consecutive rows of one column):
//   dense:    D[col * M + row]                 (M = 3m rows, Nc = 2n columns)
//   low rank: U[l * M + row] for l < k, then V[l * Nc + col]   (K_b ~ U V)
// Rows are receiver x traction component (3p + c), columns source x slip
// direction (2q + s) in the block's local (renumbered) order.

// Dense blocks, one CTA per block; consecutive threads take consecutive
// receivers of one source.
template <bool kHalf>
__global__ void __launch_bounds__(kThreads)
dense_blocks_kernel(PairGen<kHalf> gen, const double *__restrict__ recv, const int64_t *__restrict__ perm,
                    const int64_t *__restrict__ blk, const int32_t *__restrict__ ids, float *__restrict__ D,
                    const int64_t *__restrict__ d_off)
{
    const int b = ids[blockIdx.x];
    const int64_t r0 = blk[4 * b], r1 = blk[4 * b + 1], c0 = blk[4 * b + 2], c1 = blk[4 * b + 3];
    const int m = (int)(r1 - r0), n = (int)(c1 - c0);
    const int64_t M = 3 * (int64_t)m;
    float *Db = D + d_off[b];
    for (int64_t e = threadIdx.x; e < (int64_t)m * n; e += kThreads) {
        const int q = (int)(e / m), p = (int)(e % m);
        double ts[3], td[3];
        gen(perm[c0 + q], recv + kRecvStride * perm[r0 + p], ts, td);
        float *col_s = Db + (int64_t)(2 * q) * M + 3 * p;
        float *col_d = col_s + M;
        for (int c = 0; c < 3; ++c) {
            col_s[c] = (float)ts[c];
            col_d[c] = (float)td[c];
        }
    }
}

// Copy the converged ACA factors (FP64, U as k rows of length M, then V as k
// rows of length Nc) to FP32 storage in the same order.
__global__ void pack_factors_kernel(const double *__restrict__ UV, const int64_t *__restrict__ uv_off,
                                    const int64_t *__restrict__ blk, const int32_t *__restrict__ kcap,
                                    const int32_t *__restrict__ rank, const int32_t *__restrict__ ids,
                                    float *__restrict__ out, const int64_t *__restrict__ out_off)
{
    const int b = ids[blockIdx.x];
    const int M = 3 * (int)(blk[4 * b + 1] - blk[4 * b]), Nc = 2 * (int)(blk[4 * b + 3] - blk[4 * b + 2]);
    const int k = rank[b], K = kcap[b];
    const double *U = UV + uv_off[b];
    const double *V = U + (int64_t)K * M;
    float *Uo = out + out_off[b];
    float *Vo = Uo + (int64_t)M * k;
    for (int64_t e = threadIdx.x; e < (int64_t)M * k; e += blockDim.x) Uo[e] = (float)U[e];
    for (int64_t e = threadIdx.x; e < (int64_t)k * Nc; e += blockDim.x) Vo[e] = (float)V[e];
}

// ---------------------------------------------------------------------------
// product  Y[r][3e + c] = sum over blocks of the H-matrix rows of element e
//
// Arithmetic: FP32 entries times the right-hand side split into FP32 hi + lo
// (2 FMAs per entry), FP32 partial sums over at most one block segment (or
// 1024 columns), then float-float (FF) sums; FP64 only for the final sum of a
// row's per-warp partials.

struct Acc2 {   // FP32 partial sum of one lane
    float s, c;
};

__device__ __forceinline__ void acc2_add(Acc2 &a, float k, float2 x)
{
    a.s = fmaf(k, x.x, a.s);
    a.c = fmaf(k, x.y, a.c);
}


// Float-float (unevaluated sum hi + lo) accumulation with FP32 operations
// only (Knuth's TwoSum), for the reductions of the low-rank product: GB300's
// FP64 rate is 1/64 of FP32, and an FP64 reduction per rank row made that
// kernel FP64-bound.
struct FF {
    float hi, lo;
};

__device__ __forceinline__ FF ff_add(FF a, FF b)
{
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    const float l = __fadd_rn(__fadd_rn(a.lo, b.lo), e);
    const float h = __fadd_rn(s, l);
    return FF{h, __fsub_rn(l, __fsub_rn(h, s))};
}

__device__ __forceinline__ FF warp_sum_ff(FF v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        FF w;
        w.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
        w.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
        v = ff_add(v, w);
    }
    return v;
}

__device__ __forceinline__ float2 split2(double x)
{
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
}

// X (FP64, [B][2N], element order) -> Xs ([B][2N] float (hi, lo) pairs, permuted order)
// run r takes part iff act == NULL or act[r * act_stride] != 0
__device__ __forceinline__ bool run_on(const int32_t *act, int act_stride, int r)
{
    return act == nullptr || act[(int64_t)r * act_stride] != 0;
}

__global__ void permute_split_kernel(const double *__restrict__ X, const int64_t *__restrict__ perm, int64_t N, int B,
                                     float2 *__restrict__ Xs, const int32_t *act, int act_stride)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (i >= 2 * N || r >= B || !run_on(act, act_stride, r)) return;
    const int64_t q = i >> 1;
    Xs[(int64_t)r * 2 * N + i] = split2(X[(int64_t)r * 2 * N + 2 * perm[q] + (i & 1)]);
}

// T[w * B + r] = V_b[l] . x_r[cols of b] as an FP32 (hi, lo) pair for rank
// row w (row l of low-rank block b).  Two work lists, built by the host with
// the split at 8,192 columns.  The shorter rows come in groups of up to 4
// consecutive rows of one block (t_grp: one 16-byte record per group holding
// the first row's storage offset, first x column and length, the first rank
// row and the group size), kTGroupsPerWarp consecutive groups per warp: the
// warp loads the next group's record while it streams the current group, so
// no dependent descriptor load sits between two groups, and consecutive
// groups of one block find their x values in L1.  The longer rows (t_sched
// tail, t_info records) take one CTA each with the columns cut into kTWarps
// contiguous pieces (a warp streams only a few KB in flight, so a long row on
// one warp would be the tail) and the partial sums added in warp order.
// Runs are the fastest-varying part of the block index, so the B CTAs that
// read the same factor rows run together and share them in L2.
constexpr int kTWarps = 4;
constexpr int kTGroupsPerWarp = 2;

__device__ __forceinline__ FF t_row_part(const float *__restrict__ v, const float2 *__restrict__ x, int xs,
                                         int c_begin, int c_end, int lane)
{
    FF sum{0.f, 0.f};
    for (int c0k = c_begin; c0k < c_end; c0k += 1024) {
        const int cend = min(c_end, c0k + 1024);
        Acc2 a0{0.f, 0.f}, a1{0.f, 0.f};
        int col = c0k + lane;
        // 16 columns per lane in flight: an average rank row (~630 columns)
        // is one or two rounds
        for (; col + 480 < cend; col += 512) {
            float k[16];
            float2 xv[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                k[u] = __ldg(v + col + 32 * u);
                xv[u] = x[(col + 32 * u) * xs];
            }
#pragma unroll
            for (int u = 0; u < 16; u += 2) {
                acc2_add(a0, k[u], xv[u]);
                acc2_add(a1, k[u + 1], xv[u + 1]);
            }
        }
        for (; col + 96 < cend; col += 128) {
            float k[4];
            float2 xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                k[u] = __ldg(v + col + 32 * u);
                xv[u] = x[(col + 32 * u) * xs];
            }
            acc2_add(a0, k[0], xv[0]);
            acc2_add(a1, k[1], xv[1]);
            acc2_add(a0, k[2], xv[2]);
            acc2_add(a1, k[3], xv[3]);
        }
        for (; col < cend; col += 32) acc2_add(a0, __ldg(v + col), x[col * xs]);
        // the hi and lo parts of the FP32 partial sums of this chunk
        sum = ff_add(sum, FF{a0.s, 0.f});
        sum = ff_add(sum, FF{a1.s, 0.f});
        sum = ff_add(sum, FF{__fadd_rn(a0.c, a1.c), 0.f});
    }
    return warp_sum_ff(sum);
}

// Up to 4 consecutive short rank rows of one block on one warp: the rows
// share their x values, so a lane loads x once per column for all of them and
// keeps 8 columns of every row in flight; a warp therefore moves ~4x the bytes
// per memory round trip of a one-row walk (the ~630-column rows were bound by
// their round trips).  Row j starts at v + j * nc.  Columns beyond the end
// are predicated off (zero terms); partial sums move to float-float every
// 1024 columns.
__device__ __forceinline__ void t_row_group(const float *__restrict__ v, int nc, int g, const float2 *__restrict__ x,
                                            int lane, FF (&out)[4])
{
    FF sum[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[j] = FF{0.f, 0.f};
    for (int c0k = 0; c0k < nc; c0k += 1024) {
        Acc2 a[4];   // one FMA chain pair per row: the 4 rows give the pipeline its independent chains
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = Acc2{0.f, 0.f};
        const int cend = min(nc, c0k + 1024);
        for (int col = c0k + lane; col - lane < cend; col += 256) {
            float2 xv[8];
            float k[4][8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const int c = col + 32 * u;
                const bool ok = c < cend;
                xv[u] = ok ? x[c] : make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j][u] = (ok && j < g) ? __ldg(v + (int64_t)j * nc + c) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc2_add(a[j], k[j][u], xv[u]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            sum[j] = ff_add(sum[j], FF{a[j].s, 0.f});
            sum[j] = ff_add(sum[j], FF{a[j].c, 0.f});
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j] = warp_sum_ff(sum[j]);
}

// CTA cta of the rank rows of run r (of B): all threads of a block of kTWarps warps.
__device__ __forceinline__ void lowrank_T_cta(int64_t cta, const float *__restrict__ data,
                                              const longlong2 *__restrict__ t_info, const int32_t *__restrict__ t_sched,
                                              const longlong2 *__restrict__ t_grp, int64_t ngrp, int64_t nshort,
                                              int64_t nlong, int64_t short_ctas, const float2 *__restrict__ xr, int B,
                                              int r, float2 *__restrict__ T, FF *part)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (cta < short_ctas) {
        const int64_t g0 = (cta * kTWarps + wid) * kTGroupsPerWarp;
        if (g0 >= ngrp) return;
        const int64_t g1 = min(ngrp, g0 + kTGroupsPerWarp);
        // record of group gi: .x = V offset | row length << 40 | size << 56,
        // .y = first x column | first rank row << 32
        longlong2 nrec = t_grp[g0];
        for (int64_t gi = g0; gi < g1; ++gi) {
            const longlong2 rec = nrec;
            if (gi + 1 < g1) nrec = t_grp[gi + 1];
            const int64_t off = rec.x & ((1ll << 40) - 1);
            const int nc = (int)((rec.x >> 40) & 0xffff), g = (int)(rec.x >> 56);
            const int64_t w0 = (int64_t)((uint64_t)rec.y >> 32);
            FF sg[4];
            t_row_group(data + off, nc, g, xr + (int32_t)(rec.y & 0xffffffffll), lane, sg);
            if (lane == 0)
                for (int j = 0; j < g; ++j) T[(w0 + j) * (int64_t)B + r] = make_float2(sg[j].hi, sg[j].lo);
        }
        return;
    }
    const int64_t q = cta - short_ctas;
    if (q >= nlong) return;   // uniform per CTA
    const int w = t_sched[nshort + q];
    const longlong2 info = t_info[w];
    const int Nc = (int)(info.y >> 32);
    const int piece = (Nc / kTWarps + 31) / 32 * 32;
    const int c_begin = min(Nc, wid * piece), c_end = min(Nc, (wid + 1) * piece);
    const FF s = t_row_part(data + info.x, xr + (int32_t)(info.y & 0xffffffffll), 1, c_begin, c_end, lane);
    if (lane == 0) part[wid] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        FF t = part[0];
        for (int k = 1; k < kTWarps; ++k) t = ff_add(t, part[k]);
        T[w * (int64_t)B + r] = make_float2(t.hi, t.lo);
    }
}

__global__ void __launch_bounds__(kTWarps * 32, 6)
lowrank_T_kernel(const float *__restrict__ data, const longlong2 *__restrict__ t_info,
                 const int32_t *__restrict__ t_sched, const longlong2 *__restrict__ t_grp, int64_t ngrp,
                 int64_t nshort, int64_t nlong, int64_t short_ctas,
                 const float2 *__restrict__ Xs, int64_t N, int B, float2 *__restrict__ T, const int32_t *act,
                 int act_stride)
{
    __shared__ FF part[kTWarps];
    const int r = (int)(blockIdx.x % (unsigned)B);
    const int64_t cta = blockIdx.x / (unsigned)B;
    if (!run_on(act, act_stride, r)) return;   // uniform per CTA
    lowrank_T_cta(cta, data, t_info, t_sched, t_grp, ngrp, nshort, nlong, short_ctas, Xs + (int64_t)r * 2 * N, B, r, T,
                  part);
}

// The same for a batch's only run that takes part (list: run_list_kernel).
__global__ void __launch_bounds__(kTWarps * 32, 6)
lowrank_T_only_kernel(const float *__restrict__ data, const longlong2 *__restrict__ t_info,
                      const int32_t *__restrict__ t_sched, const longlong2 *__restrict__ t_grp, int64_t ngrp,
                      int64_t nshort, int64_t nlong, int64_t short_ctas, const float2 *__restrict__ xr,
                      float2 *__restrict__ T, const int32_t *__restrict__ list)
{
    __shared__ FF part[kTWarps];
    if (list[0] != 1) return;
    lowrank_T_cta(blockIdx.x, data, t_info, t_sched, t_grp, ngrp, nshort, nlong, short_ctas, xr, 1, 0, T, part);
}

// ---------------------------------------------------------------------------
// Several right-hand sides: every loaded entry of H is used for up to 8 runs
// (4 in the rank rows), with each run's arithmetic -- the same terms, partial
// sums and order -- that of the one-run kernels above, so that a run's bits do
// not depend on its batch.
//
// The runs that take part are numbered in order (list[0] of them, list[1 + i]
// = run i) and go into groups of 8, the last one 2, 4 or 8 wide.  The x and T
// values of two runs lie side by side, [pair][column] of 16 bytes: a warp's 32
// columns of a pair are four full lines (with all 8 runs of a column together,
// its loads touched every line of 2 KB four times over).
//
// Bound: L2 in the rank rows (the entries once per 4 runs and the x values:
// 8.3 TB/s), FP32 issue in the leaf rows (2 FMAs per entry and run, one packed
// f32x2 FMA; 47 % of the FMA pipe) -- beside 0.2 ms of HBM.  N = 30,000,
// B = 16: 2.17 ms with a CTA per (leaf, run) -- 16 walks over the blocks from L2,
// 19 instructions per 192 products -- 1.46 ms with 8 runs per entry (rank rows
// 0.58, leaf rows 0.85), 1.06 ms with the loads kept in flight, the float-float
// sums of two runs in one instruction and the row passes on two CTAs (0.35 and
// 0.69), 1.02 ms with more L1 left to the leaf rows (0.64).  A second set of
// registers for the next entries spills: 1.50 ms.

__host__ __device__ inline int group_width(int left) { return left > 4 ? 8 : (left > 2 ? 4 : 2); }
// slots of n runs (B > 1)
__host__ __device__ inline int64_t run_slots(int n)
{
    return n <= 1 ? n : 8 * (int64_t)(n / 8) + (n % 8 ? group_width(n % 8) : 0);
}

__global__ void run_list_kernel(int B, const int32_t *act, int act_stride, int32_t *__restrict__ list)
{
    const int lane = threadIdx.x;
    int n = 0;
    for (int r0 = 0; r0 < B; r0 += 32) {
        const bool on = r0 + lane < B && run_on(act, act_stride, r0 + lane);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) list[1 + n + __popc(m & ((1u << lane) - 1u))] = r0 + lane;
        n += __popc(m);
    }
    if (lane == 0) list[0] = n;
}

// the (hi, lo) products of one entry and one run: two FMAs in one instruction
__device__ __forceinline__ uint64_t pack2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t k, uint64_t x)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(k), "l"(x));
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

typedef ulonglong2 Pair2;   // (hi, lo) of two runs, as f32x2 operands

// ff_add of two runs at once (hi and lo of the two side by side), and with an
// addend without a low part
struct __align__(16) FFPair {
    uint64_t hi, lo;
};
__device__ __forceinline__ uint64_t two_sum2(uint64_t a, uint64_t b, uint64_t &e)
{
    const uint64_t s = add2(a, b), bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
    return s;
}
__device__ __forceinline__ FFPair ff_close2(uint64_t s, uint64_t l)
{
    const uint64_t h = add2(s, l);
    return FFPair{h, sub2(l, sub2(h, s))};
}
__device__ __forceinline__ FFPair ff_add2p(FFPair a, FFPair b)
{
    uint64_t e;
    const uint64_t s = two_sum2(a.hi, b.hi, e);
    return ff_close2(s, add2(add2(a.lo, b.lo), e));
}
__device__ __forceinline__ FFPair ff_add2p(FFPair a, uint64_t b)
{
    uint64_t e;
    const uint64_t s = two_sum2(a.hi, b, e);
    return ff_close2(s, add2(a.lo, e));
}

__global__ void permute_split_runs_kernel(const double *__restrict__ X, const int64_t *__restrict__ perm, int64_t N,
                                          const int32_t *__restrict__ list, bool only, Pair2 *__restrict__ Xs)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int left = list[0] - 8 * (int)blockIdx.y;
    if (i >= 2 * N || left <= 0) return;
    const int64_t col = 2 * perm[i >> 1] + (i & 1);
    const int32_t *run = list + 1 + 8 * blockIdx.y;
    if (only && list[0] == 1) {
        reinterpret_cast<float2 *>(Xs)[i] = split2(X[(int64_t)run[0] * 2 * N + col]);
        return;
    }
    for (int h = 0; h < group_width(left) / 2; ++h) {
        float2 v[2];
        for (int j = 0; j < 2; ++j)
            v[j] = 2 * h + j < left ? split2(X[(int64_t)run[2 * h + j] * 2 * N + col]) : make_float2(0.f, 0.f);
        Xs[(4 * (int64_t)blockIdx.y + h) * 2 * N + i] = make_ulonglong2(pack2(v[0].x, v[0].y), pack2(v[1].x, v[1].y));
    }
}

// t_row_group for NR runs (pair h of the x values at x + h * xs, of the sums at
// T + h * ts); kept: 2 NR float-float sums a lane in shared memory, stride 32,
// for rows of more than 1024 columns.  An entry's register takes the column 128
// further on as soon as it is used, so that loads are always in flight without a
// second set of registers.  The 4 NR sums are reduced together: at each step
// of the butterfly a lane keeps half of them (16 additions for 16 sums instead
// of 80; every sum is added in warp_sum_ff's tree, and the two-sum is symmetric
// in its operands), two runs in one instruction.
template <int NR>
__device__ __forceinline__ void t_row_group_runs(const float *__restrict__ v, int nc, int g, const Pair2 *__restrict__ x,
                                                 int64_t xs, int lane, Pair2 *__restrict__ T, int64_t ts, FFPair *kept)
{
    constexpr int U = 4, P = 2 * NR;   // columns a lane per step; pairs of sums
    const float *row[4];               // rows past the group's last repeat it; their sums are not stored
#pragma unroll
    for (int j = 0; j < 4; ++j) row[j] = v + (int64_t)min(j, g - 1) * nc + lane;
    x += lane;
    float k[U][4];
    auto load = [&](int u, int c) {   // entries of the column c + lane (past the last: that one, its x is zero)
        const int cc = min(c, nc - 1 - lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) k[u][j] = __ldg(row[j] + cc);
    };
    FFPair sum[P];
#pragma unroll
    for (int u = 0; u < U; ++u) load(u, 32 * u);
    for (int c0k = 0; c0k < nc; c0k += 1024) {
        uint64_t a[2 * P];
#pragma unroll
        for (int q = 0; q < 2 * P; ++q) a[q] = 0ull;
        const int cend = min(nc, c0k + 1024);
        for (int c = c0k; c < cend; c += 32 * U) {
            const bool whole = c + 32 * U <= cend;
            Pair2 xv[U][NR / 2];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int h = 0; h < NR / 2; ++h)
                    xv[u][h] = whole || c + lane + 32 * u < cend ? x[h * xs + c + 32 * u] : make_ulonglong2(0ull, 0ull);
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t kk = pack2(k[u][j], k[u][j]);
#pragma unroll
                    for (int h = 0; h < NR / 2; ++h) {
                        fma2(a[j * NR + 2 * h], kk, xv[u][h].x);
                        fma2(a[j * NR + 2 * h + 1], kk, xv[u][h].y);
                    }
                }
                load(u, c + 32 * (U + u));
            }
        }
#pragma unroll
        for (int q = 0; q < P; ++q) {
            const float2 p0 = unpack2(a[2 * q]), p1 = unpack2(a[2 * q + 1]);
            const uint64_t s = pack2(p0.x, p1.x), c = pack2(p0.y, p1.y);
            if (c0k == 0) {
                sum[q].hi = two_sum2(s, c, sum[q].lo);   // what adding both to zero gives
            } else {
                sum[q] = ff_add2p(ff_add2p(kept[32 * q], s), c);
            }
            if (cend < nc) kept[32 * q] = sum[q];
        }
    }
    int idx = 0, o = 16;
#pragma unroll
    for (int n = P / 2; n >= 1; n >>= 1, o >>= 1) {   // n pairs stay
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < n; ++q) {
            const FFPair keep = up ? sum[q + n] : sum[q], give = up ? sum[q] : sum[q + n];
            FFPair other;
            other.hi = __shfl_xor_sync(0xffffffffu, give.hi, o);
            other.lo = __shfl_xor_sync(0xffffffffu, give.lo, o);
            sum[q] = ff_add2p(keep, other);
        }
        idx = 2 * idx + (up ? 1 : 0);
    }
    FF one;   // the last pair: a run to each half
    {
        const bool up = (lane & o) != 0;
        const float2 h = unpack2(sum[0].hi), l = unpack2(sum[0].lo);
        FF other;
        other.hi = __shfl_xor_sync(0xffffffffu, up ? h.x : h.y, o);
        other.lo = __shfl_xor_sync(0xffffffffu, up ? l.x : l.y, o);
        one = ff_add(FF{up ? h.y : h.x, up ? l.y : l.x}, other);
        idx = 2 * idx + (up ? 1 : 0);
    }
    for (int p = o >> 1; p > 0; p >>= 1) {
        FF other;
        other.hi = __shfl_xor_sync(0xffffffffu, one.hi, p);
        other.lo = __shfl_xor_sync(0xffffffffu, one.lo, p);
        one = ff_add(one, other);
    }
    if ((lane & (o - 1)) == 0 && idx / NR < g)
        reinterpret_cast<float2 *>(T + (idx % NR / 2) * ts + idx / NR)[idx & 1] = make_float2(one.hi, one.lo);
}

__global__ void __launch_bounds__(kTWarps * 32, 4)
lowrank_T_runs_kernel(const float *__restrict__ data, const longlong2 *__restrict__ t_info,
                      const int32_t *__restrict__ t_sched, const longlong2 *__restrict__ t_grp, int64_t ngrp,
                      int64_t nshort, int64_t nlong, int64_t short_ctas, const Pair2 *__restrict__ Xs, int64_t N,
                      int64_t t_rows, int nquads, Pair2 *__restrict__ T, const int32_t *__restrict__ list, bool only)
{
    __shared__ FF part[kTWarps];
    __shared__ FFPair kept[kTWarps][8 * 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int quad = (int)(blockIdx.x % (unsigned)nquads), grp = quad >> 1, half = quad & 1;
    const int64_t cta = blockIdx.x / (unsigned)nquads;
    const int left = list[0] - 8 * grp;
    if (left <= 4 * half || (only && list[0] == 1)) return;   // uniform per CTA
    const int nr = min(4, group_width(left));
    const Pair2 *xg = Xs + (4 * grp + 2 * half) * 2 * N;
    Pair2 *Tg = T + (4 * grp + 2 * half) * t_rows;
    if (cta < short_ctas) {
        const int64_t g0 = (cta * kTWarps + wid) * kTGroupsPerWarp;
        const int64_t g1 = min(ngrp, g0 + kTGroupsPerWarp);
        if (g0 >= ngrp) return;
        longlong2 nrec = t_grp[g0];
        for (int64_t gi = g0; gi < g1; ++gi) {
            const longlong2 rec = nrec;
            if (gi + 1 < g1) nrec = t_grp[gi + 1];
            const int64_t off = rec.x & ((1ll << 40) - 1);
            const int nc = (int)((rec.x >> 40) & 0xffff), g = (int)(rec.x >> 56);
            const int64_t w0 = (int64_t)((uint64_t)rec.y >> 32);
            const Pair2 *x = xg + (rec.y & 0xffffffffll);
            if (nr == 4) t_row_group_runs<4>(data + off, nc, g, x, 2 * N, lane, Tg + w0, t_rows, &kept[wid][lane]);
            else t_row_group_runs<2>(data + off, nc, g, x, 2 * N, lane, Tg + w0, t_rows, &kept[wid][lane]);
        }
        return;
    }
    const int64_t q = cta - short_ctas;
    if (q >= nlong) return;   // uniform per CTA
    const int row = t_sched[nshort + q];
    const longlong2 info = t_info[row];
    const int Nc = (int)(info.y >> 32);
    const int piece = (Nc / kTWarps + 31) / 32 * 32;
    const int c_begin = min(Nc, wid * piece), c_end = min(Nc, (wid + 1) * piece);
    for (int j = 0; j < min(nr, left - 4 * half); ++j) {
        const float2 *x = reinterpret_cast<const float2 *>(xg + (j >> 1) * 2 * N + (info.y & 0xffffffffll)) + (j & 1);
        const FF s = t_row_part(data + info.x, x, 2, c_begin, c_end, lane);
        __syncthreads();
        if (lane == 0) part[wid] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            FF t = part[0];
            for (int k = 1; k < kTWarps; ++k) t = ff_add(t, part[k]);
            reinterpret_cast<float2 *>(Tg + (j >> 1) * t_rows + row)[j & 1] = make_float2(t.hi, t.lo);
        }
    }
}

// One CTA per (leaf row cluster, run), the run fastest in the block index so
// that the B CTAs of one leaf read its blocks together (L2 reuse).
//
// Lane j of every warp owns rows j, j + 32, ... of the leaf (up to kPassRows
// rows per pass).  The work of the leaf -- the columns of its dense blocks and
// the rank columns of its low-rank blocks, in list order -- is cut into 8
// contiguous ranges, one per warp; a warp walks its range column by column
// (a coalesced 128-byte load per 32 rows, the column's x value broadcast),
// and the 8 per-warp partial sums of a row are added in warp order through
// shared memory.  The result does not depend on B or on timing.
struct BlkDesc {
    int64_t off;    // storage offset (floats)
    int64_t x0;     // dense: first column in Xs (2 c0); low rank: first T row (t_off)
    int32_t row0;   // first local row of this leaf in the block
    int32_t M;      // rows of the block (column stride)
    int32_t w;      // work columns: Nc (dense) or k (low rank)
    int32_t dense;
};

constexpr int kMaxLeafBlocks = 160;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxR = 6;
constexpr int kPassRows = 32 * kMaxR;

template <int R>
__device__ __forceinline__ void leaf_segment(const float *__restrict__ col0, int64_t M, const float2 *__restrict__ xp,
                                             int64_t xs, int ca, int cb, bool last_ok, FF (&acc)[kMaxR])
{
    constexpr int U = 4;   // columns in flight per warp
    Acc2 a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = Acc2{0.f, 0.f};
    int c = ca;
    for (; c + U <= cb; c += U) {
        float k[U][R];
        float2 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float *p = col0 + (int64_t)(c + u) * M;
            x[u] = xp[(int64_t)(c + u) * xs];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const bool ok = (i < R - 1) || last_ok;
                k[u][i] = ok ? __ldg(p + 32 * i) : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < R; ++i) acc2_add(a[i], k[u][i], x[u]);
    }
    for (; c < cb; ++c) {
        const float *p0 = col0 + (int64_t)c * M;
        const float2 x0 = xp[(int64_t)c * xs];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const bool ok = (i < R - 1) || last_ok;
            acc2_add(a[i], ok ? __ldg(p0 + 32 * i) : 0.f, x0);
        }
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        acc[i] = ff_add(acc[i], FF{a[i].s, 0.f});
        acc[i] = ff_add(acc[i], FF{a[i].c, 0.f});
    }
}

template <int R>
__device__ __forceinline__ void leaf_range(const BlkDesc *desc, const int *wpre, int nq, int64_t lo, int64_t hi, int pr0, int prow,
                           const float *__restrict__ data, const float2 *__restrict__ xr,
                           const float2 *__restrict__ T, int B, int r, FF (&acc)[kMaxR])
{
    const int lane = threadIdx.x & 31;
    const bool last_ok = lane + 32 * (R - 1) < prow;
    // first descriptor whose range ends after lo
    int q = 0;
    while (q < nq && wpre[q + 1] <= lo) ++q;
    for (; q < nq && wpre[q] < hi; ++q) {
        const BlkDesc d = desc[q];
        const int ca = (int)max((int64_t)0, lo - wpre[q]);
        const int cb = (int)min((int64_t)d.w, hi - wpre[q]);
        if (ca >= cb) continue;
        const float *col0 = data + d.off + d.row0 + pr0 + lane;
        if (d.dense) leaf_segment<R>(col0, d.M, xr + d.x0, 1, ca, cb, last_ok, acc);
        else leaf_segment<R>(col0, d.M, T + d.x0 * B + r, B, ca, cb, last_ok, acc);
    }
}

// Descriptors and column prefix sums of the blocks qs .. qs + nq of a leaf
// whose rows start at p0 (all threads of the CTA).
__device__ __forceinline__ void load_leaf_blocks(BlkDesc *desc, int *wpre, int nq, int64_t qs, int64_t p0,
                                                 const int64_t *__restrict__ off, const int64_t *__restrict__ blk,
                                                 const int32_t *__restrict__ rank,
                                                 const int32_t *__restrict__ leaf_blocks,
                                                 const int64_t *__restrict__ t_off)
{
    __syncthreads();
    for (int i = threadIdx.x; i < nq; i += kThreads) {
        const int bb = leaf_blocks[qs + i];
        const int64_t r0 = blk[4 * bb], c0 = blk[4 * bb + 2];
        const int k = rank[bb];
        BlkDesc d;
        d.off = off[bb];
        d.row0 = 3 * (int)(p0 - r0);
        d.M = 3 * (int)(blk[4 * bb + 1] - r0);
        d.dense = k < 0;
        d.w = k < 0 ? 2 * (int)(blk[4 * bb + 3] - c0) : k;
        d.x0 = k < 0 ? 2 * c0 : t_off[bb];
        desc[i] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int i = 0; i < nq; ++i) { wpre[i] = s; s += desc[i].w; }
        wpre[nq] = s;
    }
    __syncthreads();
}

// Leaf L of run r (of B), whose x values are xr and whose output is Yr: all threads.
__device__ __forceinline__ void leaf_rows_cta(int L, const float *__restrict__ data, const int64_t *__restrict__ off,
                                              const int64_t *__restrict__ blk, const int32_t *__restrict__ rank,
                                              const int64_t *__restrict__ leaf, const int64_t *__restrict__ leaf_ptr,
                                              const int32_t *__restrict__ leaf_blocks, const int64_t *__restrict__ perm,
                                              const float2 *__restrict__ xr, const float2 *__restrict__ T,
                                              const int64_t *__restrict__ t_off, int B, int r, double *__restrict__ Yr,
                                              BlkDesc *desc, int *wpre, double (*red)[kPassRows])
{
    const int64_t p0 = leaf[2 * L], p1 = leaf[2 * L + 1];
    const int rows = 3 * (int)(p1 - p0);
    const int64_t q0 = leaf_ptr[L], q1 = leaf_ptr[L + 1];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int pr0 = 0; pr0 < rows; pr0 += kPassRows) {
        const int prow = min(kPassRows, rows - pr0);
        const int R = (prow + 31) / 32;
        FF acc[kMaxR];
#pragma unroll
        for (int i = 0; i < kMaxR; ++i) acc[i] = FF{0.f, 0.f};
        for (int64_t qs = q0; qs < q1; qs += kMaxLeafBlocks) {
            const int nq = (int)min((int64_t)kMaxLeafBlocks, q1 - qs);
            load_leaf_blocks(desc, wpre, nq, qs, p0, off, blk, rank, leaf_blocks, t_off);
            const int64_t W = wpre[nq];
            const int64_t lo = W * wid / kWarps, hi = W * (wid + 1) / kWarps;
            switch (R) {
                case 1: leaf_range<1>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
                case 2: leaf_range<2>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
                case 3: leaf_range<3>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
                case 4: leaf_range<4>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
                case 5: leaf_range<5>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
                default: leaf_range<6>(desc, wpre, nq, lo, hi, pr0, prow, data, xr, T, B, r, acc); break;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kMaxR; ++i) red[wid][lane + 32 * i] = (double)acc[i].hi + (double)acc[i].lo;
        __syncthreads();
        for (int lr = threadIdx.x; lr < prow; lr += kThreads) {
            double s = 0.0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += red[w][lr];
            const int row = pr0 + lr;
            Yr[3 * perm[p0 + row / 3] + row % 3] = s;
        }
    }
}

__global__ void __launch_bounds__(kThreads, 3)
leaf_rows_kernel(const float *__restrict__ data, const int64_t *__restrict__ off, const int64_t *__restrict__ blk,
                 const int32_t *__restrict__ rank, const int64_t *__restrict__ leaf, const int64_t *__restrict__ leaf_ptr,
                 const int32_t *__restrict__ leaf_blocks, const int64_t *__restrict__ perm, const float2 *__restrict__ Xs,
                 const float2 *__restrict__ T, const int64_t *__restrict__ t_off, int64_t N, int B,
                 double *__restrict__ Y, const int32_t *act, int act_stride)
{
    __shared__ BlkDesc desc[kMaxLeafBlocks];
    __shared__ int wpre[kMaxLeafBlocks + 1];
    __shared__ double red[kWarps][kPassRows];
    const int L = (int)(blockIdx.x / (unsigned)B), r = (int)(blockIdx.x % (unsigned)B);
    if (!run_on(act, act_stride, r)) return;   // uniform per CTA: before any barrier
    leaf_rows_cta(L, data, off, blk, rank, leaf, leaf_ptr, leaf_blocks, perm, Xs + (int64_t)r * 2 * N, T, t_off, B, r,
                  Y + (int64_t)r * 3 * N, desc, wpre, red);
}

// The same for a batch's only run that takes part.
__global__ void __launch_bounds__(kThreads, 3)
leaf_rows_only_kernel(const float *__restrict__ data, const int64_t *__restrict__ off, const int64_t *__restrict__ blk,
                      const int32_t *__restrict__ rank, const int64_t *__restrict__ leaf,
                      const int64_t *__restrict__ leaf_ptr, const int32_t *__restrict__ leaf_blocks,
                      const int64_t *__restrict__ perm, const float2 *__restrict__ xr, const float2 *__restrict__ T,
                      const int64_t *__restrict__ t_off, int64_t N, double *__restrict__ Y,
                      const int32_t *__restrict__ list)
{
    __shared__ BlkDesc desc[kMaxLeafBlocks];
    __shared__ int wpre[kMaxLeafBlocks + 1];
    __shared__ double red[kWarps][kPassRows];
    if (list[0] != 1) return;
    leaf_rows_cta((int)blockIdx.x, data, off, blk, rank, leaf, leaf_ptr, leaf_blocks, perm, xr, T, t_off, 1, 0,
                  Y + (int64_t)list[1] * 3 * N, desc, wpre, red);
}

// The leaf rows for NR runs: as leaf_rows_kernel, a CTA per (leaf, group of
// runs), the work columns in the same 8 ranges.  Lanes own up to kRunRows / NR
// rows (24 f32x2 accumulators a lane).  The x values of 32 columns come into
// shared memory by asynchronous copies (a lane takes its column's pairs), the
// next 32 while these are used; an entry's register takes the column 8 further
// on (4 in wide passes) as soon as it is used; the float-float sums, touched
// once per block segment, live in shared memory.  The row passes of a leaf are
// independent: two CTAs take every other one (N = 30,000: 512 leaves are 1,024
// CTAs for 304 places, whose last round was half empty).  What a CTA leaves of its
// share of shared memory is L1: with the warps' sums in place of the staged x, no
// longer needed then, 60 KB instead of 28 (N = 29,756: 16 runs 1,028 -> 985 us, 2 runs
// 418 -> 365).
constexpr int kRunRows = 24;
constexpr int kRunMaxR = 6;
constexpr int kRunPasses = 2;   // CTAs of a leaf and run group
constexpr int kRunFF = kRunRows * kThreads * (int)sizeof(float2);                  // float-float sums
constexpr int kRunX = kWarps * 2 * 32 * 4 * (int)sizeof(Pair2);                    // staged x, two chunks
constexpr int kRunRed = kWarps * 32 * kRunMaxR * (int)sizeof(double);              // one run's warp sums
constexpr int kRunSmem = kRunFF + (kRunX > kRunRed ? kRunX : kRunRed);

__device__ __forceinline__ void copy16_async(void *smem, const void *gmem)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// xp: column 0 of the segment's x values (pair h at xp + h * xs); row: offset
// of the lane's last row in a column (a lane without one repeats the leaf's last)
template <int R, int NR>
__device__ __forceinline__ void leaf_segment_runs(const float *__restrict__ col0, int row, int M,
                                                  const Pair2 *__restrict__ xp, int64_t xs, int ca, int cb, Pair2 *sx,
                                                  FFPair *ff)
{
    constexpr int H = NR / 2, U = R <= 3 ? 8 : 4;   // columns in flight (24 entries a lane)
    const int lane = threadIdx.x & 31;
    uint64_t a[R * NR];
#pragma unroll
    for (int i = 0; i < R * NR; ++i) a[i] = 0ull;
    auto stage = [&](int c0, int buf) {   // one group of copies per chunk, empty past the end
        if (c0 + lane < cb)
#pragma unroll
            for (int h = 0; h < H; ++h) copy16_async(&sx[buf * 32 * H + lane * H + h], xp + h * xs + c0 + lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float k[U][R];
    const float *coll = col0 + row;
    auto load = [&](int u, int c) {   // entries of column c (past the last: that one, unused)
        const int64_t o = min(c, cb - 1) * (int64_t)M;
#pragma unroll
        for (int i = 0; i < R - 1; ++i) k[u][i] = __ldg(col0 + o + 32 * i);
        k[u][R - 1] = __ldg(coll + o);
    };
    auto column = [&](int u, const Pair2 *x0) {
        uint64_t kk[R];
#pragma unroll
        for (int i = 0; i < R; ++i) kk[i] = pack2(k[u][i], k[u][i]);
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const Pair2 x = x0[h];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                fma2(a[i * NR + 2 * h], kk[i], x.x);
                fma2(a[i * NR + 2 * h + 1], kk[i], x.y);
            }
        }
    };
    __syncwarp();   // the last segment's chunks have been read
    stage(ca, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) load(u, ca + u);
    int buf = 0;
    for (int c0 = ca; c0 < cb; c0 += 32, buf ^= 1) {
        stage(c0 + 32, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();   // this chunk is in, from every lane
        const Pair2 *x0 = sx + buf * 32 * H;
        const int n = min(32, cb - c0);
        int c = 0;
        for (; c + U <= n; c += U)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                column(u, x0 + (c + u) * H);
                load(u, c0 + c + U + u);
            }
#pragma unroll
        for (int u = 0; u < U - 1; ++u)   // the segment's last columns
            if (c + u < n) column(u, x0 + (c + u) * H);
        __syncwarp();   // the chunk has been read: the next but one goes there
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < R * H; ++i) {
        const float2 v0 = unpack2(a[2 * i]), v1 = unpack2(a[2 * i + 1]);
        ff[i * kThreads] = ff_add2p(ff_add2p(ff[i * kThreads], pack2(v0.x, v1.x)), pack2(v0.y, v1.y));
    }
}

template <int R, int NR>
__device__ __forceinline__ void leaf_range_runs(const BlkDesc *desc, const int *wpre, int nq, int64_t lo, int64_t hi,
                                                int pr0, int prow, const float *__restrict__ data,
                                                const Pair2 *__restrict__ xg, const Pair2 *__restrict__ Tg,
                                                int64_t N, int64_t t_rows, Pair2 *sx, FFPair *ff)
{
    const int lane = threadIdx.x & 31;
    const int row = min(32 * (R - 1), prow - 1 - lane);
    int q = 0;
    while (q < nq && wpre[q + 1] <= lo) ++q;
    for (; q < nq && wpre[q] < hi; ++q) {
        const BlkDesc d = desc[q];
        const int ca = (int)max((int64_t)0, lo - wpre[q]);
        const int cb = (int)min((int64_t)d.w, hi - wpre[q]);
        if (ca >= cb) continue;
        leaf_segment_runs<R, NR>(data + d.off + d.row0 + pr0 + lane, row, d.M, (d.dense ? xg : Tg) + d.x0,
                                 d.dense ? 2 * N : t_rows, ca, cb, sx, ff);
    }
}

template <int NR>
__device__ __forceinline__ void leaf_rows_runs(const float *__restrict__ data, const int64_t *__restrict__ off,
                                               const int64_t *__restrict__ blk, const int32_t *__restrict__ rank,
                                               int64_t p0, int64_t p1, int64_t q0, int64_t q1,
                                               const int32_t *__restrict__ leaf_blocks, const int64_t *__restrict__ perm,
                                               const Pair2 *__restrict__ xg, const Pair2 *__restrict__ Tg,
                                               const int64_t *__restrict__ t_off, int64_t t_rows, int64_t N, int runs,
                                               const int32_t *__restrict__ run, double *__restrict__ Y, int pass0, int pass_rows, BlkDesc *desc,
                                               int *wpre, char *smem)
{
    constexpr int kR = kRunRows / NR < kRunMaxR ? kRunRows / NR : kRunMaxR;
    constexpr int kPass = 32 * kR;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    FFPair *ff = reinterpret_cast<FFPair *>(smem) + threadIdx.x;
    Pair2 *sx = reinterpret_cast<Pair2 *>(smem + kRunFF) + wid * 2 * 32 * 4;
    double *red = reinterpret_cast<double *>(smem + kRunFF);   // once the staged x is done with
    const int rows = 3 * (int)(p1 - p0);
    const int pass = min(kPass, pass_rows);
    for (int pr0 = pass0 * pass; pr0 < rows; pr0 += kRunPasses * pass) {
        const int prow = min(pass, rows - pr0);
        const int R = (prow + 31) / 32;
        for (int i = 0; i < kR * NR / 2; ++i) ff[i * kThreads] = FFPair{0ull, 0ull};
        for (int64_t qs = q0; qs < q1; qs += kMaxLeafBlocks) {
            const int nq = (int)min((int64_t)kMaxLeafBlocks, q1 - qs);
            load_leaf_blocks(desc, wpre, nq, qs, p0, off, blk, rank, leaf_blocks, t_off);
            const int64_t W = wpre[nq];
            const int64_t lo = W * wid / kWarps, hi = W * (wid + 1) / kWarps;
            if (R == 1) leaf_range_runs<1, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
            else if (R == 2) leaf_range_runs<2, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
            else if (R == 3 || kR == 3) leaf_range_runs<3, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
            else if (R == 4) leaf_range_runs<kR < 4 ? kR : 4, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
            else if (R == 5) leaf_range_runs<kR < 5 ? kR : 5, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
            else leaf_range_runs<kR, NR>(desc, wpre, nq, lo, hi, pr0, prow, data, xg, Tg, N, t_rows, sx, ff);
        }
        for (int j = 0; j < runs; ++j) {
            __syncthreads();
            for (int i = 0; i < kR; ++i) {
                const FFPair f = ff[(i * NR + j) / 2 * kThreads];
                const float2 h = unpack2(f.hi), l = unpack2(f.lo);
                red[wid * kPass + lane + 32 * i] = j & 1 ? (double)h.y + (double)l.y : (double)h.x + (double)l.x;
            }
            __syncthreads();
            double *Yr = Y + (int64_t)run[j] * 3 * N;
            for (int lr = threadIdx.x; lr < prow; lr += kThreads) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) s += red[w * kPass + lr];
                const int row = pr0 + lr;
                Yr[3 * perm[p0 + row / 3] + row % 3] = s;
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads, 2)
leaf_rows_runs_kernel(const float *__restrict__ data, const int64_t *__restrict__ off, const int64_t *__restrict__ blk,
                      const int32_t *__restrict__ rank, const int64_t *__restrict__ leaf,
                      const int64_t *__restrict__ leaf_ptr, const int32_t *__restrict__ leaf_blocks,
                      const int64_t *__restrict__ perm, const Pair2 *__restrict__ Xs, const Pair2 *__restrict__ T,
                      const int64_t *__restrict__ t_off, int64_t t_rows, int64_t N, int ngroups,
                      const int32_t *__restrict__ list, bool only, int pass_rows, double *__restrict__ Y)
{
    extern __shared__ __align__(16) char smem_runs[];
    __shared__ BlkDesc desc[kMaxLeafBlocks];
    __shared__ int wpre[kMaxLeafBlocks + 1];
    const int grp = (int)(blockIdx.x % (unsigned)ngroups);
    const unsigned lp = blockIdx.x / (unsigned)ngroups;
    const int L = (int)(lp / kRunPasses), pass0 = (int)(lp % kRunPasses);
    const int left = list[0] - 8 * grp;
    if (left <= 0 || (only && list[0] == 1)) return;   // uniform per CTA
    const int w = group_width(left), runs = min(left, 8);
    const Pair2 *xg = Xs + 4 * grp * 2 * N, *Tg = T + 4 * grp * t_rows;
    const int32_t *run = list + 1 + 8 * grp;
    const int64_t p0 = leaf[2 * L], p1 = leaf[2 * L + 1], q0 = leaf_ptr[L], q1 = leaf_ptr[L + 1];
    if (w == 8)
        leaf_rows_runs<8>(data, off, blk, rank, p0, p1, q0, q1, leaf_blocks, perm, xg, Tg, t_off, t_rows, N, runs, run, Y, pass0,
                          pass_rows, desc, wpre, smem_runs);
    else if (w == 4)
        leaf_rows_runs<4>(data, off, blk, rank, p0, p1, q0, q1, leaf_blocks, perm, xg, Tg, t_off, t_rows, N, runs, run, Y, pass0,
                          pass_rows, desc, wpre, smem_runs);
    else
        leaf_rows_runs<2>(data, off, blk, rank, p0, p1, q0, q1, leaf_blocks, perm, xg, Tg, t_off, t_rows, N, runs, run, Y, pass0,
                          pass_rows, desc, wpre, smem_runs);
}

}  // namespace hm
}  // namespace pq3d

using namespace pq3d;
using namespace pq3d::hm;

static inline double poisson_(double mu, double lam) { return 1.0 / (1.0 + lam / mu) / 2.0; }

// Table layout written by pq3d_gf_setup: source [kSrcStride][N], receiver
// [N][kRecvStride], image [kImgStride][N], side table [kFscStride][N].
template <bool kHalf>
static PairGen<kHalf> make_gen(const double *tables, int64_t N, double mu, double lambda_)
{
    const double nu = poisson_(mu, lambda_);
    const double *img = tables + (size_t)(kSrcStride + kRecvStride) * N;
    return PairGen<kHalf>{tables, img, img + (size_t)kImgStride * N, N, nu, 1.0 / (8.0 * kPi * (1.0 - nu)),
                          2.0 * mu, lambda_};
}

extern "C" int pq3d_hmat_aca(const double *tables, int64_t N, const int64_t *perm, int nblocks, const int64_t *blk,
                             const int32_t *kcap, double tol, double mu, double lambda_, int halfspace, double *UV,
                             const int64_t *uv_off, uint8_t *used, const int64_t *used_off, int32_t *rank,
                             int32_t *status, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(tables && perm && blk && kcap && UV && uv_off && used && used_off && rank && status && N > 0,
                 "pq3d_hmat_aca: bad arguments");
    if (nblocks <= 0) return PQ3D_OK;
    const double *recv = tables + (size_t)kSrcStride * N;
    cudaStream_t st = (cudaStream_t)stream;
    // the work order lives for this call only (stream-ordered scratch); a grid of
    // nblocks CTAs serves any split, those past the last leave, and fewer blocks than
    // SMs exceed the average share of one, so that many clusters do (as many as blocks
    // took 0.4 ms to come and go for 7,822 of them)
    int dev, sms;
    PQ3D_CUDA_TRY(cudaGetDevice(&dev));
    PQ3D_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int32_t *split = nullptr;
    PQ3D_CUDA_TRY(cudaMallocAsync(&split, ((size_t)nblocks + 2) * sizeof(int32_t), st));
    aca_order_kernel<<<1, 1024, 0, st>>>(blk, nblocks, sms, split + 2, split);
    auto launch = [&](auto kernel, auto gen) -> cudaError_t {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kAcaCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(nblocks < sms ? nblocks : sms) * kAcaCluster);
        cfg.blockDim = dim3(kAcaThreads);
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        const int32_t *order = split + 2;
        cudaError_t e = cudaGetLastError();   // of aca_order_kernel
        if (e == cudaSuccess)
            e = cudaLaunchKernelEx(&cfg, kernel, true, gen, recv, perm, blk, order, (const int32_t *)split, nblocks, kcap,
                                   tol, UV, uv_off, used, used_off, rank, status);
        if (e == cudaSuccess)
            e = launch_chained(kernel, dim3((unsigned)nblocks), dim3(kAcaThreads), 0, st, false, gen, recv, perm, blk,
                               order, (const int32_t *)split, nblocks, kcap, tol, UV, uv_off, used, used_off, rank,
                               status);
        return e;
    };
    const cudaError_t launched = halfspace ? launch(aca_kernel<true>, make_gen<true>(tables, N, mu, lambda_))
                                           : launch(aca_kernel<false>, make_gen<false>(tables, N, mu, lambda_));
    PQ3D_CUDA_TRY(cudaFreeAsync(split, st));
    PQ3D_CUDA_TRY(launched);
    return PQ3D_OK;
}

extern "C" int pq3d_hmat_dense_blocks(const double *tables, int64_t N, const int64_t *perm, const int64_t *blk,
                                      const int32_t *ids, int nids, double mu, double lambda_, int halfspace,
                                      float *D, const int64_t *d_off, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(tables && perm && blk && ids && D && d_off && N > 0, "pq3d_hmat_dense_blocks: bad arguments");
    PQ3D_REQUIRE(((uintptr_t)D & 3u) == 0, "pq3d_hmat_dense_blocks: D must be 4-byte aligned");
    if (nids <= 0) return PQ3D_OK;
    const double *recv = tables + (size_t)kSrcStride * N;
    cudaStream_t st = (cudaStream_t)stream;
    if (halfspace)
        dense_blocks_kernel<true><<<nids, kThreads, 0, st>>>(make_gen<true>(tables, N, mu, lambda_), recv, perm, blk,
                                                             ids, D, d_off);
    else
        dense_blocks_kernel<false><<<nids, kThreads, 0, st>>>(make_gen<false>(tables, N, mu, lambda_), recv, perm,
                                                              blk, ids, D, d_off);
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}

extern "C" int pq3d_hmat_pack_factors(const double *UV, const int64_t *uv_off, const int64_t *blk, const int32_t *kcap,
                                      const int32_t *rank, const int32_t *ids, int nids, float *out,
                                      const int64_t *out_off, void *stream)
{
    clear_error();
    if (nids <= 0) return PQ3D_OK;
    pack_factors_kernel<<<nids, 256, 0, (cudaStream_t)stream>>>(UV, uv_off, blk, kcap, rank, ids, out, out_off);
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}

extern "C" int pq3d_hmat_apply_masked(const pq3d_hmat *H, const double *X, int B, double *Y,
                                      const int32_t *run_active, int active_stride, void *workspace,
                                      size_t workspace_bytes, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(H && X && Y && workspace && B >= 1, "pq3d_hmat_apply: bad arguments");
    const int64_t N = H->N;
    const size_t need = pq3d_hmat_workspace_bytes(H, B);
    PQ3D_REQUIRE(workspace_bytes >= need && aligned16(workspace), "pq3d_hmat_apply: workspace too small (%zu < %zu)",
                 workspace_bytes, need);
    cudaStream_t st = (cudaStream_t)stream;
    const longlong2 *t_info = (const longlong2 *)H->t_info, *t_grp = (const longlong2 *)H->t_grp;
    const int64_t nshort = H->t_rows - H->t_nlong;
    const int64_t short_ctas = (H->t_ngrp + kTWarps * kTGroupsPerWarp - 1) / (kTWarps * kTGroupsPerWarp);
    const int64_t t_ctas = short_ctas + H->t_nlong;
    const unsigned cols = (unsigned)((2 * N + 255) / 256);
    int dev, sms;
    PQ3D_CUDA_TRY(cudaGetDevice(&dev));
    PQ3D_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // One run, or so few leaves that a CTA for each and every run (three to an SM) still
    // finds room on the chip: run by run, the run fastest in the block index.  (8 runs:
    // N = 900, 32 leaves 35 us, 47 in a group; N = 2,500, 64 leaves 76, 71.)
    if (B == 1 || (int64_t)H->nleaves * B <= 3 * sms) {
        PQ3D_REQUIRE(t_ctas * B < (int64_t)INT32_MAX && (int64_t)H->nleaves * B < (int64_t)INT32_MAX,
                     "pq3d_hmat_apply: too many rank rows or leaves x runs");
        float2 *Xs = (float2 *)workspace, *T = Xs + (size_t)B * 2 * N;
        permute_split_kernel<<<dim3(cols, (unsigned)B), 256, 0, st>>>(X, H->perm, N, B, Xs, run_active, active_stride);
        if (H->t_rows > 0)
            lowrank_T_kernel<<<(unsigned)(t_ctas * B), kTWarps * 32, 0, st>>>(
                H->data, t_info, H->t_sched, t_grp, H->t_ngrp, nshort, H->t_nlong, short_ctas, Xs, N, B, T, run_active,
                active_stride);
        leaf_rows_kernel<<<(unsigned)(H->nleaves * B), kThreads, 0, st>>>(
            H->data, H->off, H->blk, H->rank, H->leaf, H->leaf_ptr, H->leaf_blocks, H->perm, Xs, T, H->t_off, N, B, Y,
            run_active, active_stride);
        PQ3D_CUDA_TRY(cudaGetLastError());
        return PQ3D_OK;
    }
    const int64_t slots = run_slots(B);
    const int ngroups = (B + 7) / 8;
    PQ3D_REQUIRE(t_ctas * 2 * ngroups < (int64_t)INT32_MAX &&
                     (int64_t)H->nleaves * ngroups * kRunPasses < (int64_t)INT32_MAX && ngroups < 65536,
                 "pq3d_hmat_apply: too many rank rows or leaves x runs");
    Pair2 *Xs = (Pair2 *)workspace, *T = Xs + (size_t)(slots / 2) * 2 * N;
    int32_t *list = (int32_t *)(T + (size_t)(slots / 2) * H->t_rows);
    // Rows of a leaf's pass: half of them where the leaves of one group of runs leave
    // SMs without a CTA, so that a leaf's second CTA takes the rest (2 runs: N = 8,100,
    // 184 leaves 144 us, whole passes 158; N = 12,100, 256 leaves 188, 175; 20 runs,
    // N = 2,200: an iteration 190 us, 176).
    const int pass_rows = ngroups == 1 && 3 * H->nleaves <= 4 * sms ? kPassRows / 2 : kPassRows;
    // How many runs take part is known on the device only.  A batch's only run does
    // better with the one-run kernels, from about four leaves an SM on (N = 99,856:
    // 1,075 us, 1,189 as half a pair; N = 29,756, 512 leaves: 362, 361): they follow
    // those below, which leave it to them, and else end at once (15 us there).
    const bool only = run_active && H->nleaves > 4 * sms;
    PQ3D_CUDA_TRY(allow_smem(leaf_rows_runs_kernel, kRunSmem));
    run_list_kernel<<<1, 32, 0, st>>>(B, run_active, active_stride, list);
    permute_split_runs_kernel<<<dim3(cols, (unsigned)ngroups), 256, 0, st>>>(X, H->perm, N, list, only, Xs);
    if (H->t_rows > 0)
        lowrank_T_runs_kernel<<<(unsigned)(t_ctas * 2 * ngroups), kTWarps * 32, 0, st>>>(
            H->data, t_info, H->t_sched, t_grp, H->t_ngrp, nshort, H->t_nlong, short_ctas, Xs, N, H->t_rows, 2 * ngroups,
            T, list, only);
    leaf_rows_runs_kernel<<<(unsigned)(H->nleaves * ngroups * kRunPasses), kThreads, kRunSmem, st>>>(
        H->data, H->off, H->blk, H->rank, H->leaf, H->leaf_ptr, H->leaf_blocks, H->perm, Xs, T, H->t_off, H->t_rows, N,
        ngroups, list, only, pass_rows, Y);
    if (only) {
        const float2 *x1 = (const float2 *)Xs;
        float2 *T1 = (float2 *)T;
        if (H->t_rows > 0)
            lowrank_T_only_kernel<<<(unsigned)t_ctas, kTWarps * 32, 0, st>>>(
                H->data, t_info, H->t_sched, t_grp, H->t_ngrp, nshort, H->t_nlong, short_ctas, x1, T1, list);
        leaf_rows_only_kernel<<<(unsigned)H->nleaves, kThreads, 0, st>>>(
            H->data, H->off, H->blk, H->rank, H->leaf, H->leaf_ptr, H->leaf_blocks, H->perm, x1, T1, H->t_off, N, Y,
            list);
    }
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}

extern "C" int pq3d_hmat_apply(const pq3d_hmat *H, const double *X, int B, double *Y, void *workspace,
                               size_t workspace_bytes, void *stream)
{
    return pq3d_hmat_apply_masked(H, X, B, Y, nullptr, 0, workspace, workspace_bytes, stream);
}

extern "C" size_t pq3d_hmat_workspace_bytes(const pq3d_hmat *H, int B)
{
    if (!H || B < 1) return 0;
    // x and T values of every run slot, then the list of runs (B > 1)
    return (size_t)run_slots(B) * (2 * (size_t)H->N + (size_t)H->t_rows) * sizeof(float2) +
           (B > 1 ? ((size_t)B + 1) * sizeof(int32_t) : 0);
}
