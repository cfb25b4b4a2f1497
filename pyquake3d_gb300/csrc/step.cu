// Dense quasi-dynamic stepping on the GPU (plain FP64 path, or the FP32
// operator copy).
//
// Reference behaviour (src/QDsim_gpu.py):
//   traction product K.(V - Vpl), once per accepted step        948-957
//   right-hand side (aging law, radiation damping)             830-891, in
//     reciprocal form with the reference formula's error (rhs_recip<true>)
//   Dormand-Prince 5(4) attempt, max-relative error norm      1128-1262
//   accept / reject and dt control                              959-985
//   closed-form slip rate, rake, slip integration              994-1027
//
// GPU design, per accepted step two launches queued back to back (no host
// synchronisation between steps): (1) the traction product, a warp per
// receiver (two or four on small meshes) streaming its three operator rows
// (16-byte loads) against the interleaved slip-rate deficit v', at the full
// occupancy of a small kernel;
// (2) one cooperative kernel: every thread runs the 7 right-hand-side
// evaluations of its cells in registers (the traction rates are frozen over
// the step, so the stages are cell-local), block-max + one atomicMax per block
// give the two error norms, one grid barrier, every thread takes the same
// accept/reject decision, retry until accepted; (3) the state update writes v'
// for the next step's product.  The step's control values (dt, time, attempt
// count) live in the control block between launches.  Grid barriers are
// bounded.  (The product inside one persistent kernel for all steps ran at
// the occupancy of the attempt code and took ~10 % longer: 4.93 against
// 4.50 ms per step at N = 20,000.)
#include <math.h>

#include "common.cuh"
#include "rk_device.cuh"

namespace pq3d {
namespace step {

using namespace ::pq3d::rk;

// ---------------------------------------------------------------------------
// traction product: rows 3i..3i+2 of K times v' (interleaved strike/dip)

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp: rows 3i + c, c = 0..2, over the sources [j0, j1).  K rows have N
// double2 (strike, dip).
__device__ __forceinline__ void rows3_f64(const double2 *__restrict__ K, const double2 *__restrict__ v, int64_t N,
                                          int64_t i, int64_t j0, int64_t j1, int lane, double acc[3])
{
    const double2 *r0 = K + (3 * i) * N, *r1 = r0 + N, *r2 = r1 + N;
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, b0 = 0.0, b1 = 0.0, b2 = 0.0;
    int64_t j = j0 + lane;
    for (; j + 32 < j1; j += 64) {
        const double2 x0 = __ldg(v + j), x1 = __ldg(v + j + 32);
        const double2 k00 = __ldcs(r0 + j), k10 = __ldcs(r1 + j), k20 = __ldcs(r2 + j);
        const double2 k01 = __ldcs(r0 + j + 32), k11 = __ldcs(r1 + j + 32), k21 = __ldcs(r2 + j + 32);
        a0 = fma(k00.x, x0.x, a0); a0 = fma(k00.y, x0.y, a0);
        a1 = fma(k10.x, x0.x, a1); a1 = fma(k10.y, x0.y, a1);
        a2 = fma(k20.x, x0.x, a2); a2 = fma(k20.y, x0.y, a2);
        b0 = fma(k01.x, x1.x, b0); b0 = fma(k01.y, x1.y, b0);
        b1 = fma(k11.x, x1.x, b1); b1 = fma(k11.y, x1.y, b1);
        b2 = fma(k21.x, x1.x, b2); b2 = fma(k21.y, x1.y, b2);
    }
    for (; j < j1; j += 32) {
        const double2 x0 = __ldg(v + j);
        const double2 k00 = __ldcs(r0 + j), k10 = __ldcs(r1 + j), k20 = __ldcs(r2 + j);
        a0 = fma(k00.x, x0.x, a0); a0 = fma(k00.y, x0.y, a0);
        a1 = fma(k10.x, x0.x, a1); a1 = fma(k10.y, x0.y, a1);
        a2 = fma(k20.x, x0.x, a2); a2 = fma(k20.y, x0.y, a2);
    }
    acc[0] = warp_sum(a0 + b0);
    acc[1] = warp_sum(a1 + b1);
    acc[2] = warp_sum(a2 + b2);
}

// FP32 operator: rows of N float2.  The products and sums are compensated so
// that the result is the FP32-rounded operator applied exactly (to ~2^-44):
// v' is split into hi + lo floats, k * vhi is formed exactly as p + e
// (TwoProduct with an FMA), the running sum is carried as s + c (TwoSum).  The
// _rn intrinsics keep the compiler from contracting these sequences.  FP32
// operations are ~64x cheaper than FP64 ones on this part, so the ~11 FP32
// operations per entry stay below the HBM time of the 4-byte entry.
struct Acc2 {
    float s, c;
};

__device__ __forceinline__ void acc2_add(Acc2 &a, float k, float vh, float vl)
{
    const float p = __fmul_rn(k, vh);
    const float e = __fmaf_rn(k, vh, -p);
    const float t = __fadd_rn(a.s, p);
    const float bp = __fsub_rn(t, a.s);
    const float err = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
    a.s = t;
    a.c = __fmaf_rn(k, vl, __fadd_rn(a.c, __fadd_rn(err, e)));
}

// v' of one cell split into FP32 pieces: (hi1, hi2, lo1, lo2), v ~= hi + lo.
__device__ __forceinline__ float4 split_v(double v1, double v2)
{
    const float h1 = (float)v1, h2 = (float)v2;
    return make_float4(h1, h2, (float)(v1 - (double)h1), (float)(v2 - (double)h2));
}

template <int U>   // 64 U sources in flight
__device__ __forceinline__ void rows3_f32(const float2 *__restrict__ K, const float4 *__restrict__ v, int64_t N,
                                          int64_t i, int64_t j0, int64_t j1, int lane, double acc[3])
{
    const float2 *r0 = K + (3 * i) * N, *r1 = r0 + N, *r2 = r1 + N;
    Acc2 a0{0.f, 0.f}, a1{0.f, 0.f}, a2{0.f, 0.f};
    int64_t j = j0 + lane;
#pragma unroll U
    for (; j + 32 < j1; j += 64) {
        const float4 x0 = __ldg(v + j), x1 = __ldg(v + j + 32);
        const float2 k00 = __ldcs(r0 + j), k10 = __ldcs(r1 + j), k20 = __ldcs(r2 + j);
        const float2 k01 = __ldcs(r0 + j + 32), k11 = __ldcs(r1 + j + 32), k21 = __ldcs(r2 + j + 32);
        acc2_add(a0, k00.x, x0.x, x0.z); acc2_add(a0, k00.y, x0.y, x0.w);
        acc2_add(a1, k10.x, x0.x, x0.z); acc2_add(a1, k10.y, x0.y, x0.w);
        acc2_add(a2, k20.x, x0.x, x0.z); acc2_add(a2, k20.y, x0.y, x0.w);
        acc2_add(a0, k01.x, x1.x, x1.z); acc2_add(a0, k01.y, x1.y, x1.w);
        acc2_add(a1, k11.x, x1.x, x1.z); acc2_add(a1, k11.y, x1.y, x1.w);
        acc2_add(a2, k21.x, x1.x, x1.z); acc2_add(a2, k21.y, x1.y, x1.w);
    }
    for (; j < j1; j += 32) {
        const float4 x0 = __ldg(v + j);
        const float2 k00 = __ldcs(r0 + j), k10 = __ldcs(r1 + j), k20 = __ldcs(r2 + j);
        acc2_add(a0, k00.x, x0.x, x0.z); acc2_add(a0, k00.y, x0.y, x0.w);
        acc2_add(a1, k10.x, x0.x, x0.z); acc2_add(a1, k10.y, x0.y, x0.w);
        acc2_add(a2, k20.x, x0.x, x0.z); acc2_add(a2, k20.y, x0.y, x0.w);
    }
    acc[0] = warp_sum((double)a0.s + (double)a0.c);
    acc[1] = warp_sum((double)a1.s + (double)a1.c);
    acc[2] = warp_sum((double)a2.s + (double)a2.c);
}

// The three sums of receiver i by S neighbouring warps of a block of 8 (each a
// contiguous part of the sources, the parts added in order); valid in lane 0
// of the first.  A warp has two rounds of loads in flight, so a small operator
// (in L2) needs more than N warps to keep the FP64 pipe fed: N = 1,600 with S =
// 1 (11 warps per SM) 46.9 us, S = 2 39.1 us, against 24.5 us of multiply-adds.
template <bool kF32, int S, int U>
__device__ __forceinline__ void receiver_rows(const void *K, const void *v, int64_t N, int64_t i, double acc[3])
{
    __shared__ double part[8][3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = w % S;
    const int64_t len = (N + 32 * S - 1) / (32 * S) * 32, j0 = p * len, j1 = min(N, j0 + len);
    if (i < N) {
        if (kF32) rows3_f32<U>((const float2 *)K, (const float4 *)v, N, i, j0, j1, lane, acc);
        else rows3_f64((const double2 *)K, (const double2 *)v, N, i, j0, j1, lane, acc);
    }
    if (S == 1) return;
    if (lane == 0) { part[w][0] = acc[0]; part[w][1] = acc[1]; part[w][2] = acc[2]; }
    __syncthreads();
    if (p == 0)
        for (int q = 1; q < S; ++q)
            for (int c = 0; c < 3; ++c) acc[c] += part[w + q][c];
}

// How a product is launched: S warps per receiver (1, 2 or 4), and for the FP32
// operator the blocks that an SM holds (2 with 256 sources in flight a warp, 3 with
// the same in fewer registers, 4 with 64).
struct RowShape {
    int s, r;
};

// b: an SM's blocks of 8 receivers.  Up to two of them the warps per receiver are
// those for which the busiest SM's blocks times a block's time (its sources and
// about 200 more for its start and sums) is least; more, and none are split
// (FP64), since blocks come and go.  The FP32 operator is bound by the loads in
// flight, and its blocks are best all resident at once: three and four take the
// builds that allow it, and from five on two warps per receiver even out the last
// round of blocks where it is less than two thirds full.  us (one warp per receiver
// and 2 blocks per SM / as chosen; a step at N = 6,500 237 us, split 242):
// FP64 N = 400 8.1 / 6.2, 1,000 18.3 / 18.3 (with 4 warps 23.4), 1,600 43.6 / 37.4;
// FP32 N = 304 4.8 / 4.0, 2,500 37.9 / 29.6, 3,000 52.0 / 38.0, 4,000 70.1 / 65.6,
// 5,000 120 / 105, 8,000 259 / 249, 20,000 1,458 / 1,401.
static RowShape row_shape(int64_t N, bool f32, int sms)
{
    const int64_t b = (N + 8 * sms - 1) / (8 * (int64_t)sms);
    if (b > 2) {
        if (!f32) return RowShape{1, 2};
        if (b <= 4) return RowShape{1, (int)b};
        const int64_t round = 2 * sms, last = ((N + 7) / 8 - 1) % round + 1;
        return 3 * last < 2 * round ? RowShape{2, 3} : RowShape{1, 2};
    }
    int best = 1;
    int64_t cost = INT64_MAX;
    for (int s = 1; s <= 4 && 32 * (s - 1) < N; s *= 2) {   // none without sources
        const int64_t blocks = (N * s + 7) / 8, c = (blocks + sms - 1) / sms * (N / s + 200);
        if (c < cost) { cost = c; best = s; }
    }
    return RowShape{best, 2};
}

// the builds' registers (FP64: the compiler's own choice) and loads in flight
#define PQ3D_ROWS_BOUNDS __launch_bounds__(256, kF32 ? R : 0)
template <int R>
constexpr int kRowsUnroll = R == 4 ? 1 : 4;

template <bool kF32, int S, int R>
__global__ void PQ3D_ROWS_BOUNDS matvec_kernel(const void *__restrict__ K, const void *__restrict__ v,
                                                     int64_t N, double *__restrict__ out)
{
    const int64_t i = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) / S;
    double acc[3];
    receiver_rows<kF32, S, kRowsUnroll<R>>(K, v, N, i, acc);
    if (i < N && (threadIdx.x & 31) == 0 && (threadIdx.x >> 5) % S == 0) {
        out[3 * i] = acc[0];
        out[3 * i + 1] = acc[1];
        out[3 * i + 2] = acc[2];
    }
}

// ---------------------------------------------------------------------------
// pore-pressure dilatancy (src/QDsim_gpu.py:611-671)

constexpr int kMaxDepth = 64;   // tridiagonal unknowns per cell (the reference uses 59)

// table layout (pq3d_dilatancy_table): lower, diag, upper of the diffusion
// matrix (n each; M = dt * this + I), then the scalars below
enum DilaScalar { D_BC0, D_BCN, D_G, D_T1, D_T2, D_TG, D_DP, D_NSCAL };

// One implicit step for the cells [cell0, cell1) of this block (called by all
// threads of every block with the same h): the Thomas factorisation of M is formed once
// per block in shared memory (M is diagonally dominant by rows, so no
// pivoting is needed; the reference factorises with partial pivoting).
__device__ __noinline__ void dilatancy_step(const pq3d_dense_sim &S, double h, double *cp, double *inv, int64_t cell0,
                                            int64_t cell1)
{
    const int n = S.ndepth;
    const double *lo = S.dila, *di = lo + n, *up = di + n, *sc = up + n;
    __syncthreads();
    if (threadIdx.x == 0) {
        double prev = 0.0;
        for (int k = 0; k < n; ++k) {
            const double den = (1.0 + di[k] * h) - (k ? lo[k] * h * prev : 0.0);
            inv[k] = 1.0 / den;
            prev = (k + 1 < n) ? up[k] * h * inv[k] : 0.0;
            cp[k] = prev;
        }
    }
    __syncthreads();
    const int64_t N = S.N;
    for (int64_t i = cell0 + threadIdx.x; i < cell1; i += blockDim.x) {
        const double theta = S.dc[i] / S.V0 * exp((S.state[i] - S.f0[i]) / S.b[i]);
        const double dthetadt = 1.0 - S.slipv[i] * theta / S.dc[i];
        const double g = -sc[D_G] / theta * dthetadt;
        double *col = S.Parr + i;   // Parr[k * N + i]
        // forward sweep: d'_k into Parr
        double dprev = 0.0;
        for (int k = 0; k < n; ++k) {
            double b = col[k * N];
            if (k == 0) b -= sc[D_BC0] * g * h;
            if (k == n - 1) b += h * sc[D_BCN];
            const double d = (b - (k ? lo[k] * h * dprev : 0.0)) * inv[k];
            col[k * N] = d;
            dprev = d;
        }
        // back substitution
        double x = dprev;
        for (int k = n - 2; k >= 0; --k) {
            x = col[k * N] - cp[k] * x;
            col[k * N] = x;
        }
        const double x0 = col[0], x1 = col[N];
        const double term1 = -sc[D_T1] * (x0 - x1 + sc[D_TG] * g);
        const double term2 = sc[D_T2] * (x1 - x0);
        S.dPdt[i] = sc[D_DP] * (term1 + term2);
        S.P[i] = x0;
    }
}

// v' of every cell from its current slip rate (src/QDsim_gpu.py:948-949); the
// FP32 operator takes it as its hi/lo FP32 split
template <bool kF32>
__global__ void __launch_bounds__(256) vprime_kernel(pq3d_dense_sim S)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= S.N) return;
    const double v1 = S.slipv1[i] - S.Vpl * cos(S.rake0[i]), v2 = S.slipv2[i] - S.Vpl * sin(S.rake0[i]);
    if (kF32) reinterpret_cast<float4 *>(S.vprime)[i] = split_v(v1, v2);
    else reinterpret_cast<double2 *>(S.vprime)[i] = make_double2(v1, v2);
}

// (1) traction rates of one step (src/QDsim_gpu.py:948-957): the normal
// component with the normal loading added (or the loading alone with fix_Tn)
template <bool kF32, int S, int R>
__global__ void PQ3D_ROWS_BOUNDS step_rates_kernel(pq3d_dense_sim D)
{
    const int64_t i = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) / S;
    double acc[3];
    receiver_rows<kF32, S, kRowsUnroll<R>>(kF32 ? (const void *)D.K32 : (const void *)D.K64, D.vprime, D.N, i, acc);
    if (i < D.N && (threadIdx.x & 31) == 0 && (threadIdx.x >> 5) % S == 0) {
        D.rates[3 * i] = acc[0];
        D.rates[3 * i + 1] = acc[1];
        D.rates[3 * i + 2] = D.fix_Tn ? D.normal_loading[i] : acc[2] + D.normal_loading[i];
    }
}

// (2)-(3) the rest of one accepted step, one cooperative launch: attempts
// until one is accepted (grid barrier per attempt for the error norms; every
// thread takes the same decision), the state update with v' for the next
// product, the dilatancy step.  `step` indexes h_hist / t_hist / h_force.
//
// Bound (small meshes): one chain of FP64 latency per cell.  N = 1,600: 133 us
// with the reference formula's 15 divisions and 6 exponentials per right-hand
// side, two pow calls by every thread of the grid (16 warps per SM through a
// pipe of 2 lanes per clock) and a microsecond between looks at the barrier;
// 77 us with the reciprocal form, the pow calls by two threads of a block and
// one block per SM (a second one's warps would share its FP64 pipe); 42 us with
// four lanes per cell (kQuad: one cell per four threads, its candidate state
// in their registers).
template <bool kF32, bool kQuad>
__global__ void __launch_bounds__(256) dense_attempt_kernel(pq3d_dense_sim S, int step, double *h_hist, double *t_hist,
                                                            const double *h_force)
{
    __shared__ unsigned long long red[32];
    __shared__ double dil_cp[kMaxDepth], dil_inv[kMaxDepth];
    __shared__ double s_c[2], s_hn[2];
    pq3d_step_ctrl *C = S.ctrl;
    // read before the first grid barrier (the lead changes them only after it)
    if (*(volatile int32_t *)&C->status != PQ3D_OK) return;   // same for every block
    const double dttry = *(volatile double *)&C->dttry, time = *(volatile double *)&C->time;
    int64_t attempt = *(volatile int64_t *)&C->attempts;      // rotates the error slots
    const int64_t N = S.N;
    const bool lead = (blockIdx.x == 0 && threadIdx.x == 0);
    unsigned *bc = &C->bar_count, *bg = &C->bar_gen;
    const unsigned nb = gridDim.x;
    double2 *vp = (double2 *)S.vprime;
    float4 *vs = (float4 *)S.vprime;
    // cells of this block: a contiguous share of N / gridDim, so that every SM
    // gets cells (N is often below the grid's thread count)
    const int64_t chunk = (N + nb - 1) / nb;
    const int64_t cell0 = (int64_t)blockIdx.x * chunk, cell1 = cell0 + chunk < N ? cell0 + chunk : N;
    if (lead) C->maxv_bits = 0ull;   // the update's atomicMax comes after at least one grid barrier

    // kQuad: this thread's cell and variable (tau1, tau2, psi, sigma); lanes
    // past the last cell shadow it
    const int var = threadIdx.x & 3;
    const int64_t ic = cell0 + (threadIdx.x >> 2);
    const bool mine = ic < cell1;
    const int64_t iq = mine ? ic : (cell1 > cell0 ? cell1 - 1 : 0);
    double *const state_of = var == 0 ? S.Tt1o : (var == 1 ? S.Tt2o : (var == 2 ? S.state : S.Tno));
    double yq = 0.0;

    // (2) attempts until one is accepted
    double h = h_force ? h_force[step] : dttry, dtnext = 0.0;
    int nrjct = 0;
    for (;;) {
        const int slot = (int)(attempt % 3);
        double m1 = 0.0, m2 = 0.0;
        if (kQuad) {
            if ((threadIdx.x & ~31) < 4 * (cell1 - cell0)) {   // warps with a cell
                const Cell c{S.a[iq], S.b[iq], S.dc[iq], S.f0[iq], S.shear_loading[iq], S.slipv[iq], 0.0, 0.0,
                             S.rates[3 * iq + 2], S.P ? S.P[iq] : 0.0, S.dPdt ? S.dPdt[iq] : 0.0};
                double e;
                dp_attempt_quad(c, var, var < 2 ? S.rates[3 * iq + var] : 0.0, S.V0, S.eta, h, state_of[iq], yq, e);
                if (mine) (var == 2 ? m1 : m2) = e;
            }
        } else
        for (int64_t i = cell0 + threadIdx.x; i < cell1; i += blockDim.x) {
            const Cell c{S.a[i], S.b[i], S.dc[i], S.f0[i], S.shear_loading[i], S.slipv[i],
                         S.rates[3 * i], S.rates[3 * i + 1], S.rates[3 * i + 2],
                         S.P ? S.P[i] : 0.0, S.dPdt ? S.dPdt[i] : 0.0};
            const double y[4] = {S.Tno[i], S.Tt1o[i], S.Tt2o[i], S.state[i]};
            double yo[4], e1, e2;
            dp_attempt<true, true>(c, S.V0, S.eta, h, y, yo, e1, e2);
            reinterpret_cast<double4_16a *>(S.cand)[i] = make_double4_16a(yo[0], yo[1], yo[2], yo[3]);
            m1 = (isnan(m1) || isnan(e1)) ? NAN : fmax(m1, e1);
            m2 = (isnan(m2) || isnan(e2)) ? NAN : fmax(m2, e2);
        }
        const unsigned long long b1 = block_max_bits(dbits(m1), red);
        const unsigned long long b2 = block_max_bits(dbits(m2), red);
        if (threadIdx.x == 0) {
            atomicMax((unsigned long long *)&C->err_slot[2 * slot], b1);
            atomicMax((unsigned long long *)&C->err_slot[2 * slot + 1], b2);
        }
        if (!grid_barrier(bc, bg, nb)) { if (threadIdx.x == 0) C->status = PQ3D_ERR_TIMEOUT; return; }
        if (threadIdx.x < 2) {
            const double err =
                __longlong_as_double((long long)*((volatile unsigned long long *)&C->err_slot[2 * slot + threadIdx.x])) + 1e-10;
            s_c[threadIdx.x] = err / kRelTol;
            s_hn[threadIdx.x] = h * 0.9 * pow(kRelTol / err, 0.2);
        }
        __syncthreads();
        if (lead) {
            // the slot of the attempt before this one: every thread has read it
            const int z = (int)((attempt + 2) % 3);
            C->err_slot[2 * z] = 0ull;
            C->err_slot[2 * z + 1] = 0ull;
            C->attempts += 1;
        }
        ++attempt;
        const double c1 = s_c[0], c2 = s_c[1], hn1 = s_hn[0], hn2 = s_hn[1];
        if (h_force || (fmax(c1, c2) < 1.0 && !(isnan(c1) || isnan(c2)))) {
            dtnext = pymin(1.5 * h, pymin(hn1, hn2));
            break;
        }
        ++nrjct;
        h = pymax(0.5 * h, pymin(hn1, hn2));
        if (h < 1.e-15 || nrjct > 20) {
            if (lead) { C->status = PQ3D_ERR_STEP; C->dttry = h; C->time = time; }
            return;
        }
    }

    // (3) state update (src/QDsim_gpu.py:994-1027)
    double vmax = 0.0;
    if (kQuad) {
        if ((threadIdx.x & ~31) < 4 * (cell1 - cell0)) {
            const double st = __shfl_sync(0xffffffffu, yq, 2, 4), Tno = __shfl_sync(0xffffffffu, yq, 3, 4);
            const double a = S.a[iq];
            const double vk = (2.0 * S.V0) * exp(-st / a) * sinh(yq / Tno / a);   // lanes 0, 1
            const double T1 = __shfl_sync(0xffffffffu, yq, 0, 4), T2 = __shfl_sync(0xffffffffu, yq, 1, 4);
            const double v1 = __shfl_sync(0xffffffffu, vk, 0, 4), v2 = __shfl_sync(0xffffffffu, vk, 1, 4);
            // |tau| and |V| on two lanes; the slips and their length
            const double p = var == 0 ? T1 : v1, q = var == 0 ? T2 : v2;
            const double len = sqrt(p * p + q * q);
            const double Tt = __shfl_sync(0xffffffffu, len, 0, 4);
            double v = __shfl_sync(0xffffffffu, len, 1, 4);
            if (v < 1e-30) v = 1e-30;
            double *const slip_of = var == 0 ? S.slip1 : S.slip2;
            const double sk = var < 2 ? slip_of[iq] + vk * h : 0.0;
            const double s1 = __shfl_sync(0xffffffffu, sk, 0, 4), s2 = __shfl_sync(0xffffffffu, sk, 1, 4);
            double sr, cr;
            sincos(S.rake0[iq], &sr, &cr);
            const double wk = vk - S.Vpl * (var == 0 ? cr : sr);
            const double w1 = __shfl_sync(0xffffffffu, wk, 0, 4), w2 = __shfl_sync(0xffffffffu, wk, 1, 4);
            if (mine) {
                state_of[iq] = yq;
                if (var < 2) {
                    (var == 0 ? S.slipv1 : S.slipv2)[iq] = vk;
                    slip_of[iq] = sk;
                }
                if (var == 0) {
                    S.slipv[iq] = v;
                    S.slip[iq] = sqrt(s1 * s1 + s2 * s2);
                    if (kF32) vs[iq] = split_v(w1, w2);
                    else vp[iq] = make_double2(w1, w2);
                } else if (var == 1) {
                    S.Tt[iq] = Tt;
                    S.fric[iq] = S.P ? Tt / (Tno - S.P[iq] * 1e-6) : Tt / Tno;   // pressure before its update
                } else if (var == 2) {
                    S.rake[iq] = atan2(v2, v1);
                }
                vmax = isnan(v) ? NAN : v;
            }
        }
    } else
    for (int64_t i = cell0 + threadIdx.x; i < cell1; i += blockDim.x) {
        const double4_16a y = reinterpret_cast<const double4_16a *>(S.cand)[i];
        const double Tno = y.x, T1 = y.y, T2 = y.z, st = y.w, a = S.a[i];
        S.Tno[i] = Tno; S.Tt1o[i] = T1; S.Tt2o[i] = T2; S.state[i] = st;
        S.Tt[i] = sqrt(T1 * T1 + T2 * T2);
        const double e = (2.0 * S.V0) * exp(-st / a);
        const double v1 = e * sinh(T1 / Tno / a);
        const double v2 = e * sinh(T2 / Tno / a);
        double v = sqrt(v1 * v1 + v2 * v2);
        S.slipv1[i] = v1; S.slipv2[i] = v2;
        S.rake[i] = atan2(v2, v1);
        if (v < 1e-30) v = 1e-30;
        S.slipv[i] = v;
        vmax = (isnan(vmax) || isnan(v)) ? NAN : fmax(vmax, v);
        const double s1 = S.slip1[i] + v1 * h, s2 = S.slip2[i] + v2 * h;
        S.slip1[i] = s1; S.slip2[i] = s2;
        S.slip[i] = sqrt(s1 * s1 + s2 * s2);
        S.fric[i] = S.P ? S.Tt[i] / (Tno - S.P[i] * 1e-6) : S.Tt[i] / Tno;   // pressure before its update
        double sr, cr;
        sincos(S.rake0[i], &sr, &cr);
        const double w1 = v1 - S.Vpl * cr, w2 = v2 - S.Vpl * sr;
        if (kF32) vs[i] = split_v(w1, w2);
        else vp[i] = make_double2(w1, w2);
    }
    const unsigned long long bv = block_max_bits(dbits(vmax), red);
    if (threadIdx.x == 0) atomicMax((unsigned long long *)&C->maxv_bits, bv);
    // (3b) pore-pressure diffusion of every cell with the new state and
    // slip rate (src/QDsim_gpu.py:628-671, after the update 1119-1120)
    if (S.Parr) dilatancy_step(S, h, dil_cp, dil_inv, cell0, cell1);
    // the last block to get here closes the step (no barrier: nobody waits;
    // bar_count is 0 again since the attempt's barrier)
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(bc, 1u) + 1u == nb) {
            __threadfence();
            *(volatile unsigned *)bc = 0u;
            if (h_hist) h_hist[step] = h;
            if (t_hist) t_hist[step] = time + h;
            C->steps_done += 1;
            C->dttry = dtnext;
            C->time = time + h;
            C->maxv = __longlong_as_double((long long)*(volatile unsigned long long *)&C->maxv_bits);
        }
    }
}

}  // namespace step
}  // namespace pq3d

extern "C" size_t pq3d_dilatancy_table_len(int ndepth) { return ndepth > 0 ? (size_t)3 * ndepth + pq3d::step::D_NSCAL : 0; }

// The reference's matrix (src/QDsim_gpu.py:611-626) and right-hand-side
// constants (628-671) for depth nodes z[0..ndepth].
extern "C" int pq3d_dilatancy_table(const double *z, int ndepth, double c_hyd, double dilatancy, double thickness,
                                    double compressibility, double P0, double *out)
{
    using namespace pq3d;
    using namespace pq3d::step;
    clear_error();
    PQ3D_REQUIRE(z && out && ndepth >= 2 && ndepth <= kMaxDepth, "pq3d_dilatancy_table: bad arguments (ndepth %d)",
                 ndepth);
    const int n = ndepth;
    double *lo = out, *di = lo + n, *up = di + n, *sc = up + n;
    for (int i = 0; i < n; ++i) {
        const double dz = z[i + 1] - z[i];
        const double em = exp(-(2 * z[i] - dz / 2)), ep = exp(-(2 * z[i] + dz / 2));
        if (i == 0) {
            di[0] = c_hyd * (em + ep) / (dz * dz);
            up[0] = -c_hyd * (em + ep) / (dz * dz);
            lo[0] = 0.0;
        } else {
            di[i] = c_hyd * (em + ep) / (dz * dz);
            up[i] = (i + 1 < n) ? -c_hyd * ep / (dz * dz) : 0.0;
            lo[i] = -c_hyd * em / (dz * dz);
        }
    }
    const double dz0 = z[1] - z[0], dzl = z[n] - z[n - 1];
    sc[D_BC0] = 2.0 * c_hyd * exp(-(z[0] - dz0 / 2)) / dz0;
    sc[D_BCN] = 1.0 / (dzl * dzl) * c_hyd * exp(-(z[n - 1] - dzl / 2)) * P0;
    sc[D_G] = dilatancy * thickness / (2.0 * compressibility * c_hyd);
    sc[D_T1] = exp(-(z[0] - dz0 / 2));
    sc[D_T2] = exp(-(z[0] + dz0 / 2));
    sc[D_TG] = 2 * dz0 * exp(z[0]);
    sc[D_DP] = c_hyd * exp(-z[0]) / (dz0 * dz0);
    return PQ3D_OK;
}

namespace pq3d {
namespace step {

struct LaunchCfg {
    int device = -1;
    int sms = 0, grid64 = 0, grid32 = 0;
};
static thread_local LaunchCfg g_cfg;

static int launch_cfg(LaunchCfg **out)
{
    int dev;
    PQ3D_CUDA_TRY(cudaGetDevice(&dev));
    if (g_cfg.device != dev) {
        int sms = 0, coop = 0, b64 = 0, b32 = 0;
        PQ3D_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        PQ3D_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        if (!coop) return set_error(PQ3D_ERR_UNSUPPORTED, "device has no cooperative launch");
        int q64 = 0, q32 = 0;
        PQ3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b64, dense_attempt_kernel<false, false>, 256, 0));
        PQ3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b32, dense_attempt_kernel<true, false>, 256, 0));
        PQ3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q64, dense_attempt_kernel<false, true>, 256, 0));
        PQ3D_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q32, dense_attempt_kernel<true, true>, 256, 0));
        if (b64 < 1 || b32 < 1 || q64 < 1 || q32 < 1) return set_error(PQ3D_ERR_UNSUPPORTED, "stepper kernel does not fit on an SM");
        g_cfg.device = dev;
        g_cfg.sms = sms;
        g_cfg.grid64 = sms * b64;
        g_cfg.grid32 = sms * b32;
    }
    *out = &g_cfg;
    return PQ3D_OK;
}

// Blocks of the attempt kernel: one per SM while its 256 threads hold the
// SM's cells, else all that are resident.
static int attempt_grid(const LaunchCfg &c, bool f32, int64_t N)
{
    return N <= 256 * (int64_t)c.sms ? c.sms : (f32 ? c.grid32 : c.grid64);
}

// Four lanes per cell up to this many cells per SM (one block's 256 threads
// would hold 64): there a warp per SM and cell count of 32 is as much work for
// the FP64 pipe as four warps of quads, whose chains are three times shorter.
constexpr int64_t kQuadCells = 32;

// kernel<kF32, S, R> of a shape
#define PQ3D_ROWS_LAUNCH(kernel, shape, N, st, ...)                                                        \
    do {                                                                                                   \
        const unsigned blocks_ = (unsigned)(((N) * (shape).s + 7) / 8);                                    \
        if (!kF32 || (shape).r == 2) {                                                                     \
            if ((shape).s == 1) kernel<kF32, 1, 2><<<blocks_, 256, 0, st>>>(__VA_ARGS__);                  \
            else if ((shape).s == 2) kernel<kF32, 2, 2><<<blocks_, 256, 0, st>>>(__VA_ARGS__);             \
            else kernel<kF32, 4, 2><<<blocks_, 256, 0, st>>>(__VA_ARGS__);                                 \
        } else if constexpr (kF32) {                                                                       \
            if ((shape).r == 4) kernel<true, 1, 4><<<blocks_, 256, 0, st>>>(__VA_ARGS__);                  \
            else if ((shape).s == 1) kernel<true, 1, 3><<<blocks_, 256, 0, st>>>(__VA_ARGS__);             \
            else kernel<true, 2, 3><<<blocks_, 256, 0, st>>>(__VA_ARGS__);                                 \
        }                                                                                                  \
    } while (0)

template <bool kF32>
static void launch_rates(const pq3d_dense_sim &S, RowShape shape, cudaStream_t st)
{
    PQ3D_ROWS_LAUNCH(step_rates_kernel, shape, S.N, st, S);
}

template <bool kF32>
static void launch_matvec(const void *K, const void *v, int64_t N, RowShape shape, double *out, cudaStream_t st)
{
    PQ3D_ROWS_LAUNCH(matvec_kernel, shape, N, st, K, v, N, out);
}

}  // namespace step
}  // namespace pq3d

using namespace pq3d;
using namespace pq3d::step;

static int matvec(const void *K, int64_t N, const void *v, double *out, void *stream, bool f32)
{
    clear_error();
    PQ3D_REQUIRE(N > 0 && K && v && out, "pq3d_dense_matvec: bad arguments");
    PQ3D_REQUIRE(aligned16(v) && (f32 ? ((uintptr_t)K & 7u) == 0 : aligned16(K)),
                 "pq3d_dense_matvec: K and v must be aligned (16 bytes for FP64, 8 for FP32)");
    LaunchCfg *cfg;
    const int rc = launch_cfg(&cfg);
    if (rc) return rc;
    const RowShape shape = row_shape(N, f32, cfg->sms);
    if (f32) launch_matvec<true>(K, v, N, shape, out, (cudaStream_t)stream);
    else launch_matvec<false>(K, v, N, shape, out, (cudaStream_t)stream);
    PQ3D_CUDA_TRY(cudaGetLastError());
    return PQ3D_OK;
}

extern "C" int pq3d_dense_matvec_f64(const double *K64, int64_t N, const double *v, double *out, void *stream)
{
    return matvec(K64, N, v, out, stream, false);
}

extern "C" int pq3d_dense_matvec_f32(const float *K32, int64_t N, const float *vsplit, double *out, void *stream)
{
    return matvec(K32, N, vsplit, out, stream, true);
}

extern "C" int pq3d_dense_step(const pq3d_dense_sim *sim, int nsteps, double *h_hist, double *t_hist,
                               const double *h_force, void *stream)
{
    clear_error();
    PQ3D_REQUIRE(sim && sim->N > 0 && nsteps >= 0 && sim->ctrl, "pq3d_dense_step: bad arguments");
    PQ3D_REQUIRE((sim->K64 != nullptr) != (sim->K32 != nullptr), "pq3d_dense_step: exactly one of K64/K32");
    PQ3D_REQUIRE(aligned16(sim->vprime) && aligned16(sim->cand) && aligned16(sim->K64 ? (const void *)sim->K64
                                                                                      : (const void *)sim->K32),
                 "pq3d_dense_step: vprime, cand and K must be 16-byte aligned");
    if (sim->Parr)
        PQ3D_REQUIRE(sim->P && sim->dPdt && sim->dila && sim->ndepth >= 2 && sim->ndepth <= kMaxDepth,
                     "pq3d_dense_step: dilatancy needs P, dPdt, dila and 2 <= ndepth <= %d", kMaxDepth);
    if (nsteps == 0) return PQ3D_OK;
    const bool f32 = sim->K32 != nullptr;
    LaunchCfg *cfg;
    const int rc = launch_cfg(&cfg);
    if (rc) return rc;
    const int grid = attempt_grid(*cfg, f32, sim->N);
    const RowShape shape = row_shape(sim->N, f32, cfg->sms);
    // clear the reduction slots and the barrier counter of the control block
    cudaStream_t st = (cudaStream_t)stream;
    PQ3D_CUDA_TRY(cudaMemsetAsync(&sim->ctrl->err_slot[0], 0, sizeof(uint64_t) * 7 + sizeof(uint32_t), st));
    pq3d_dense_sim S = *sim;
    const unsigned cell_blocks = (unsigned)((sim->N + 255) / 256);
    if (f32) vprime_kernel<true><<<cell_blocks, 256, 0, st>>>(S);
    else vprime_kernel<false><<<cell_blocks, 256, 0, st>>>(S);
    PQ3D_CUDA_TRY(cudaGetLastError());
    const bool quad = S.N <= kQuadCells * cfg->sms;
    const void *attempt = f32 ? (quad ? (const void *)dense_attempt_kernel<true, true>
                                      : (const void *)dense_attempt_kernel<true, false>)
                              : (quad ? (const void *)dense_attempt_kernel<false, true>
                                      : (const void *)dense_attempt_kernel<false, false>);
    int step = 0;
    void *args[] = {(void *)&S, (void *)&step, (void *)&h_hist, (void *)&t_hist, (void *)&h_force};
    for (; step < nsteps; ++step) {
        if (f32) launch_rates<true>(S, shape, st);
        else launch_rates<false>(S, shape, st);
        PQ3D_CUDA_TRY(cudaGetLastError());
        PQ3D_CUDA_TRY(cudaLaunchCooperativeKernel(attempt, grid, 256, args, 0, st));
    }
    return PQ3D_OK;
}
