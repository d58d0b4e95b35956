// ntlp_stats.cu -- particle_xy_stats (particles.f90:3370-3770) and
// radius_histogram (:5011-5021) over one box's cell-sorted droplets.
//
// Deterministic reductions without floating-point atomics.  The columns
// (ipt, jpt) of the cell key are contiguous ranges of the sorted list.
//   k_stats_columns  a warp per column, lanes striding through its droplets
//            (cell order, lid order within a cell): counts, the six 0th-order
//            sums, extrema, the column's LWP and the radius histogram (integer
//            weights, shared-memory int64 bins); a block's warps take
//            kStatCols columns and leave one partial;
//   k_stats_levels   a warp per 32 stats levels L = minloc(z > xp3) - 1 and
//            every kStatWarps-th column of a block's kStatCols: a lane sums its
//            level's 24 quantities over the two cells (kuv = L-1, L) that can
//            hold its droplets;
//   k_stats_reduce   the block partials, interleaved over kStatWarps threads
//            per value and then added in thread order.
// Every sum therefore has a fixed order (not the list order of the
// reference); counts and extrema are exact.
//
// Bound by latency: about 13 gathered doubles a droplet, twice, and little
// arithmetic, so what counts is how many droplets are in flight.  Blocks of 128
// columns with a thread per column and a thread per level kept 130 blocks
// half busy: 0.72 ms for 1 M droplets on 128^3; five steps with statistics
// went from 14.1 to 11.3 ms.
#include <cuda_runtime.h>

#include "../../include/ntlp_gpu.h"
#include "ntlp_dev.cuh"
#include "ntlp_kernels.h"

namespace ntlp {

namespace {

// 0th-order partial: [0] numpart, [1] numdrop, [2..7] sums (Rep, Volp*rhow,
// Volp*rhop, Volp, radius, radius^2), [8..13] max (radius, Tp, qinf, vp1..3),
// [14..19] min (same order)
constexpr int kS0Count = 0, kS0Drop = 1, kS0Sum = 2, kS0Max = 8, kS0Min = 14;

__device__ __forceinline__ void s0_init(double *a) {
    for (int q = 0; q < kS0Max; ++q) a[q] = 0.0;
    for (int q = 0; q < 6; ++q) {
        a[kS0Max + q] = -ntlp_inf();
        a[kS0Min + q] = ntlp_inf();
    }
}

// combines partial w into v, quantity q of the 0th-order values
__device__ __forceinline__ double s0_join(int q, double v, double w) {
    return q < kS0Max ? v + w : (q < kS0Min ? fmax(v, w) : fmin(v, w));
}

__global__ void __launch_bounds__(kStatThreads)
k_stats_columns(const DevBox *boxes, int box, const DevParams *pp, double *tile0, double *colsum, long long *hrad) {
    const DevBox &B = boxes[box];
    const DevParams &p = pp[0];
    const DevGrid &g = B.g;
    const DevState &S = B.st[B.cur];
    const int nz1 = g.nnz + 1;
    const int ncols = (g.nnx + 1) * (g.nny + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ double s_part[kStatWarps][kS0N];
    __shared__ long long s_h[NTLP_HIST_N];
    if (hrad != nullptr) {
        for (int b = threadIdx.x; b < NTLP_HIST_N; b += blockDim.x) s_h[b] = 0;
        __syncthreads();
    }
    const double pi = p.pi2 * 0.5;     // 4*atan(1) (pi2 = 2*(4*atan(1)), les.F)
    double a[kS0N];
    s0_init(a);
    for (int c = warp; c < kStatCols; c += kStatWarps) {
        const int col = blockIdx.x * kStatCols + c;
        if (col >= ncols) break;
        double lwp = 0.0;
        const int lo = B.cell_start[col * nz1], hi = B.cell_start[(col + 1) * nz1];
        for (int at = lo + lane; at < hi; at += 32) {
            const int t = B.perm[at];
            const double r = S.r[t], Tp = S.Tp[t], qinf = S.qinf[t], m_s = S.m_s[t];
            double vp[3], uf[3];
            for (int k = 0; k < 3; ++k) { vp[k] = S.v[k][t]; uf[k] = S.uf[k][t]; }
            const double mult = (double)S.mult[t];
            a[kS0Count] += 1.0;
            if (r > S.rc[t]) a[kS0Drop] += 1.0;
            const double Volp = p.vol * cube(r);
            const double rhop = (m_s + Volp * p.rhow) / Volp;
            const double d0 = vp[0] - uf[0], d1 = vp[1] - uf[1], d2 = vp[2] - uf[2];
            const double diffnorm = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
            const double Rep = 2.0 * r * diffnorm / p.nuf;
            a[kS0Sum + 0] += Rep;
            a[kS0Sum + 1] += Volp * p.rhow;
            a[kS0Sum + 2] += Volp * rhop;
            a[kS0Sum + 3] += Volp;
            a[kS0Sum + 4] += r;
            a[kS0Sum + 5] += r * r;
            const double ext[6] = {r, Tp, qinf, vp[0], vp[1], vp[2]};
            for (int q = 0; q < 6; ++q) {
                a[kS0Max + q] = fmax(a[kS0Max + q], ext[q]);
                a[kS0Min + q] = fmin(a[kS0Min + q], ext[q]);
            }
            lwp += mult * (p.rhow * 4.0 / 3.0 * pi * cube(r));
            if (hrad != nullptr) {
                const int b = ntlp_hist_bin(p.hb[NTLP_H_RADDEATH], ntlp_log10(r));
                atomicAdd((unsigned long long *)&s_h[b], (unsigned long long)S.mult[t]);
            }
        }
        for (int o = 16; o > 0; o >>= 1) lwp += __shfl_xor_sync(0xffffffffu, lwp, o);
        if (lane == 0) colsum[col] = lwp;
    }
#pragma unroll
    for (int q = 0; q < kS0N; ++q) {
        for (int o = 16; o > 0; o >>= 1) a[q] = s0_join(q, a[q], __shfl_xor_sync(0xffffffffu, a[q], o));
        if (lane == 0) s_part[warp][q] = a[q];
    }
    __syncthreads();
    if (threadIdx.x < kS0N) {
        const int q = threadIdx.x;
        double v = s_part[0][q];
        for (int w = 1; w < kStatWarps; ++w) v = s0_join(q, v, s_part[w][q]);
        tile0[(long long)blockIdx.x * kS0N + q] = v;
    }
    if (hrad != nullptr) {
        for (int b = threadIdx.x; b < NTLP_HIST_N; b += blockDim.x)
            if (s_h[b] != 0) atomicAdd((unsigned long long *)&hrad[b], (unsigned long long)s_h[b]);
    }
}

// grid: (column tiles, groups of 32 levels)
__global__ void __launch_bounds__(kStatThreads)
k_stats_levels(const DevBox *boxes, int box, const DevParams *pp, double *tileL) {
    constexpr int Q = NTLP_STATS_LEVEL_QTYS;
    const DevBox &B = boxes[box];
    const DevParams &p = pp[0];
    const DevGrid &g = B.g;
    const DevState &S = B.st[B.cur];
    const int nz1 = g.nnz + 1;
    const int ncols = (g.nnx + 1) * (g.nny + 1);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L = 1 + 32 * blockIdx.y + lane;
    const double pi = p.pi2 * 0.5;
    __shared__ double s_part[kStatWarps][Q][32];
    double acc[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) acc[q] = 0.0;
    if (L <= g.nnz) {
        const double zlo = g.z[L - 1], zhi = g.z[L];
        for (int c = warp; c < kStatCols; c += kStatWarps) {
            const int col = blockIdx.x * kStatCols + c;
            if (col >= ncols) break;
            // cells L-1 and L of the column are neighbours in the list
            const int key = L - 1 + nz1 * col;
            const int lo = B.cell_start[key], hi = B.cell_start[key + 2];
            for (int at = lo; at < hi; ++at) {
                const int t = B.perm[at];
                const double x3 = S.x[2][t];
                if (!(zlo <= x3 && x3 < zhi)) continue;
                const double v1 = S.v[0][t], v2 = S.v[1][t], v3 = S.v[2][t];
                const double u1 = S.uf[0][t], u2 = S.uf[1][t], u3 = S.uf[2][t];
                const double Tp = S.Tp[t], r = S.r[t];
                const double mult = (double)S.mult[t];
                acc[0] += 1.0;
                acc[1] += v1; acc[2] += v2; acc[3] += v3;
                acc[4] += v1 * v1; acc[5] += v2 * v2; acc[6] += v3 * v3;
                acc[7] += v1 * v3;
                acc[8] += u1; acc[9] += u2; acc[10] += u3;
                acc[11] += u1 * u1; acc[12] += u2 * u2; acc[13] += u3 * u3;
                acc[14] += Tp; acc[15] += Tp * Tp; acc[16] += S.Tf[t];
                acc[17] += r; acc[18] += r * r;
                acc[19] += S.qinf[t];
                acc[20] += Tp * v3;
                acc[21] += mult;
                acc[22] += mult * (p.rhow * 4.0 / 3.0 * pi * cube(r));
                acc[23] += S.qstar[t];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) s_part[warp][q][lane] = acc[q];
    __syncthreads();
    for (int e = threadIdx.x; e < Q * 32; e += kStatThreads) {
        const int q = e / 32, l = 32 * blockIdx.y + e % 32;
        if (l >= g.nnz) continue;
        double v = s_part[0][q][e % 32];
        for (int w = 1; w < kStatWarps; ++w) v = v + s_part[w][q][e % 32];
        tileL[((long long)blockIdx.x * Q + q) * g.nnz + l] = v;
    }
}

// tile partials -> box totals: 32 values a block, the tiles interleaved over
// kStatWarps threads per value; the last block takes the 0th-order values
__global__ void __launch_bounds__(kStatThreads)
k_stats_reduce(int ntiles, int nnz, const double *tile0, const double *tileL, double *out0, double *outL) {
    __shared__ double s_part[kStatWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool zeroth = blockIdx.x == gridDim.x - 1;
    const int n = zeroth ? kS0N : NTLP_STATS_LEVEL_QTYS * nnz;
    const int e = (zeroth ? 0 : 32 * (int)blockIdx.x) + lane;
    const double *part = zeroth ? tile0 : tileL;
    const int op = zeroth ? e : 0;      // level sums add, as the first 0th-order values do
    double v = op < kS0Max ? 0.0 : (op < kS0Min ? -ntlp_inf() : ntlp_inf());
    if (e < n) {
#pragma unroll 4
        for (int k = warp; k < ntiles; k += kStatWarps) v = s0_join(op, v, part[(long long)k * n + e]);
    }
    s_part[warp][lane] = v;
    __syncthreads();
    if (warp == 0 && e < n) {
        for (int w = 1; w < kStatWarps; ++w) v = s0_join(op, v, s_part[w][lane]);
        (zeroth ? out0 : outL)[e] = v;
    }
}

}  // namespace

int stats_tile_count(const DevGrid &g) { return ((g.nnx + 1) * (g.nny + 1) + kStatCols - 1) / kStatCols; }

void launch_stats(const DevBox *boxes, int box, const DevGrid &g, const DevParams *pp, const StatsScratch &w,
                  bool radius_hist, cudaStream_t st) {
    const int nt = stats_tile_count(g);
    if (radius_hist) cudaMemsetAsync(w.hrad, 0, sizeof(long long) * NTLP_HIST_N, st);
    k_stats_columns<<<nt, kStatThreads, 0, st>>>(boxes, box, pp, w.tile0, w.colsum, radius_hist ? w.hrad : nullptr);
    k_stats_levels<<<dim3(nt, (g.nnz + 31) / 32), kStatThreads, 0, st>>>(boxes, box, pp, w.tileL);
    const int n = NTLP_STATS_LEVEL_QTYS * g.nnz;
    k_stats_reduce<<<(n + 31) / 32 + 1, kStatThreads, 0, st>>>(nt, g.nnz, w.tile0, w.tileL, w.out0, w.outL);
}

}  // namespace ntlp
