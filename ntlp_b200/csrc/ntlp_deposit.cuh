// ntlp_deposit.cuh -- deterministic two-way-coupling deposition
// (particle_coupling_update, particles.f90:1151-1276, and the single-domain
// periodic fold of particle_coupling_exchange, :1078-1113).
//
// Every output node sums the contributions of the droplets in its (up to) 8
// neighbouring cells in list order (ascending lid): the cell lists are
// lid-sorted, so each node is an 8-way merge.  Nodes with ix <= 2 or iy <= 2
// also receive their periodic images (ix+nnx, iy+nny), combined in the order
// of the fold (x first, then y).
//
// The tiled kernels stage, per tile of TX x TY x TZ nodes, the droplets of
// the tile's (TX+1)(TY+1)(TZ+1) cells in shared memory (each (x, y) column of
// cells is one contiguous range of the sorted list) and merge from there;
// the periodic images (ix > nnx or iy > nny) are nodes of their own, folded in
// by k_fold.  Tiles holding more droplets than the shared buffer (and, for
// boxes without an image buffer, FP64 tiles on the periodic edges) merge
// straight from global memory.  Both paths perform the same operations in the
// same order.
//
// FP64 (k_deposit64): each contribution is formed as the reference writes it,
// ((P*wtt)/dV)*mult with wtt = wtx*wty*wtz, subtracted term by term.
// Mixed (k_deposit_tiled): the FP32 payload (cell-relative fractions, momentum/heat/
// vapour factors, mult/dV), FP32 weights, FP64 sums, grouped by cell: each
// of the node's 8 cells sums its droplets in list order from zero (S_o),
// and the node adds S_0 .. S_7 in order.  Deterministic, not list order;
// the grouping lets boxes with many droplets per cell form every S_o once
// per cell (k_cellsums32) instead of once per node visit.
#pragma once

#include <cuda_runtime.h>

#include "ntlp_dev.cuh"
#include "ntlp_kernels.h"
#include "ntlp_overflow.h"

namespace ntlp {
namespace {

constexpr int kDepCapMixed = 768;                                 // droplets staged per tile (mixed)
// mixed stage: the six source factors of a droplet in FP64 (signs applied,
// converted once per droplet, not once per node), then fx, fy, fz, mult/dV
constexpr int kStageD = 6, kStageF = 4;

// droplets of a cell sum whose loads are in flight together: 2 M droplets at 31
// per cell with 1 / 2 / 4 / 8: deposition 0.162 / 0.119 / 0.119 / 0.118 ms, 67 M in
// overflow tiles 6.7 / 6.0 / 6.5 / 7.4 ms
constexpr int kSumAhead = 2;

struct DropVals {
    double x1, x2, x3, D[3], V[3], T0, H0, E1, E2, mult;
};

// FP64 contribution, formed as the reference writes it
__device__ __forceinline__ void contribute64(const DevGrid &g, const DevParams &p, const DropVals &d, int kpt,
                                             double xv, double yv, double zv, double acc[6]) {
    const double wtx = (1.0 - fabs(d.x1 - xv) / g.dx);
    const double wty = (1.0 - fabs(d.x2 - yv) / g.dy);
    const double wtz = (1.0 - fabs(d.x3 - zv) / g.dzu[kpt + 1]);
    const double wtt = wtx * wty * wtz;
    const double dV = g.dx * g.dy * g.dzu[kpt + 1];
    if (p.icouple == 1) {
        for (int a = 0; a < 3; ++a) {
            acc[a] = acc[a] - d.D[a] * wtt / dV * d.mult;
            acc[a] = acc[a] - d.V[a] * wtt / dV * d.mult;
        }
    }
    if (p.iTcouple == 1) acc[3] = acc[3] - d.T0 * wtt / dV * d.mult;
    if (p.iHcouple == 1) {
        acc[4] = acc[4] - d.H0 * wtt / dV * d.mult;
        acc[5] = acc[5] - d.E1 * wtt / dV * d.mult + d.E2 * wtt / dV * d.mult;
    }
}

// mixed contribution from the FP32 payload; (i, j, k) is the node's offset
// from the droplet's cell, so the weight along x is fx (i = 1) or 1 - fx
__device__ __forceinline__ void contribute32(const DevParams &p, const float *v, int i, int j, int k,
                                             double acc[6]) {
    const float wx = i ? v[P32_FX] : 1.0f - v[P32_FX];
    const float wy = j ? v[P32_FY] : 1.0f - v[P32_FY];
    const float wz = k ? v[P32_FZ] : 1.0f - v[P32_FZ];
    const double c = (double)(wx * wy * wz * v[P32_FAC]);
    // explicit FMAs: every kernel that forms a cell sum rounds alike
    if (p.icouple == 1)
        for (int a = 0; a < 3; ++a) acc[a] = fma(-(double)v[P32_DV0 + a], c, acc[a]);
    if (p.iTcouple == 1) acc[3] = fma(-(double)v[P32_T0], c, acc[3]);
    if (p.iHcouple == 1) {
        acc[4] = fma(-(double)v[P32_H0], c, acc[4]);
        acc[5] = fma((double)v[P32_E], c, acc[5]);
    }
}

// one cell's sum for corner o = (i, j, k): its droplets (sorted positions
// a..e) in list order, from zero
__device__ __forceinline__ void cell_sum32(const DevBox &B, const DevParams &p, int a, int e, int i, int j, int k,
                                           double S[6]) {
    for (int q = 0; q < 6; ++q) S[q] = 0.0;
    // kSumAhead droplets' loads in flight together
    for (int at = a; at < e; at += kSumAhead) {
        int t[kSumAhead];
        float v[kSumAhead][P32_N];
#pragma unroll
        for (int m = 0; m < kSumAhead; ++m) t[m] = B.perm[min(at + m, e - 1)];
#pragma unroll
        for (int m = 0; m < kSumAhead; ++m) load_payload32(B.pay32, t[m], v[m]);
#pragma unroll
        for (int m = 0; m < kSumAhead; ++m)
            if (at + m < e) contribute32(p, v[m], i, j, k, S);
    }
}

// FP64: merge of up to 8 lid-sorted ranges from global memory through the
// sorted list (positions index B.perm)
__device__ __forceinline__ void merge_ranges(const DevBox &B, const DevParams &p, int n, int pos[8],
                                             const int end[8], const int ck[8], int px, int py, int pz,
                                             double acc[6]) {
    const DevGrid &g = B.g;
    for (int q = 0; q < 6; ++q) acc[q] = 0.0;
    if (n == 0) return;
    const DevState &O = B.st[B.cur];
    int head[8];
    for (int c = 0; c < n; ++c) head[c] = O.lid[B.perm[pos[c]]];
    const double xv = g.dx * (double)(px + g.ioff - 1);
    const double yv = g.dy * (double)(py + g.joff - 1);
    const double zv = g.zz[pz];
    while (true) {
        int best = -1, bl = 0x7fffffff;
        for (int c = 0; c < n; ++c)
            if (pos[c] < end[c] && head[c] < bl) { bl = head[c]; best = c; }
        if (best < 0) break;
        const int at = pos[best];
        const int kpt = ck[best];
        pos[best]++;
        if (pos[best] < end[best]) head[best] = O.lid[B.perm[pos[best]]];
        DropVals d;
        const int t = B.perm[at];
        double v[P64_N];
        int lid, key;
        load_payload64(B.pay, t, v, lid, key);
        d.x1 = O.x[0][t]; d.x2 = O.x[1][t]; d.x3 = O.x[2][t];
        for (int a = 0; a < 3; ++a) { d.D[a] = v[P64_D + a]; d.V[a] = v[P64_V + a]; }
        d.T0 = v[P64_T0]; d.H0 = v[P64_H0]; d.E1 = v[P64_E1]; d.E2 = v[P64_E2]; d.mult = v[P64_MULT];
        contribute64(g, p, d, kpt, xv, yv, zv, acc);
    }
}

// a / d, correctly rounded, from y = RN(1/d): two residual corrections.  The
// first leaves a quotient within one ulp of a/d, and then the second returns
// RN(a/d) (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990, theorem on q + r y with r = a - q d exact),
// provided that d's significand is not all ones and nothing over- or
// underflows: DevGrid::rdV is only set when the grid's denominators qualify,
// and the caller has looked at the numerators.  5 operations for the
// division's 14 instructions and its branch.
__device__ __forceinline__ double div_by(double a, double d, double y) {
    const double q0 = a * y;
    const double q1 = fma(fma(-q0, d, a), y, q0);
    return fma(fma(-q1, d, a), y, q1);
}

// numerators div_by may take: zero, or 2^-600 <= |v| < 2^900 (times weights
// of at least 2^-159, their residuals stay normal numbers)
__device__ __forceinline__ bool plain_num(double v) {
    const unsigned hi = (unsigned)(__double_as_longlong(v) >> 32) & 0x7fffffffu;
    return v == 0.0 || (hi >= ((1023u - 600u) << 20) && hi < ((1023u + 900u) << 20));
}

// Stage of an FP64 tile: lid, slot and trilinear weights of up to `cap`
// droplets, one array per value.  The factors stay in the payload, whose three
// 32-byte words a node reads where it needs them (L1, mostly): staged as
// well, they took 140 bytes a droplet and held the SM at two CTAs of 128
// registers (16.8 M droplets: 4.69 ms, against 4.15 at three CTAs of 80, and
// 4.66 at four of 64).
enum { V64_WX = 0, V64_WY = 2, V64_WZ = 4, V64_N = 6 };
constexpr int kStage64 = V64_N * 8 + 2 * 4;   // bytes per droplet

// One node from the stage: its cells' lists (run[c]: first stage position, end
// << 16; c = i<<2 | j<<1 | k) merged by lid.  dV, rdV: cell volume of the
// droplet's cell and its reciprocal, for k = 0 and 1.
template <bool FAST, int CAP>
__device__ __forceinline__ void merge_staged64(const DevBox &B, const DevParams &p, const int *s_lid, const int *s_t, const double *s_w,
                                               int (&run)[8], const double dV[2], const double rdV[2],
                                               double acc[6]) {
    constexpr int kNone = 0x7fffffff;   // no lid is this large
    int head[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) head[c] = (run[c] & 0xffff) < (run[c] >> 16) ? s_lid[run[c] & 0xffff] : kNone;
    for (int q = 0; q < 6; ++q) acc[q] = 0.0;
    while (true) {
        int least = head[0];
#pragma unroll
        for (int c = 1; c < 8; ++c) least = min(least, head[c]);
        if (least == kNone) break;
        int o = 0, sel = 0;
#pragma unroll
        for (int c = 7; c >= 0; --c)
            if (head[c] == least) { o = c; sel = run[c]; }
        const int at = sel & 0xffff;
        const int next = at + 1 < (sel >> 16) ? s_lid[at + 1] : kNone;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            if (c == o) { head[c] = next; run[c] = sel + 1; }
        const double *w = s_w + at;
        const double d = (o & 1) ? dV[1] : dV[0], y = (o & 1) ? rdV[1] : rdV[0];
        const double wtx = w[(V64_WX + (o >> 2)) * CAP];
        const double wty = w[(V64_WY + ((o >> 1) & 1)) * CAP];
        const double wtz = w[(V64_WZ + (o & 1)) * CAP];
        const double wtt = wtx * wty * wtz;
        double v[P64_N];
        int lid, key;
        load_payload64(B.pay, s_t[at], v, lid, key);
        const double mult = v[P64_MULT];
        auto term = [&](int q) {
            const double a = v[q] * wtt;
            return (FAST ? div_by(a, d, y) : a / d) * mult;
        };
        if (p.icouple == 1) {
            for (int a = 0; a < 3; ++a) {
                acc[a] = acc[a] - term(P64_D + a);
                acc[a] = acc[a] - term(P64_V + a);
            }
        }
        if (p.iTcouple == 1) acc[3] = acc[3] - term(P64_T0);
        if (p.iHcouple == 1) {
            acc[4] = acc[4] - term(P64_H0);
            acc[5] = acc[5] - term(P64_E1) + term(P64_E2);
        }
    }
}

// Mixed: the node's cells in the fixed order (i, j, k) = (0,0,0), (0,0,1),
// ..., (1,1,1), each cell's droplets in its (lid-sorted) list order; the
// staged and the global path below perform the same operations in the same
// order, so every tile shape gives the same sums.
__device__ __forceinline__ void image_global32(const DevBox &B, const DevParams &p, int px, int py, int pz,
                                               double acc[6]) {
    const DevGrid &g = B.g;
    for (int q = 0; q < 6; ++q) acc[q] = 0.0;
#pragma unroll 1
    for (int o = 0; o < 8; ++o) {
        const int i = o >> 2, j = (o >> 1) & 1, k = o & 1;
        const int ci = px - i, cj = py - j, ckk = pz - k;
        if (ci < 1 || ci > g.nnx + 1 || cj < 1 || cj > g.nny + 1 || ckk < 0 || ckk > g.nnz) continue;
        const int key = ckk + (g.nnz + 1) * ((cj - 1) + (g.nny + 1) * (ci - 1));
        const int a = B.cell_start[key], b = B.cell_start[key + 1];
        if (a == b) continue;
        double S[6];
        cell_sum32(B, p, a, b, i, j, k, S);
        for (int q = 0; q < 6; ++q) acc[q] += S[q];
    }
}

// one pre-fold node image from the per-cell sums of a dense box
__device__ __forceinline__ void image_cells32(const DevBox &B, int px, int py, int pz, double acc[6]) {
    const DevGrid &g = B.g;
    for (int q = 0; q < 6; ++q) acc[q] = 0.0;
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        const int i = o >> 2, j = (o >> 1) & 1, k = o & 1;
        const int ci = px - i, cj = py - j, ckk = pz - k;
        if (ci < 1 || ci > g.nnx + 1 || cj < 1 || cj > g.nny + 1 || ckk < 0 || ckk > g.nnz) continue;
        const long long key = ckk + (long long)(g.nnz + 1) * ((cj - 1) + (long long)(g.nny + 1) * (ci - 1));
        if (B.cell_start[key] == B.cell_start[key + 1]) continue;
        const double *S = B.cellsum + (key * 8 + o) * 6;
        for (int q = 0; q < 6; ++q) acc[q] += S[q];
    }
}

// FP64: one pre-fold node image from global memory
__device__ __forceinline__ void image_global64(const DevBox &B, const DevParams &p, int px, int py, int pz,
                                               double acc[6]) {
    const DevGrid &g = B.g;
    int pos[8], end[8], ck[8];
    int n = 0;
    for (int i = 0; i <= 1; ++i)
        for (int j = 0; j <= 1; ++j)
            for (int k = 0; k <= 1; ++k) {
                const int ci = px - i, cj = py - j, ckk = pz - k;
                if (ci < 1 || ci > g.nnx + 1 || cj < 1 || cj > g.nny + 1 || ckk < 0 || ckk > g.nnz) continue;
                const int key = ckk + (g.nnz + 1) * ((cj - 1) + (g.nny + 1) * (ci - 1));
                const int a = B.cell_start[key], b = B.cell_start[key + 1];
                if (a < b) { pos[n] = a; end[n] = b; ck[n] = ckk; n++; }
            }
    merge_ranges(B, p, n, pos, end, ck, px, py, pz, acc);
}

// a whole output node (with its periodic images, folded x first, then y)
template <class Image>
__device__ __forceinline__ void node_fold(const DevGrid &g, int ix, int iy, int iz, double out[6],
                                          const Image &image) {
    double a1[6];
    image(ix, iy, iz, out);
    if (g.periodic && ix <= 2) {
        image(ix + g.nnx, iy, iz, a1);
        for (int q = 0; q < 6; ++q) out[q] = out[q] + a1[q];
    }
    if (g.periodic && iy <= 2) {
        double b0[6];
        image(ix, iy + g.nny, iz, b0);
        if (g.periodic && ix <= 2) {
            image(ix + g.nnx, iy + g.nny, iz, a1);
            for (int q = 0; q < 6; ++q) b0[q] = b0[q] + a1[q];
        }
        for (int q = 0; q < 6; ++q) out[q] = out[q] + b0[q];
    }
}

// FP64: a node of a tile that does not stage, from global memory (out of line:
// its locals stay off the staged path)
__device__ __noinline__ void node_global64(const DevBox &B, const DevParams &p, int ix, int iy, int iz, bool images,
                                           double out[6]) {
    if (images)
        image_global64(B, p, ix, iy, iz, out);
    else
        node_fold(B.g, ix, iy, iz, out,
                  [&](int px, int py, int pz, double acc[6]) { image_global64(B, p, px, py, pz, acc); });
}

// Dense boxes (mixed): every cell's 8 corner sums S_o once, one thread per
// (cell, corner) -- grid.y = box, grid-stride over cells x 8
__global__ void k_cellsums32(DevBox *boxes, const __grid_constant__ DevParams P) {
    step_kernel_begin();
    const DevBox &B = boxes[blockIdx.y];
    if (B.cellsum == nullptr) return;
    const long long total = B.g.ncells * 8;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const long long cell = idx >> 3;
        const int o = (int)(idx & 7);
        double S[6];
        cell_sum32(B, P, B.cell_start[cell], B.cell_start[cell + 1], o >> 2, (o >> 1) & 1, o & 1, S);
        double *out = B.cellsum + idx * 6;
        for (int q = 0; q < 6; ++q) out[q] = S[q];
    }
}

// Dense boxes (mixed): every output node from the cell sums
__global__ void k_nodes_dense32(DevBox *boxes) {
    step_kernel_begin();
    const DevBox &B = boxes[blockIdx.y];
    if (B.cellsum == nullptr) return;
    const DevGrid &g = B.g;
    const long long total = (long long)g.snx * g.sny * g.nz2;
    for (long long node = (long long)blockIdx.x * blockDim.x + threadIdx.x; node < total;
         node += (long long)gridDim.x * blockDim.x) {
        const int iz = (int)(node % g.nz2);
        const int iy = 1 + (int)((node / g.nz2) % g.sny);
        const int ix = 1 + (int)(node / ((long long)g.nz2 * g.sny));
        double out[6];
        node_fold(g, ix, iy, iz, out,
                  [&](int px, int py, int pz, double acc[6]) { image_cells32(B, px, py, pz, acc); });
        for (int q = 0; q < 6; ++q) B.src[q][node] = out[q];
    }
}

// a deposition node: the box's own nodes to the sources, the periodic images
// (ix > nnx or iy > nny) to B.img
__device__ __forceinline__ void store_node(const DevBox &B, int ix, int iy, int iz, const double out[6]) {
    const DevGrid &g = B.g;
    if (ix <= g.snx && iy <= g.sny) {
        const long long node = (long long)iz + (long long)g.nz2 * ((long long)(iy - 1) + (long long)g.sny * (ix - 1));
        for (int q = 0; q < 6; ++q) B.src[q][node] = out[q];
    } else {
        const long long at = img_index(g, ix, iy, iz), per = img_count(g);
        for (int q = 0; q < 6; ++q) B.img[q * per + at] = out[q];
    }
}

// Periodic boxes: the fold of particle_coupling_exchange on the nodes
// with ix <= 2 or iy <= 2, from their own image (in the sources) and the
// image nodes, in node_fold's order; grid (blocks, boxes, quantities)
__global__ void k_fold(DevBox *boxes, int *overflow_list) {
    step_kernel_begin();
    // the tiles listed for the overflow kernel are done: an empty list for the next deposition
    if (overflow_list != nullptr && blockIdx.x + blockIdx.y + blockIdx.z + threadIdx.x == 0)
        overflow_list[0] = 0;
    const DevBox &B = boxes[blockIdx.y];
    const DevGrid &g = B.g;
    if (!g.periodic || B.img == nullptr || B.cellsum != nullptr) return;
    const int ya = g.nny < 2 ? g.nny : 2, xb = g.nnx < 2 ? g.nnx : 2;
    // A thread per (quantity, node): one node's six values in turn made a chain
    // of loads, 14 us even in a 32^3 box; grid.z is the quantity.  The padded grid has
    // more points than there are border nodes, and fewer than 2^31: 32-bit divisions.
    // Bound by the latency of its loads: kFoldBlocks has the measurements.
    const unsigned nz2 = (unsigned)g.nz2, rows = (unsigned)(g.nny - 2);
    const unsigned na = (unsigned)ya * g.nnx * nz2;                 // iy <= 2, every ix
    const unsigned nb = g.nny > 2 ? (unsigned)xb * rows * nz2 : 0;  // ix <= 2, iy >= 3
    const int q = blockIdx.z;
    const double *I = B.img + q * img_count(g);
    for (unsigned idx = blockIdx.x * blockDim.x + threadIdx.x; idx < na + nb; idx += gridDim.x * blockDim.x) {
        int ix, iy, iz;
        if (idx < na) {
            const unsigned c = idx / nz2;
            iz = (int)(idx - c * nz2);
            iy = 1 + (int)(c % (unsigned)ya);
            ix = 1 + (int)(c / (unsigned)ya);
        } else {
            const unsigned r = idx - na, c = r / nz2;
            iz = (int)(r - c * nz2);
            iy = 3 + (int)(c % rows);
            ix = 1 + (int)(c / rows);
        }
        const long long node = (long long)iz + (long long)g.nz2 * ((long long)(iy - 1) + (long long)g.sny * (ix - 1));
        double out = B.src[q][node];
        if (ix <= 2) out = out + I[img_index(g, ix + g.nnx, iy, iz)];
        if (iy <= 2) {
            double b0 = I[img_index(g, ix, iy + g.nny, iz)];
            if (ix <= 2) b0 = b0 + I[img_index(g, ix + g.nnx, iy + g.nny, iz)];
            out = out + b0;
        }
        B.src[q][node] = out;
    }
}

// shared memory of a tile shape (TX x TY x TZ nodes)
__host__ __device__ constexpr int dep_smem_bytes(bool mixed, int TX, int TY, int TZ) {
    return (mixed ? kDepCapMixed * (kStageD * 8 + kStageF * 4) : 0) +
           (TX + 1) * (TY + 1) * (TZ + 2) * 4 + (TX + 1) * (TY + 1) * 4 + 16;
}

// The columns of a tile's cells: s_cs[col][TZ+2] the starts of their cells in
// the sorted list (absolute; levels z0-1 .. z0+TZ clamped to the grid),
// s_off[col] their offsets in the stage.  Returns the droplets in all.
template <int TX, int TY, int TZ>
__device__ __forceinline__ int tile_columns(const DevBox &B, int x0, int y0, int z0, int *s_cs, int *s_off) {
    constexpr int COLS = (TX + 1) * (TY + 1), CSW = TZ + 2;
    static_assert(COLS <= 32, "one warp scans the column counts");
    __shared__ int s_total;
    const DevGrid &g = B.g;
    const int ck_lo = max(z0 - 1, 0), ck_hi = min(z0 + TZ - 1, g.nnz);
    for (int e = threadIdx.x; e < COLS * CSW; e += blockDim.x) {
        const int cc = e / CSW, lzz = e % CSW;
        const int ci = x0 - 1 + cc / (TY + 1), cj = y0 - 1 + cc % (TY + 1);
        int v = 0;
        if (ci >= 1 && cj >= 1 && ci <= g.nnx + 1 && cj <= g.nny + 1) {
            const int ck = min(max(z0 - 1 + lzz, ck_lo), ck_hi + 1);
            v = B.cell_start[ck + (g.nnz + 1) * ((cj - 1) + (g.nny + 1) * (ci - 1))];
        }
        s_cs[e] = v;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        // exclusive scan of the columns' droplet counts (stage offsets)
        const int cc = threadIdx.x;
        const int cnt = cc < COLS ? s_cs[cc * CSW + CSW - 1] - s_cs[cc * CSW] : 0;
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (cc >= o) incl += y;
        }
        if (cc < COLS) s_off[cc] = incl - cnt;
        if (cc == COLS - 1) s_total = incl;
    }
    __syncthreads();
    return s_total;
}

// FP64 tiles (z fastest); tile shapes 2x4x32, 4x4x16 and 2x2x64 nodes are
// instantiated (autotuned).
//
// Bound by the latency of the merge: a node merges about 8 droplets at one per
// cell, each of them 10 terms of a multiply, a division, a multiply and a
// subtraction, and half of a warp's lanes wait for the longest list.  Issue is at
// 52%, the L1 data pipe at 58%, the FP64 pipe at 29% with 21 warps on an SM
// (profiles/k_deposit64_2M_droplets_128cube.md); more warps help, fewer
// instructions do not.  The trilinear weights (6 a droplet) are formed while
// staging, not 3 per node, the divisions by the cell volume take div_by, and the
// merge keeps its 8 list heads in registers.  16.8 M droplets on 256^3: 7.90 ->
// 4.04 ms; 1 M on 128^3: 0.71 -> 0.375 ms, where the edge tiles' merges from global
// memory counted most.
template <int TX, int TY, int TZ, int CAP>
__global__ void __launch_bounds__(kDepositThreads, 3)
k_deposit64(DevBox *boxes, const Tile *tiles, int first, int ntiles, const __grid_constant__ DevParams P,
            int *overflow_list) {
    step_kernel_begin<false>();
    static_assert(TX * TY * TZ == kDepositThreads, "one thread per node of the tile");
    constexpr int COLS = (TX + 1) * (TY + 1), CSW = TZ + 2;
    extern __shared__ __align__(16) unsigned char sm[];
    double *s_w = (double *)sm;                        // [V64_N][CAP]
    int *s_lid = (int *)(sm + V64_N * 8 * CAP);        // [CAP]
    int *s_t = s_lid + CAP;                            // [CAP]
    int *s_cs = s_t + CAP, *s_off = s_cs + COLS * CSW;
    const Tile tl = tiles[blockIdx.x];   // of the run that starts at tile `first` of ntiles
    const DevBox &B = boxes[tl.box];
    const DevGrid &g = B.g;
    const int ntz = (g.nz2 + TZ - 1) / TZ, nty = (g.dny + TY - 1) / TY;
    const int tzi = tl.start % ntz, tyi = (tl.start / ntz) % nty, txi = tl.start / (ntz * nty);
    const int x0 = 1 + txi * TX, y0 = 1 + tyi * TY, z0 = tzi * TZ;
    const int lz = threadIdx.x % TZ, ly = (threadIdx.x / TZ) % TY, lx = threadIdx.x / (TZ * TY);
    const int ix = x0 + lx, iy = y0 + ly, iz = z0 + lz;
    const bool valid = ix <= g.dnx && iy <= g.dny && iz <= g.nnz + 1;
    // whether periodic images are nodes of their own (or there are none):
    // otherwise the tiles on the periodic edges fold theirs from global memory
    const bool images = !g.periodic || B.img != nullptr;
    double out[6];
    bool staged = images || ((x0 > 2) && (y0 > 2));
    if (staged) {
        const int total = tile_columns<TX, TY, TZ>(B, x0, y0, z0, s_cs, s_off);
        if (total == 0) {
            const double zero[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            if (valid) store_node(B, ix, iy, iz, zero);
            return;
        }
        staged = total <= CAP;
        if (staged) {
            // two droplets per pass: their loads are in flight together
            const DevState &O = B.st[B.cur];
            bool fast = g.rdV != nullptr;
            auto stage = [&](int k, int c, int t, const double *v, const double *w, int l, int key) {
                s_lid[k] = l;
                s_t[k] = t;
#pragma unroll
                for (int q = 0; q < P64_MULT; ++q) fast = fast && plain_num(v[q]);
                // the weights of the cell's lower (0) and upper (1) nodes
                const int ci = x0 - 1 + c / (TY + 1), cj = y0 - 1 + c % (TY + 1);
                const int ck = key - (g.nnz + 1) * ((cj - 1) + (g.nny + 1) * (ci - 1));
                const double dz = g.dzu[ck + 1];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const double ax = fabs(w[0] - g.dx * (double)(ci + m + g.ioff - 1));
                    const double ay = fabs(w[1] - g.dy * (double)(cj + m + g.joff - 1));
                    const double az = fabs(w[2] - g.zz[ck + m]);
                    const bool f = g.rdV != nullptr;
                    s_w[(V64_WX + m) * CAP + k] = 1.0 - (f ? div_by(ax, g.dx, g.rdx) : ax / g.dx);
                    s_w[(V64_WY + m) * CAP + k] = 1.0 - (f ? div_by(ay, g.dy, g.rdy) : ay / g.dy);
                    s_w[(V64_WZ + m) * CAP + k] = 1.0 - (f ? div_by(az, dz, g.rdzu[ck + 1]) : az / dz);
                }
            };
            for (int k0 = threadIdx.x; k0 < total; k0 += 2 * blockDim.x) {
                const int k1 = k0 + blockDim.x;
                const bool two = k1 < total;
                int c0 = 0, c1 = 0;
                while (c0 + 1 < COLS && s_off[c0 + 1] <= k0) ++c0;
                while (c1 + 1 < COLS && s_off[c1 + 1] <= k1) ++c1;
                const int t0 = B.perm[s_cs[c0 * CSW] + (k0 - s_off[c0])];
                const int t1 = two ? B.perm[s_cs[c1 * CSW] + (k1 - s_off[c1])] : t0;
                double v0[P64_N], v1[P64_N];
                int l0, l1, e0, e1;
                load_payload64(B.pay, t0, v0, l0, e0);
                load_payload64(B.pay, t1, v1, l1, e1);
                const double w0[3] = {O.x[0][t0], O.x[1][t0], O.x[2][t0]};
                const double w1[3] = {O.x[0][t1], O.x[1][t1], O.x[2][t1]};
                stage(k0, c0, t0, v0, w0, l0, e0);
                if (two) stage(k1, c1, t1, v1, w1, l1, e1);
            }
            fast = __syncthreads_and(fast) != 0;
            if (valid) {
                int run[8];
                double dV[2], rdV[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int ck = iz - k;
                    const bool in = ck >= 0 && ck <= g.nnz;
                    dV[k] = in ? g.dx * g.dy * g.dzu[ck + 1] : 1.0;
                    rdV[k] = in && g.rdV != nullptr ? g.rdV[ck + 1] : 1.0;
#pragma unroll
                    for (int ij = 0; ij < 4; ++ij) {
                        const int cc = (lx + 1 - (ij >> 1)) * (TY + 1) + (ly + 1 - (ij & 1));
                        const int *cs = s_cs + cc * CSW + lz + 1 - k;
                        const int base = s_off[cc] - s_cs[cc * CSW];
                        run[ij << 1 | k] = in ? (base + cs[0]) | (base + cs[1]) << 16 : 0;
                    }
                }
                if (fast) merge_staged64<true, CAP>(B, P, s_lid, s_t, s_w, run, dV, rdV, out);
                else merge_staged64<false, CAP>(B, P, s_lid, s_t, s_w, run, dV, rdV, out);
            }
        }
    }
    if (!staged && overflow_list != nullptr) {
        // above the stage capacity: k_deposit64_overflow, which has the
        // registers of the global path
        if (threadIdx.x == 0)
            overflow_put(overflow_list, ntiles, first + blockIdx.x, [](int *n) { return atomicAdd(n, 1); });
        return;
    }
    if (!valid) return;
    if (!staged) node_global64(B, P, ix, iy, iz, images, out);
    store_node(B, ix, iy, iz, out);
}

// FP64 tiles listed by k_deposit64: each node's own image merged from global
// memory; grid-stride over the list
template <int TX, int TY, int TZ>
__global__ void __launch_bounds__(kDepositThreads, 2)
k_deposit64_overflow(DevBox *boxes, const Tile *tiles, int ntiles, const __grid_constant__ DevParams P,
                     const int *overflow_list) {
    step_kernel_begin();
    const int n = overflow_count(overflow_list, ntiles);
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const Tile tl = tiles[overflow_list[1 + e]];
        const DevBox &B = boxes[tl.box];
        const DevGrid &g = B.g;
        const int ntz = (g.nz2 + TZ - 1) / TZ, nty = (g.dny + TY - 1) / TY;
        const int tzi = tl.start % ntz, tyi = (tl.start / ntz) % nty, txi = tl.start / (ntz * nty);
        const int lz = threadIdx.x % TZ, ly = (threadIdx.x / TZ) % TY, lx = threadIdx.x / (TZ * TY);
        const int ix = 1 + txi * TX + lx, iy = 1 + tyi * TY + ly, iz = tzi * TZ + lz;
        if (ix > g.dnx || iy > g.dny || iz > g.nnz + 1) continue;
        double out[6];
        image_global64(B, P, ix, iy, iz, out);
        store_node(B, ix, iy, iz, out);
    }
}

// Mixed tiles (z fastest), the same shapes.
template <int kDepTX, int kDepTY, int kDepTZ>
__global__ void __launch_bounds__(kDepositThreads, 4)
k_deposit_tiled(DevBox *boxes, const Tile *tiles, const __grid_constant__ DevParams P, int *overflow_list,
                int any_dense) {
    step_kernel_begin<false>();
    static_assert(kDepTX * kDepTY * kDepTZ == kDepositThreads, "one thread per node of the tile");
    constexpr int kDepCols = (kDepTX + 1) * (kDepTY + 1);
    constexpr int kDepCSW = kDepTZ + 2;
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int CAP = kDepCapMixed;
    // stage: values first (8-byte aligned), then cell starts, column offsets
    double *s_v = (double *)sm;                                         // [kStageD][CAP]
    float *s_f = (float *)(sm + kStageD * CAP * 8);                     // [kStageF][CAP]
    int *s_cs = (int *)(sm + CAP * (kStageD * 8 + kStageF * 4));        // [cols][TZ+2], absolute
    int *s_off = s_cs + kDepCols * kDepCSW;                             // [cols] stage offset
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    if (any_dense && B.cellsum != nullptr) return;   // dense box: k_cellsums32 + k_nodes_dense32
    const DevParams &p = P;
    const DevGrid &g = B.g;
    const int ntz = (g.nz2 + kDepTZ - 1) / kDepTZ, nty = (g.dny + kDepTY - 1) / kDepTY;
    const int tzi = tl.start % ntz, tyi = (tl.start / ntz) % nty, txi = tl.start / (ntz * nty);
    const int x0 = 1 + txi * kDepTX, y0 = 1 + tyi * kDepTY, z0 = tzi * kDepTZ;
    const int lz = threadIdx.x % kDepTZ, ly = (threadIdx.x / kDepTZ) % kDepTY, lx = threadIdx.x / (kDepTZ * kDepTY);
    const int ix = x0 + lx, iy = y0 + ly, iz = z0 + lz;
    const bool valid = ix <= g.dnx && iy <= g.dny && iz <= g.nnz + 1;
    const int total = tile_columns<kDepTX, kDepTY, kDepTZ>(B, x0, y0, z0, s_cs, s_off);
    if (total == 0) {
        const double zero[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (valid) store_node(B, ix, iy, iz, zero);
        return;
    }
    if (total > CAP) {
        // above the stage capacity: k_deposit_overflow32, which has the
        // registers of the global path
        if (threadIdx.x == 0)
            overflow_put(overflow_list, gridDim.x, blockIdx.x, [](int *n) { return atomicAdd(n, 1); });
        return;
    }
    // two droplets per pass: their perm and payload loads are in flight
    // together
    for (int k0 = threadIdx.x; k0 < total; k0 += 2 * blockDim.x) {
        const int k1 = k0 + blockDim.x;
        int c0 = 0, c1 = 0;
        while (c0 + 1 < kDepCols && s_off[c0 + 1] <= k0) ++c0;
        while (c1 + 1 < kDepCols && s_off[c1 + 1] <= k1) ++c1;
        const bool two = k1 < total;
        const int t0 = B.perm[s_cs[c0 * kDepCSW] + (k0 - s_off[c0])];
        const int t1 = two ? B.perm[s_cs[c1 * kDepCSW] + (k1 - s_off[c1])] : t0;
        float v0[P32_N], v1[P32_N];
        load_payload32(B.pay32, t0, v0);
        load_payload32(B.pay32, t1, v1);
        // the factors as contribute32 applies them: -DV, -T0, -H0, +E
        auto stage = [&](int k, const float *v) {
            const double d[kStageD] = {-(double)v[P32_DV0], -(double)v[P32_DV1], -(double)v[P32_DV2],
                                       -(double)v[P32_T0], -(double)v[P32_H0], (double)v[P32_E]};
#pragma unroll
            for (int q = 0; q < kStageD; ++q) s_v[q * CAP + k] = d[q];
            s_f[0 * CAP + k] = v[P32_FX];
            s_f[1 * CAP + k] = v[P32_FY];
            s_f[2 * CAP + k] = v[P32_FZ];
            s_f[3 * CAP + k] = v[P32_FAC];
        };
        stage(k0, v0);
        if (two) stage(k1, v1);
    }
    __syncthreads();
    if (!valid) return;
    double out[6];
    for (int q = 0; q < 6; ++q) out[q] = 0.0;
    // the corner loop stays rolled: a smaller kernel (instruction fetch was a
    // leading stall)
#pragma unroll 1
    for (int o = 0; o < 8; ++o) {
        const int i = o >> 2, j = (o >> 1) & 1, k = o & 1;
        const int ckk = iz - k;
        if (ckk < 0 || ckk > g.nnz) continue;
        const int cc = (lx + 1 - i) * (kDepTY + 1) + (ly + 1 - j);
        const int lzz = lz + 1 - k;
        const int base = s_off[cc] - s_cs[cc * kDepCSW];
        const int a = base + s_cs[cc * kDepCSW + lzz];
        const int b = base + s_cs[cc * kDepCSW + lzz + 1];
        if (a == b) continue;
        double S[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int at = a; at < b; ++at) {
            // contribute32 with the factors staged in FP64 (the same values,
            // so the same bits)
            const float fx = s_f[at], fy = s_f[CAP + at], fz = s_f[2 * CAP + at];
            const float wx = i ? fx : 1.0f - fx;
            const float wy = j ? fy : 1.0f - fy;
            const float wz = k ? fz : 1.0f - fz;
            const double c = (double)(wx * wy * wz * s_f[3 * CAP + at]);
            if (p.icouple == 1)
                for (int a3 = 0; a3 < 3; ++a3) S[a3] = fma(s_v[a3 * CAP + at], c, S[a3]);
            if (p.iTcouple == 1) S[3] = fma(s_v[3 * CAP + at], c, S[3]);
            if (p.iHcouple == 1) {
                S[4] = fma(s_v[4 * CAP + at], c, S[4]);
                S[5] = fma(s_v[5 * CAP + at], c, S[5]);
            }
        }
        for (int q = 0; q < 6; ++q) out[q] += S[q];
    }
    store_node(B, ix, iy, iz, out);
}

// Mixed tiles listed by k_deposit_tiled (overflow_list[0] of them in
// overflow_list[1..], above the stage capacity): each node's own image from
// global memory, stored like the tiled kernel's; grid-stride over the list
template <int kDepTX, int kDepTY, int kDepTZ>
__global__ void __launch_bounds__(kDepositThreads)
k_deposit_overflow32(DevBox *boxes, const Tile *tiles, int ntiles, const __grid_constant__ DevParams P,
                     const int *overflow_list) {
    step_kernel_begin();
    const int n = overflow_count(overflow_list, ntiles);
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const Tile tl = tiles[overflow_list[1 + e]];
        const DevBox &B = boxes[tl.box];
        const DevGrid &g = B.g;
        const int ntz = (g.nz2 + kDepTZ - 1) / kDepTZ, nty = (g.dny + kDepTY - 1) / kDepTY;
        const int tzi = tl.start % ntz, tyi = (tl.start / ntz) % nty, txi = tl.start / (ntz * nty);
        const int lz = threadIdx.x % kDepTZ, ly = (threadIdx.x / kDepTZ) % kDepTY,
                  lx = threadIdx.x / (kDepTZ * kDepTY);
        const int ix = 1 + txi * kDepTX + lx, iy = 1 + tyi * kDepTY + ly, iz = tzi * kDepTZ + lz;
        if (ix > g.dnx || iy > g.dny || iz > g.nnz + 1) continue;
        double out[6];
        image_global32(B, P, ix, iy, iz, out);
        store_node(B, ix, iy, iz, out);
    }
}

}  // namespace
}  // namespace ntlp
