// ntlp_sort.cu -- cell binning, counting sort and step bookkeeping.
//
// After an update kernel has written every droplet's new cell key, the
// droplets are bucketed by key (a counting sort: histogram, per-box
// exclusive scan, scatter) and each cell's list is put in list order
// (ascending lid).  The ranked index list becomes the next step's read
// permutation, and the cell offsets drive the deposition.  Keys are the
// reference's binning (floor(x/dx)+1, minloc on zz), so cell membership is
// exact; the per-cell lid order makes the layout deterministic even though
// the scatter uses atomics.
#include <cuda_runtime.h>

#include <algorithm>

#include "ntlp_dev.cuh"
#include "ntlp_kernels.h"

namespace ntlp {

// ---- histogram: counted by the kernels that write the keys (the update
// kernels and k_keys_initial add 1 to cell_cnt[key]); cell_cnt is zero
// between sorts (the scatter counts each cell back down to zero)
// ---- scan (three phases over tiles of kScanTile buckets) -----------------
__device__ __forceinline__ long long nbuckets(const DevBox &B) { return B.g.ncells + 2; }

__global__ void k_scan_sums(DevBox *boxes, const Tile *tiles, long long *sums) {
    step_kernel_begin();
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    const long long nb = nbuckets(B);
    long long s = 0;
    for (int i = threadIdx.x; i < kScanTile; i += blockDim.x) {
        long long c = (long long)tl.start + i;
        if (c < nb) s += B.cell_cnt[c];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ long long sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long tot = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += sh[w];
        sums[blockIdx.x] = tot;
    }
}

// one block per box: exclusive scan of the box's tile sums, in place
__global__ void k_scan_offsets(const int *box_first_tile, long long *sums) {
    step_kernel_begin();
    const int b = blockIdx.x;
    const int a = box_first_tile[b], e = box_first_tile[b + 1];
    __shared__ long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = a; base < e; base += blockDim.x) {
        int i = base + threadIdx.x;
        long long v = (i < e) ? sums[i] : 0;
        // block inclusive scan
        long long x = v;
        for (int o = 1; o < 32; o <<= 1) {
            long long y = __shfl_up_sync(0xffffffffu, x, o);
            if ((threadIdx.x & 31) >= o) x += y;
        }
        __shared__ long long wsum[32];
        if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = x;
        __syncthreads();
        if (threadIdx.x < 32) {
            long long w = (threadIdx.x < (blockDim.x >> 5)) ? wsum[threadIdx.x] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                long long y = __shfl_up_sync(0xffffffffu, w, o);
                if (threadIdx.x >= o) w += y;
            }
            wsum[threadIdx.x] = w;
        }
        __syncthreads();
        long long incl = x + ((threadIdx.x >> 5) ? wsum[(threadIdx.x >> 5) - 1] : 0);
        if (i < e) sums[i] = carry + incl - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += incl;
        __syncthreads();
    }
}

// local exclusive scan of each tile plus its offset; counts are cleared (the
// array becomes the scatter cursor)
__global__ void k_scan_local(DevBox *boxes, const Tile *tiles, const long long *offs) {
    step_kernel_begin();
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    const long long nb = nbuckets(B);
    constexpr int PER = kScanTile / kCellThreads;
    int v[PER];
    int tsum = 0;
    const long long base = (long long)tl.start + threadIdx.x * PER;
    for (int k = 0; k < PER; ++k) {
        long long c = base + k;
        v[k] = (c < nb) ? B.cell_cnt[c] : 0;
        tsum += v[k];
    }
    // exclusive scan of per-thread sums
    int x = tsum;
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) >= o) x += y;
    }
    __shared__ int wsum[kCellThreads / 32];
    if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
        int w = (threadIdx.x < kCellThreads / 32) ? wsum[threadIdx.x] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (threadIdx.x >= o) w += y;
        }
        if (threadIdx.x < kCellThreads / 32) wsum[threadIdx.x] = w;
    }
    __syncthreads();
    long long run = offs[blockIdx.x] + (x - tsum) + ((threadIdx.x >> 5) ? wsum[(threadIdx.x >> 5) - 1] : 0);
    for (int k = 0; k < PER; ++k) {
        long long c = base + k;
        if (c < nb) {
            B.cell_start[c] = (int)run;
            run += v[k];
            if (c == nb - 1) B.cell_start[nb] = (int)run;
        }
    }
}

// ---- scatter ---------------------------------------------------------------
__global__ void k_scatter(DevBox *boxes, const Tile *tiles) {
    step_kernel_begin();
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    const int t = tl.start + threadIdx.x;
    if (t >= *B.n_alive) return;
    const int k = B.key[t];
    // counts down: the last droplet of a cell leaves its count at zero,
    // ready for the next step's histogram (the order inside a cell is
    // k_cellrank's)
    const int pos = B.cell_start[k] + atomicSub(&B.cell_cnt[k], 1) - 1;
    B.sorted[pos] = t;
}

// ---- per-cell list order (ascending lid) -----------------------------------
// One thread per sorted position: its droplet's rank among its cell's lids
// (ties, which unique lids never make, by position) is its place in the
// cell.  The order goes into the previous permutation, which is dead
// between the update and the finish, and becomes the new one.  The lids
// of a block's own positions are in shared memory, so a cell's lanes read
// them as broadcasts; only cells across its edges go to global memory.  O(n)
// per droplet of a cell of n: bound by the gathers of key and lid at one
// droplet per cell, by the loop at dozens.  It replaces an insertion sort in
// global memory, one thread per cell: the whole sort of 2 M droplets at 31 per
// cell took 0.71 ms, it takes 0.089 (16.8 M at one per cell: 0.44 -> 0.41).
__global__ void __launch_bounds__(kUpdateThreads) k_cellrank(DevBox *boxes, const Tile *tiles) {
    step_kernel_begin();
    __shared__ int s_lid[kUpdateThreads];
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    const int n = *B.n_alive;
    if (tl.start >= n) return;
    const int p = tl.start + threadIdx.x;
    const int *lid = B.st[1 - B.cur].lid;
    int tv = 0, lv = 0, a = 0, e = 0;
    if (p < n) {
        tv = B.sorted[p];
        const int c = B.key[tv];
        lv = lid[tv];
        a = B.cell_start[c];
        e = B.cell_start[c + 1];
        if (c == nbuckets(B) - 1) a = p, e = p + 1;   // killed droplets: any order
    }
    s_lid[threadIdx.x] = lv;
    __syncthreads();
    if (p >= n) return;
    int r = 0;
    if (e - a > 1) {
        const int lo = max(a, tl.start), hi = min(e, tl.start + kUpdateThreads);
        for (int q = a; q < lo; ++q) {
            const int lq = lid[B.sorted[q]];
            r += lq <= lv;                             // before p
        }
        for (int q = lo; q < hi; ++q) {
            const int lq = s_lid[q - tl.start];
            r += (lq < lv) || (lq == lv && q < p);
        }
        for (int q = hi; q < e; ++q) r += lid[B.sorted[q]] < lv;
    }
    B.perm[a + r] = tv;
}

void launch_sort(DevBox *boxes, const SortPlan &plan, cudaStream_t st) {
    launch_step_kernel(k_scan_sums, plan.n_cell_tiles, 256, 0, st, boxes, plan.cell_tiles, plan.tile_sums);
    launch_step_kernel(k_scan_offsets, plan.nbox, 1024, 0, st, plan.box_first_tile, plan.tile_sums);
    launch_step_kernel(k_scan_local, plan.n_cell_tiles, kCellThreads, 0, st, boxes, plan.cell_tiles, plan.tile_sums);
    launch_step_kernel(k_scatter, plan.n_drop_tiles, kUpdateThreads, 0, st, boxes, plan.drop_tiles);
    if (plan.n_drop_tiles > 0)
        launch_step_kernel(k_cellrank, plan.n_drop_tiles, kUpdateThreads, 0, st, boxes, plan.drop_tiles);
}

// ---- finish: flip buffers, count survivors ---------------------------------
__global__ void k_finish(DevBox *boxes, int nbox) {
    step_kernel_begin();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nbox) return;
    DevBox &B = boxes[b];
    const long long nb = B.g.ncells + 2;
    const int alive = B.cell_start[nb - 1];   // everything before the killed bucket
    *B.n_alive = alive;
    B.counters[C_NUMPART] = alive;
    B.cur = 1 - B.cur;
}

void launch_finish(DevBox *boxes, int nbox, cudaStream_t st) {
    launch_step_kernel(k_finish, (nbox + 127) / 128, 128, 0, st, boxes, nbox);
}

__global__ void k_reset_step(DevBox *boxes, int nbox) {
    step_kernel_begin();
    const DevBox &B = boxes[blockIdx.x];
    const int nz1 = B.g.nnz + 1;
    for (int i = threadIdx.x; i < kNumCounters; i += blockDim.x) B.counters[i] = 0;
    for (int i = threadIdx.x; i < nz1; i += blockDim.x) B.pflux[i] = 0.0;
    for (int i = threadIdx.x; i < 2 * nz1 * kFluxLimbs; i += blockDim.x) B.flux_fx[i] = 0;
    if (threadIdx.x == 0) {
        *B.err = 0;
        *B.ndefer = 0;
        if (B.nemig) *B.nemig = 0;
    }
}

void launch_reset_step(DevBox *boxes, int nbox, cudaStream_t st) {
    launch_step_kernel(k_reset_step, nbox, 256, 0, st, boxes, nbox);
}

// keys of a freshly uploaded state (held in st[1-cur], list order)
__global__ void k_keys_initial(DevBox *boxes, const Tile *tiles) {
    const Tile tl = tiles[blockIdx.x];
    const DevBox &B = boxes[tl.box];
    const int t = tl.start + threadIdx.x;
    if (t >= *B.n_alive) return;
    const DevState &O = B.st[1 - B.cur];
    int key = cell_key(B.g, O.x[0][t], O.x[1][t], O.x[2][t]);
    B.key[t] = key;
    atomicAdd(&B.cell_cnt[key], 1);   // the sort's histogram
}

void launch_keys_initial(DevBox *boxes, const Tile *tiles, int ntiles, cudaStream_t st) {
    if (ntiles > 0) k_keys_initial<<<ntiles, kUpdateThreads, 0, st>>>(boxes, tiles);
}

// ---- stored fields -----------------------------------------------------------
// one field value (q: u, v, w, T, q) or all of a point, in the path's form
struct StoreF64 {
    Node64 *f;
    double *w;
    __device__ __forceinline__ void one(int q, long long o, double v) const {
        if (q == 2) w[o] = v;
        else (&f[o].u)[q < 2 ? q : q - 1] = v;
    }
    __device__ __forceinline__ void all(long long o, const double v[5]) const {
        asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(f + o), "d"(v[0]), "d"(v[1]), "d"(v[3]),
                     "d"(v[4])
                     : "memory");
        w[o] = v[2];
    }
};
struct StoreF32 {   // deviations from the reference values
    float4 *f;
    float *w;
    double ref[5];
    __device__ __forceinline__ void one(int q, long long o, double v) const {
        const float d = (float)(v - ref[q]);
        if (q == 2) w[o] = d;
        else (&f[o].x)[q < 2 ? q : q - 1] = d;
    }
    __device__ __forceinline__ void all(long long o, const double v[5]) const {
        f[o] = make_float4((float)(v[0] - ref[0]), (float)(v[1] - ref[1]), (float)(v[3] - ref[3]),
                           (float)(v[4] - ref[4]));
        w[o] = (float)(v[2] - ref[2]);
    }
};

// the mixed path's store: reference values read from the source arrays
// (element ridx of each), and kept in B.ref by the grid's first thread
__device__ __forceinline__ StoreF32 store32(const DevBox &B, const FieldSrc &s, long long ridx, bool first) {
    StoreF32 S;
    S.f = const_cast<float4 *>(B.f4);
    S.w = const_cast<float *>(B.fw);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        S.ref[q] = s.p[q] ? s.p[q][ridx] : 0.0;
        if (first && s.p[q]) const_cast<double *>(B.ref)[q] = S.ref[q];
    }
    return S;
}

// flow layout u(1:nnx,1:nny,0:nnz+1) -> stored points (0:nnz+1,-1:nny+3,-1:nnx+3).
// A block takes the fields of a 32x32 tile of the (i, k) plane of one output
// row j through shared memory, so both the x-fastest reads and the z-fastest
// writes are coalesced.  HBM-bound: every value is read once (plus halos)
// and every point written once.  The mixed fields of 256^3 in device memory
// (copy, five halo fills and the FP32 pack before) took 1.1 ms, it takes 0.3.
template <class Store>
__device__ __forceinline__ void fill_tile(const FieldSrc &s, const DevGrid &g, const Store &S, double (*tile)[32][33]) {
    const int j = (int)blockIdx.z - 1;                 // -1 .. nny+3
    const int i0 = (int)blockIdx.x * 32 - 1;           // i of the tile's start
    const int k0 = (int)blockIdx.y * 32;
    const int jsrc = ((j - 1) % g.nny + g.nny) % g.nny;  // 0-based source row
    const int i = i0 + (int)threadIdx.x;
    const int isrc = ((i - 1) % g.nnx + g.nnx) % g.nnx;
    bool every = true;
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const double *p = s.p[q];
        every = every && p != nullptr;
        if (p == nullptr) continue;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int k = k0 + (int)threadIdx.y + 8 * r;
            if (k <= g.nnz + 1 && i <= g.nnx + 3)
                tile[q][threadIdx.y + 8 * r][threadIdx.x] =
                    __ldcs(p + isrc + (long long)g.nnx * (jsrc + (long long)g.nny * k));
        }
    }
    __syncthreads();
    const int k = k0 + (int)threadIdx.x;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int io = i0 + (int)threadIdx.y + 8 * r;
        if (k > g.nnz + 1 || io > g.nnx + 3) continue;
        const long long o = (long long)k + (long long)g.nz2 * ((long long)(j + 1) + (long long)g.ny5 * (io + 1));
        if (every) {
            double v[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) v[q] = tile[q][threadIdx.x][threadIdx.y + 8 * r];
            S.all(o, v);
        } else {
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (s.p[q]) S.one(q, o, tile[q][threadIdx.x][threadIdx.y + 8 * r]);
        }
    }
}

template <bool MIXED>
__global__ void __launch_bounds__(256) k_fill_flow(const __grid_constant__ DevBox B, FieldSrc s) {
    step_kernel_begin();
    __shared__ double tile[5][32][33];
    if constexpr (MIXED) {
        const bool first = blockIdx.x + blockIdx.y + blockIdx.z == 0 && threadIdx.x + threadIdx.y == 0;
        fill_tile(s, B.g, store32(B, s, (long long)B.g.nnx * B.g.nny, first), tile);   // (i, j, k) = (1, 1, 1)
    } else {
        fill_tile(s, B.g, StoreF64{const_cast<Node64 *>(B.f64), const_cast<double *>(B.fw64)}, tile);
    }
}

// halo-padded layout, the stored order already
template <bool MIXED>
__global__ void __launch_bounds__(256) k_fill_ext(const __grid_constant__ DevBox B, FieldSrc s, long long n) {
    const bool every = s.p[0] && s.p[1] && s.p[2] && s.p[3] && s.p[4];
    auto put = [&](const auto &S) {
        const long long stride = (long long)gridDim.x * blockDim.x;
        for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += stride) {
            if (every) {
                const double v[5] = {s.p[0][o], s.p[1][o], s.p[2][o], s.p[3][o], s.p[4][o]};
                S.all(o, v);
            } else {
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (s.p[q]) S.one(q, o, s.p[q][o]);
            }
        }
    };
    if constexpr (MIXED) put(store32(B, s, f32_ref_index(B.g), blockIdx.x + threadIdx.x == 0));
    else put(StoreF64{const_cast<Node64 *>(B.f64), const_cast<double *>(B.fw64)});
}

void launch_fill_fields(const DevBox &B, const FieldSrc &s, bool flow, cudaStream_t st) {
    const DevGrid &g = B.g;
    if (flow) {
        const dim3 grid((g.nnx + 5 + 31) / 32, (g.nnz + 2 + 31) / 32, g.nny + 5), block(32, 8);
        if (B.f4) launch_step_kernel(k_fill_flow<true>, grid, block, 0, st, B, s);
        else launch_step_kernel(k_fill_flow<false>, grid, block, 0, st, B, s);
        return;
    }
    const long long n = (long long)g.nz2 * g.ny5 * g.nx5;
    const int blocks = (int)std::min<long long>((n + 255) / 256, 148 * 16);
    if (B.f4) k_fill_ext<true><<<blocks, 256, 0, st>>>(B, s, n);
    else k_fill_ext<false><<<blocks, 256, 0, st>>>(B, s, n);
}

// ---- download: list-order position of every survivor -----------------------
__global__ void k_mark_lid(const DevBox *boxes, int box, int *flag) {
    const DevBox &B = boxes[box];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= *B.n_alive) return;
    flag[B.st[B.cur].lid[B.perm[t]]] = 1;
}

// exclusive scan of the flags -> rank, over tiles of kFlagTile flags (four
// consecutive per thread): tile sums, one block over the sums, tile scans.
// One block over all flags is bound by its chain of block scans (14.7 ms for
// 16.8 M flags); three passes read and write the flags once each.
constexpr int kFlagThreads = 256, kFlagTile = 4 * kFlagThreads;

__device__ __forceinline__ int block_exclusive(int v, int *total) {
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int s = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        wsum[lane] = s;
    }
    __syncthreads();
    const int before = w ? wsum[w - 1] : 0;
    *total = wsum[(blockDim.x >> 5) - 1];
    __syncthreads();   // wsum is free for the next call
    return before + x - v;
}

__global__ void __launch_bounds__(kFlagThreads) k_flag_sums(const int *flag, int n, int *sums) {
    int s = 0;
    const long long base = (long long)blockIdx.x * kFlagTile;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const long long i = base + k * kFlagThreads + threadIdx.x;
        if (i < n) s += flag[i];
    }
    int total;
    block_exclusive(s, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_flag_offsets(int *sums, int ntiles) {
    int carry = 0;
    for (int base = 0; base < ntiles; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < ntiles ? sums[i] : 0;
        int total;
        const int e = block_exclusive(v, &total);
        if (i < ntiles) sums[i] = carry + e;
        carry += total;
    }
}

__global__ void __launch_bounds__(kFlagThreads) k_flag_ranks(int *flag, int n, const int *offs) {
    const long long base = (long long)blockIdx.x * kFlagTile + 4 * threadIdx.x;
    int v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = base + k < n ? flag[base + k] : 0;
        s += v[k];
    }
    int total;
    int run = offs[blockIdx.x] + block_exclusive(s, &total);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < n) flag[base + k] = run;
        run += v[k];
    }
}

// scratch: an int per kFlagTile flags
void launch_rank_alive(DevBox *boxes, int box, int *rank_by_lid, int nlid, int *scratch, cudaStream_t st) {
    if (nlid <= 0) return;
    cudaMemsetAsync(rank_by_lid, 0, sizeof(int) * (size_t)nlid, st);
    // grid sized by nlid: survivors never exceed the uploaded count
    k_mark_lid<<<(nlid + 255) / 256, 256, 0, st>>>(boxes, box, rank_by_lid);
    const int nt = (int)(((long long)nlid + kFlagTile - 1) / kFlagTile);
    k_flag_sums<<<nt, kFlagThreads, 0, st>>>(rank_by_lid, nlid, scratch);
    k_flag_offsets<<<1, 1024, 0, st>>>(scratch, nt);
    k_flag_ranks<<<nt, kFlagThreads, 0, st>>>(rank_by_lid, nlid, scratch);
}

// slot[r]: where in st[cur] the droplet at list position r is
// (rank_by_lid == nullptr: every uploaded droplet is alive, lid is the position)
__global__ void k_slots(const int *__restrict__ perm, const int *__restrict__ lid,
                        const int *__restrict__ rank_by_lid, int *__restrict__ slot, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int s = perm[t], l = lid[s];
    slot[rank_by_lid ? rank_by_lid[l] : l] = s;
}

void launch_slots(const int *perm, const int *lid, const int *rank_by_lid, int *slot, int n, cudaStream_t st) {
    if (n > 0) k_slots<<<(n + 255) / 256, 256, 0, st>>>(perm, lid, rank_by_lid, slot, n);
}

// Droplet arrays into list order: out[r] = src[slot[r]], grid.y = array, four
// list positions per thread.  The list order is random in the cell order, so
// one side of the move is random 8-byte accesses; as reads they cost a sector
// each, as writes (out[rank] = src) a sector read and written back.  For one or
// two arrays, and for those that go to the host one by one.
__global__ void __launch_bounds__(256) k_gather_list(ListGather g, const int *__restrict__ slot, int n) {
    const double *__restrict__ src = g.src[blockIdx.y];
    double *__restrict__ dst = g.dst[blockIdx.y];
    const long long base = (long long)blockIdx.x * 1024 + threadIdx.x;
    int s[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = base + 256 * k < n ? __ldcs(slot + base + 256 * k) : 0;
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = src[s[k]];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (base + 256 * k < n) __stcs(dst + base + 256 * k, v[k]);
}

__global__ void k_gather_list_i32(const int *__restrict__ src, const int *__restrict__ slot, int *__restrict__ dst,
                                  int n) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n) dst[r] = src[slot[r]];
}

// Several arrays: packed into records of RW 32-byte words per droplet in state
// order (sequential), then each list position reads its record (random, but
// whole sectors) and writes every array (sequential).  16 bytes more per value
// than a perfect gather would move, a quarter of what 8-byte reads from random
// sectors do.  14 arrays of 67 M droplets: about 20 -> 9 ms (two steps and the
// read-back 75.6 -> 65.1 ms).
template <int RW>
__global__ void __launch_bounds__(256) k_pack_records(ListGather g, const int *__restrict__ perm,
                                                      Quad64 *__restrict__ rec, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int s = perm[t];
    double v[4 * RW];
#pragma unroll
    for (int k = 0; k < 4 * RW; ++k) v[k] = k < g.n ? __ldcs(g.src[k] + s) : 0.0;
    Quad64 *r = rec + (long long)RW * s;
#pragma unroll
    for (int w = 0; w < RW; ++w) store_quad(r + w, v[4 * w], v[4 * w + 1], v[4 * w + 2], v[4 * w + 3]);
}

template <int RW>
__global__ void __launch_bounds__(256) k_unpack_records(ListGather g, const int *__restrict__ slot,
                                                        const Quad64 *__restrict__ rec, int n) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const Quad64 *p = rec + (long long)RW * __ldcs(slot + r);
    Quad64 q[RW];
#pragma unroll
    for (int w = 0; w < RW; ++w) q[w] = load_quad(p + w);
#pragma unroll
    for (int w = 0; w < RW; ++w) {
        const double v[4] = {q[w].a, q[w].b, q[w].c, q[w].d};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (4 * w + k < g.n) __stcs(g.dst[4 * w + k] + r, v[k]);
    }
}

template <int RW>
static void list_records(const ListGather &g, const int *perm, const int *slot, int n, Quad64 *rec, cudaStream_t st) {
    k_pack_records<RW><<<(n + 255) / 256, 256, 0, st>>>(g, perm, rec, n);
    k_unpack_records<RW><<<(n + 255) / 256, 256, 0, st>>>(g, slot, rec, n);
}

void launch_list_records(const ListGather &all, const int *perm, const int *slot, int n, Quad64 *rec,
                         cudaStream_t st) {
    if (n <= 0) return;
    for (int a = 0; a < all.n; a += kRecordValues) {
        ListGather g{};
        for (int k = a; k < all.n && g.n < kRecordValues; ++k) {
            g.src[g.n] = all.src[k];
            g.dst[g.n++] = all.dst[k];
        }
        if (g.n <= 2) launch_gather_list(g, slot, n, st);
        else if (g.n <= 4) list_records<1>(g, perm, slot, n, rec, st);
        else if (g.n <= 8) list_records<2>(g, perm, slot, n, rec, st);
        else if (g.n <= 12) list_records<3>(g, perm, slot, n, rec, st);
        else list_records<4>(g, perm, slot, n, rec, st);
    }
}

void launch_gather_list(const ListGather &g, const int *slot, int n, cudaStream_t st) {
    if (n > 0 && g.n > 0)
        k_gather_list<<<dim3((unsigned)(((long long)n + 1023) / 1024), g.n), 256, 0, st>>>(g, slot, n);
}

void launch_gather_list_i32(const int *src, const int *slot, int *dst, int n, cudaStream_t st) {
    if (n > 0) k_gather_list_i32<<<(n + 255) / 256, 256, 0, st>>>(src, slot, dst, n);
}

}  // namespace ntlp
