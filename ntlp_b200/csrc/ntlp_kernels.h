// ntlp_kernels.h -- host-side declarations of the kernel launchers.
#pragma once

#include <cuda_runtime.h>

#include "ntlp_dev.cuh"
#include "ntlp_stage64.h"

namespace ntlp {

constexpr int kUpdateThreads = 128;   // droplets per update block
constexpr int kDepositThreads = 256;  // nodes per deposition block (one tile)
constexpr int kCellThreads = 256;     // cells per sort block
constexpr int kScanTile = 2048;       // cells per scan tile
constexpr int kDeferBlocks = 148;     // blocks of the deferred-droplet pass
constexpr int kUpdateLaunches = 3;    // interpolation, droplet body, deferred droplets

// Deposition tile shapes (nodes per tile in x, y, z; 256 nodes each),
// chosen per context by the autotuner.
constexpr int kDepVariants = 3;
constexpr int kDepShape[kDepVariants][3] = {{2, 4, 32}, {4, 4, 16}, {2, 2, 64}};
inline long long deposit_tile_count(int variant, int nnx, int nny, int nnz) {
    const int *s = kDepShape[variant];
    return (long long)((nnx + s[0] - 1) / s[0]) * ((nny + s[1] - 1) / s[1]) * ((nnz + 2 + s[2] - 1) / s[2]);
}
inline long long deposit_tile_count(int nnx, int nny, int nnz) { return deposit_tile_count(0, nnx, nny, nnz); }
// Droplets per block of the update kernels (autotuned).
constexpr int kNtVariants = 2;
constexpr int kNtValues[kNtVariants] = {128, 256};

// The kernels of a step follow one another on one stream, and in a small box
// each runs for a few microseconds, less than it takes to launch the next.  They
// are launched with programmatic stream serialization: a kernel's CTAs may be
// placed while its predecessor's last ones run, and wait in
// step_kernel_begin(), their first statement, until the predecessor has
// completed and its writes are visible.  Nothing runs earlier than before
// but the placement.
// A kernel that fills the SMs' shared memory (EARLY false: the staged
// interpolation, the tiled depositions) lets nothing in before it has
// completed: its successor would run on with the L1 cache that those CTAs left
// it (16.8 M droplets, update: 5.76 ms without, 5.98 with; overflow tiles of the
// spray case: 6.8 and 15 ms).  10,000 droplets on 32^3: update 47 -> 43, sort 29 ->
// 19, deposition 30 -> 24 us.
template <class... KArgs, class... Args>
inline void launch_step_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                               Args &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
#ifdef __CUDACC__
template <bool EARLY = true>
__device__ __forceinline__ void step_kernel_begin() {
    if (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

struct StepIn {
    double dt;
    double inv_dt;   // 1/dt
    int it;
    int istage;
    int write_payload;
};

// FP64, reference operation order (ntlp_fp64.cu)
void launch_update_be64(int ilin, int nt, DevBox *boxes, const Tile *tiles, int ntiles, int nbox,
                        const DevParams &P, StepIn in, cudaStream_t st);
void launch_update_rk3_64(int ilin, DevBox *boxes, const Tile *tiles, int ntiles, const DevParams &P,
                          StepIn in, cudaStream_t st);
void launch_payload64(DevBox *boxes, const Tile *tiles, int ntiles, const DevParams &P, double dt,
                      cudaStream_t st);
// nbox: boxes whose periodic images are deposited as nodes, to be folded in (0:
// none, the tiles on the periodic edges fold their own); runs: the tiles by
// their stage capacity, a launch each; overflow_list: as for the mixed
// deposition, or NULL (tiles above the capacity then merge from global memory
// within the tiled kernel)
void launch_deposit64(int variant, DevBox *boxes, const Tile *tiles, int ntiles, const DevParams &P,
                      cudaStream_t st, int nbox, const TileRun *runs, int nruns,
                      int *overflow_list);
// cells whose droplets a deposition tile stages
inline int deposit_tile_cells(int variant) {
    const int *t = kDepShape[variant];
    return (t[0] + 1) * (t[1] + 1) * (t[2] + 1);
}
constexpr int kOverflowBlocks = 1184; // grid of the overflow tiles

// mixed precision (ntlp_mixed.cu)
// blk_kb > 0 (6th order): the interpolation runs over cell blocks of
// kBlkX x kBlkY x blk_kb cells (blk_tiles: per box, the blocks in the order
// (ipt block, jpt block, kpt block), then kOobBlockTiles tiles with
// start = -1 - r for the out-of-range bucket)
void launch_update_be_mixed(int ilin, int nt, DevBox *boxes, const Tile *tiles, int ntiles, const Tile *tiles128,
                            int ntiles128, int nbox, const DevParams &P, StepIn in, cudaStream_t st, bool tex,
                            int blk_kb, const Tile *blk_tiles, int n_blk_tiles);
constexpr int kBlockThreads = 160;   // threads of a cell-block interpolation CTA
constexpr int kOobBlockTiles = 8;    // tiles per box over the out-of-range bucket
int interp_block_smem(int kb);       // dynamic shared memory of a cell-block CTA
void prepare_interp_block();         // kernel attributes, once per device
// Cells per block in z for a droplet density (droplets per cell).  Update phase
// with 8 / 16 / 32 cells: 16.7 M droplets at 0.98 per cell 5.95 / 5.61 / 6.0 ms, 4 M at
// 1.9 1.21 / 1.18 ms, 67 M at 2 (4 where there are any) 18.8 / 18.2 ms; 1 M at
// 3.6 with 4 / 8 / 16: 0.331 / 0.326 / 0.341 ms, 2 M at 29 0.624 / 0.649 / 0.786 ms.
inline int interp_block_kb(double density) { return density < 3.0 ? 16 : (density < 6.0 ? 8 : 4); }
// Whether the staged blocks beat the per-droplet kernel (the same bits): a block
// of 16 levels stages 2.4 KB of fields per cell column whether it holds
// droplets or not, and its CTAs take turns of latency that a small box cannot
// overlap.  Update phase, per droplet against staged: 0.063 against 0.143 ms (10,000
// droplets, 0.005 per cell), 0.275 against 0.341 (500,000, 0.23), 3.27 against
// 3.53 (8 M, 0.47), 0.121 against 0.126 (250,000, 0.91), 0.190 against 0.188 (500,000,
// 1.8); 0.737 against 0.732 (2 M, 0.93), 5.83 against 5.61 (16.7 M, 0.98), 1.28 against
// 1.18 (4 M, 1.9), 0.637 against 0.624 (2 M, 29); 0.660 against 0.686 (2 M, 56).
// Both rules go by the context's room for droplets; all were measured full.
inline bool interp_staged_pays(double density, double droplets) {
    return density >= 0.75 && density < 40.0 && droplets >= 1e6;
}
inline long long interp_block_count(int kb, int nnx, int nny, int nnz) {
    return (long long)((nnx + kBlkX) / kBlkX) * ((nny + kBlkY) / kBlkY) * ((nnz + kb) / kb);
}
void launch_payload_mixed(DevBox *boxes, const Tile *tiles, int ntiles, const DevParams &P, double dt,
                          cudaStream_t st);
// dense: some box has per-cell sums (cellsum), deposited by the cell-sum
// kernels instead of the tiles
// overflow_list: [2 + tiles] ints of scratch (ntlp_overflow.h), the count 0 on
// entry and on return
void launch_deposit_mixed(int variant, DevBox *boxes, const Tile *tiles, int ntiles, const DevParams &P,
                          cudaStream_t st, int nbox, bool dense, int *overflow_list);
constexpr int kDenseRatio = 16;     // mixed boxes with capacity >= 16 x cells use per-cell sums
constexpr int kDenseBlocks = 1184;  // grid.x of the cell-sum kernels
// grid.x of the periodic fold (x boxes x 6 quantities).  Deposition with one grid of 148
// blocks over (quantity, node), with 50 and with 100 blocks a quantity: 1 M droplets on
// 128^3 0.213 / 0.203 / 0.201 ms (FP64 0.391 / 0.380 / 0.378), 10,000 on 32^3 0.0197 /
// 0.0181 / 0.0183; 16.8 M on 256^3 1.822 -> 1.774.  Twice as many gave 0.002 to
// 0.004 ms on the large boxes and took as much back on the small.
constexpr int kFoldBlocks = 100;
// kernel attributes (dynamic shared memory of the deposition), set once per
// device, on the device that is current; call outside stream capture
void prepare_kernels64();
void prepare_kernels_mixed();
// true exactly once per (current device, which): guards per-device set-up
// (thread-safe); which < kOnceKinds
constexpr int kOnceKinds = 4;
enum { ONCE_DEP64 = 0, ONCE_DEP_MIXED = 1, ONCE_INTERP_BLOCK = 2 };
bool first_on_device(int which);

// sort and bookkeeping (ntlp_sort.cu)
struct SortPlan {
    const Tile *drop_tiles;  // tiles over droplet capacity (kUpdateThreads each)
    int n_drop_tiles;
    const Tile *cell_tiles;  // tiles over ncells+2 buckets (kScanTile each)
    int n_cell_tiles;
    long long *tile_sums;    // [n_cell_tiles]
    const int *box_first_tile;  // [nbox+1] first cell tile of each box
    int nbox;
};
constexpr int kSortLaunches = 5;   // kernels launched by launch_sort
void launch_sort(DevBox *boxes, const SortPlan &plan, cudaStream_t st);
void launch_finish(DevBox *boxes, int nbox, cudaStream_t st);
void launch_reset_step(DevBox *boxes, int nbox, cudaStream_t st);
void launch_keys_initial(DevBox *boxes, const Tile *tiles, int ntiles, cudaStream_t st);

// the stored fields from arrays in device memory (u, v, w, T, q; a NULL array
// leaves its field as it is): from the flow layout with the halo
// (fill_ext on one domain), or from the halo-padded layout
struct FieldSrc {
    const double *p[5];
};
void launch_fill_fields(const DevBox &host_box, const FieldSrc &src, bool flow, cudaStream_t st);

// download: position of each survivor in list order (scratch: (nlid + 1023) / 1024 ints)
void launch_rank_alive(DevBox *boxes, int box, int *rank_by_lid, int nlid, int *scratch, cudaStream_t st);
// the state's slot of each list position; rank_by_lid nullptr: lid is the position
void launch_slots(const int *perm, const int *lid, const int *rank_by_lid, int *slot, int n, cudaStream_t st);
// dst[k][r] = src[k][slot[r]] for 8-byte values (int64 bits pass through unchanged)
constexpr int kListArrays = 36;   // a droplet has 35 8-byte values
struct ListGather {
    const double *src[kListArrays];
    double *dst[kListArrays];
    int n;
};
void launch_gather_list(const ListGather &g, const int *slot, int n, cudaStream_t st);
// the same through records of kRecordValues values at a time; rec: kRecordValues
// * 8 bytes for each slot of the state
constexpr int kRecordValues = 16;
void launch_list_records(const ListGather &g, const int *perm, const int *slot, int n, Quad64 *rec, cudaStream_t st);
void launch_gather_list_i32(const int *src, const int *slot, int *dst, int n, cudaStream_t st);

// x-y column subdomains (ntlp_subdomain.cu)
// emigrants in send order (direction, then lid) by a radix sort
cudaError_t launch_emig_order(const DevBox *boxes, int box, int m, int *slot_out, int *dir_out, cudaStream_t st);
void launch_gather_slots(const void *src, int elem_bytes, const int *slot, void *out, int m, cudaStream_t st);
void launch_gather_slots_i64(const long long *src, const int *slot, long long *out, int m, cudaStream_t st);
void launch_shift_existing(DevBox *boxes, int box, int n, int m, const int *rank_by_lid, cudaStream_t st);
void launch_halo_add(DevBox *boxes, int box, int axis, const double *in, long long n_per_q, cudaStream_t st);

// particle_xy_stats and radius_histogram of one box (ntlp_stats.cu)
constexpr int kStatCols = 64;       // columns per tile (one block)
constexpr int kStatThreads = 256;
constexpr int kStatWarps = kStatThreads / 32;
constexpr int kS0N = 20;            // 0th-order values per partial
struct StatsScratch {
    double *colsum;                 // [(nnx+1)(nny+1)] LWP per column
    double *tile0;                  // [tiles][kS0N]
    double *tileL;                  // [tiles][24][nnz]
    double *out0;                   // [kS0N]
    double *outL;                   // [24][nnz]
    long long *hrad;                // [NTLP_HIST_N]
};
int stats_tile_count(const DevGrid &g);
void launch_stats(const DevBox *boxes, int box, const DevGrid &g, const DevParams *pp, const StatsScratch &w,
                  bool radius_hist, cudaStream_t st);

}  // namespace ntlp
