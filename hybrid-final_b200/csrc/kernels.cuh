// kernels.cuh -- launch wrappers for the per-step kernels (kernels.cu).
//
// Every kernel takes the whole batch: an array of device case descriptors
// and, for the warp-per-cell kernels, a prefix array item_start[ncases+1]
// that maps a global work item to its case.  A single case is a batch of one.
#pragma once
#include <cuda_runtime.h>
#include "dev.cuh"
#include "prof.cuh"

namespace hp {

// A kernel launched so that its start overlaps the end of the kernel before it
// in the stream (programmatic dependent launch; captured into a graph as such
// an edge).  Only for kernels that begin with enter_kernel(): without its wait
// a kernel would run beside the one whose results it reads.  k_fs_resid,
// k_gemm, k_pcg, k_fluid_sweep and k_fluid_diag have none and stay in plain
// stream order, as do the loader's and the allocation-free deposit's kernels.
// Not while a per-kernel profile is recorded: its marks bracket whole kernels.
// Only for launches of up to about half of the threads that fit on the chip: a
// launch's start is then a part of its time.  Measured on a B200, a step in
// plain stream order, with this rule, and with every launch so: 66.0, 63.7
// and 63.6 us at 65x33 with 20 particles per cell, 193, 172 and 172 us at 129x65
// in O2, 1.326, 1.320 and 1.327 ms at 513x257 with 200.
constexpr unsigned long long LAUNCH_NEXT_THREADS = 148 * 1024;
template <class... P, class... A>
inline cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    const unsigned long long threads = (unsigned long long)grid.x * grid.y * grid.z * block.x;
    cfg.numAttrs = prof::g_on || threads > LAUNCH_NEXT_THREADS ? 0 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Dynamic shared memory past the 48 KB that a launch may ask for unannounced;
// per device, so before every such launch.
inline cudaError_t allow_smem(const void *fn, size_t bytes) {
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)
                             : cudaSuccess;
}

struct LaunchCfg {
    int warps_per_block = 4;   // warps per CTA of Move, Deposit's cells and (at least 8) the re-binning
    int pcg_block = 512;       // PCG: threads per CTA
    int pcg_cluster_max = 16;  // PCG: upper bound on CTAs per case
    int move_unroll = 1;       // Move: ring of 5 (1), 4 (2) or 7 (4) chunks of 32 per warp
    int mcc_cells = 16;        // MCC (Ar): most consecutive cells that share collision batches (1, 2, 4, 8, 16)
};

// SMs of the current device
int sm_count();
// cells per warp of a launch on `warps` resident warps, at most `most`
int balanced_group(long long cells, long long warps, int most);
// Move: gather + push + single-cell exit test (src/cuda_Move.cu:181-270)
cudaError_t launch_move(const DevCase *cases, const int *item_start, int ncases, int items, const LaunchCfg &lc,
                        cudaStream_t st);
// SortBoundary: boundary handling + deterministic re-bin (src/cuda_Sortboundary.cu:41-258)
// the power controller of power-driven cases, after Deposit (cases without
// one return at once)
cudaError_t launch_power(DevCase *cases, int ncases, cudaStream_t st);
// surface: some case has dielectric blocks (apply the crossings Move queued)
cudaError_t launch_sort(const DevCase *cases, const int *item_start, int ncases, int items, const LaunchCfg &lc,
                        cudaStream_t st, bool surface);
// MCC, Ar set (src/cuda_mcc.cu:97-106, src/cuda_mccAr.cu:41-232)
// MCC of the Ar/O2 (gas 2) reaction set, one warp per up to four cells (mcc_oxy.cu)
cudaError_t launch_mcc_oxy(const DevCase *cases, const int *item_start, int ncases, int items, int gas,
                           cudaStream_t st);
cudaError_t launch_mcc_ar(const DevCase *cases, const int *item_start, int ncases, int items, const LaunchCfg &lc,
                          cudaStream_t st);
// Deposit: per-cell CIC sums, then node gather + boundary scale + rho/eps0 + RHS
// (src/cuda_Deposit.cu:3-20,30-104,277-325)
// max_smt: the most 1-2-1 smoothing passes any of the cases asks for (0: none)
cudaError_t launch_deposit(const DevCase *cases, const int *cell_items, const int *node_items, int ncases,
                           int n_cell_items, int n_node_items, const LaunchCfg &lc, cudaStream_t st, int max_smt);
// Field: PCG (src/cuda_Field.cu:133-181,942-1072), potential assembly and
// E at nodes (src/cuda_Field.cu:2-42,500-558,698-846).  The PCG runs one
// cluster per case; cases are grouped by cluster size (a launch has one
// cluster shape), and each case's cluster size depends only on its own grid,
// so a case gets the same reduction order alone and inside any batch.
struct PcgGroup {
    int cluster;      // CTAs per case (above 16: one cooperative launch per case over the grid)
    int block;        // threads per CTA
    const int *list;  // device array of case indices
    int n;
    int max_per, max_ngy; // most nodes per CTA and grid rows of its cases
};
// the solve with its state on chip (pcg.cu); done = false where the group's
// launch shape is outside its range.  polls: reads of one word before a wait of
// the whole-GPU form gives up (each is an L2 round trip: seconds)
cudaError_t launch_pcg_chip(const DevCase *cases, const PcgGroup &pg, cudaStream_t st, bool &done,
                            int polls = 1 << 22);
// field_mode 2 (fastsolve.cu): refinement passes with the separable inverse
constexpr int FS_CHUNK = 1024;  // nodes per CTA of the final residual pass; a case's fs_res holds
                                // 2 + 2 * ceil(G / FS_CHUNK) doubles
constexpr int FS_TILE = 32;     // edge of the output tiles of a launch per product
constexpr int FS_CLUSTER_MAX = 10000;    // unknowns up to which one cluster solves a case
constexpr size_t FS_SMEM_MAX = 220 * 1024;
// shared memory of the cluster solve of nx x ny unknowns, and the CTAs of its
// cluster (0: solved by one launch per product)
size_t fs_cluster_smem(int nx, int ny);
int fs_cluster_ctas(int nx, int ny);
struct FastGroup {
    int ctas = 0;              // CTAs per case
    const int *list = nullptr; // device: case indices
    int n = 0;
    size_t smem = 0;
};
struct FastPlan {
    FastGroup groups[2];             // cases solved by one cluster each (8 and 16 CTAs)
    const int *list = nullptr;       // the other cases: device, case indices,
    const int *item_start = nullptr; // prefix of rectangle sizes [n+1],
    const int *tile_start = nullptr; // prefix of output tiles [n+1]
    int n = 0, items = 0, tiles = 0;
    int passes = 3;
    int final_chunks = 0; // max over those cases of ceil(G / FS_CHUNK)
};
cudaError_t launch_fast_field(const DevCase *cases, const FastPlan &fp, cudaStream_t st);
cudaError_t launch_field(const DevCase *cases, const int *node_items, int ncases, int n_node_items,
                         const PcgGroup *groups, int ngroups, const FastPlan *fast, cudaStream_t st,
                         bool circuit = false);
// CTAs per case for a grid of G nodes
int pcg_cluster_for_nodes(int G);
// CTAs of the whole-GPU cooperative PCG for a case of G nodes (0: a cluster suffices)
int pcg_grid_ctas(int G, int block);
// CSR particles (5 arrays of start[C] floats back to back: x, y, vx, vy, vz)
// into the cell-blocked slots of one species; sets cnt and clears nmov
cudaError_t launch_scatter(const DevSpecies &sp, int C, const int *start, const float *src, cudaStream_t st);
// tstep += 1 for every case (device-side step counter, graph friendly)
cudaError_t launch_advance(const DevCase *cases, int ncases, cudaStream_t st);
// running sums of den and phi (N_ave accumulation, src/cuda_Diagnostic.cu:505-547)
// electron energy histogram of the cases whose eedf_every divides the step
cudaError_t launch_eedf(const DevCase *cases, const int *cell_items, int ncases, int n_cell_items, cudaStream_t st);
cudaError_t launch_accumulate(const DevCase *cases, const int *node_items, int ncases, int n_node_items,
                              cudaStream_t st);
// fluid species (fluid.cu): the continuity sweeps, one warp per line, and the
// averaging cycle, one thread per node
struct FluidPlan {
    const int *xl_items = nullptr; // device prefix [n+1] of nfsp x lines per case (0 where held fixed)
    const int *yl_items = nullptr; // the same for the y lines
    int n_x = 0, n_y = 0;          // total line items
    int len_x = 0, len_y = 0;      // longest line in cells (ncx, ncy of the widest case)
    bool any = false;              // some case runs the fluid cycle
};
constexpr size_t FLUID_SMEM_MAX = 200 * 1024;
// warps per CTA of the sweep for lines of up to L cells (0: L too long)
int fluid_sweep_warps(int L);
cudaError_t launch_fluid(const DevCase *cases, const int *node_items, int ncases, int n_node_items,
                         const FluidPlan &fp, cudaStream_t st);
// The same split around the step's particle phases: the sweeps read only the
// fluid arrays (densities, fluxes, the sources of the last averaging cycle)
// and the step counter, and nothing between k_advance and the averaging cycle
// touches those arrays, so fluid_begin (right after k_advance) runs the
// sweeps on a side stream forked from st, concurrently with Field ... Deposit,
// and fluid_end (before the accumulation) joins it back and runs the
// averaging cycle.  Without a side stream, or while a per-kernel profile is
// recorded, fluid_begin does nothing and fluid_end runs launch_fluid.
// fluid_join, for a step that fails in between, only joins (side_work.hpp).
struct FluidFork {
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
cudaError_t fluid_fork_create(FluidFork &f);
void fluid_fork_destroy(FluidFork &f);
cudaError_t fluid_begin(const DevCase *cases, int ncases, const FluidPlan &fp, const FluidFork &f, cudaStream_t st);
cudaError_t fluid_end(const DevCase *cases, const int *node_items, int ncases, int n_node_items, const FluidPlan &fp,
                      const FluidFork &f, cudaStream_t st);
cudaError_t fluid_join(const FluidPlan &fp, const FluidFork &f, cudaStream_t st);

} // namespace hp
