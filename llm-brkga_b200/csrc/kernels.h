// kernels.h -- host-side launch interface of the engine's CUDA kernels.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace bk {

enum Mode : int32_t {
    MODE_INIT = 0,
    MODE_GEN = 1,
    MODE_EVAL = 2,
    MODE_NSGA_OFF = 3,
    MODE_NSGA_REFILL = 4,
    MODE_LSEARCH = 5,  // TSPJ random 2-opt on the top ranks (task = rank)
};

// classes of kinds with a row kernel each: one-objective tours and the greedy knapsack (an
// argsort and a sum), TSPJ (two argsorts), MO-VRP (an argsort of derived values), fitness
// straight from the keys, the bi-objective TSP (NSGA-II builds, two tours)
enum RowClass : int32_t { ROWS_ORDER = 0, ROWS_TSPJ = 1, ROWS_MOVRP = 2, ROWS_KEYS = 3, ROWS_BITSP = 4 };
inline int row_class(int kind) {
    if (kind == TSPJ) return ROWS_TSPJ;
    if (kind == MOVRP) return ROWS_MOVRP;
    if (kind == BITSP_COORDS || kind == BITSP_MATRIX) return ROWS_BITSP;
    return (kind == KNAP_THRESHOLD || kind == JOBSCHED || kind == CONTINUOUS) ? ROWS_KEYS : ROWS_ORDER;
}

// one unit of row work: population `pid`, row `row` of that population
struct Task {
    int32_t pid;
    int32_t row;
};

// tile shape chosen per size bucket: threads per row and float4 groups per thread.  A thread
// holds the ranks of its keys in an array of this many groups (row_group.cuh), so no row is
// launched with fewer threads than that covers.
constexpr int kMaxTileGroups = 16;
struct RowTile {
    int block;
    int groups;
};

struct RowLaunch {
    PopDesc* descs;          // device descriptors (nullptr: use `single`)
    PopDesc single;          // descriptor passed by value
    const Task* tasks;       // device task list (nullptr: rows 0..ntasks-1 of `single`)
    int32_t ntasks;
    int32_t mode;
    int32_t* perm_out;       // optional decoded permutations [rows][n] (MODE_EVAL)
    int32_t groups_per_cta;  // row groups per CTA (0, 1: one)
    int32_t keep_keys;       // rows keep their keys in shared memory (set by launch_rows)
    int32_t max_n;           // largest chromosome among the populations launched
    int32_t max_points;      // largest coordinate count (n, or n+1 with a depot)
    int32_t stage_xy;        // stage coordinates in shared memory
    void* gscratch;          // global-scratch kernel (RowTile{0,0}): grid slices of gstride bytes
    size_t gstride;
    int32_t task_group;      // with a task list: tasks dealt to CTAs in units of this many (0, 1: one; <= 32)
    int32_t* work;           // dynamic dealing (batches and the server): [next group, CTAs done],
                             // zero before the launch and left zero by its last CTA; nullptr:
                             // group g goes to CTA g % grid
    int32_t ls_moves;        // MODE_LSEARCH: segment reversals per individual
    int32_t ls_force;        // MODE_LSEARCH: run whatever the generation (operator); rank q = row q
};

// the default tile for `rows` rows of n keys (0: a launch's rows fill the GPU whatever the tile)
RowTile pick_tile(int n, int kind, int rows);
// every compiled tile whose capacity covers n without being far larger (autotuning set)
int tile_candidates(int n, RowTile* out, int cap);
// shared memory bytes for one CTA of the row kernel
size_t row_smem_bytes(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy, int groups_per_cta);
// row groups a CTA of this tile holds in a launch over many populations of mixed sizes
int row_groups_shared(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy);
// row groups a CTA of this tile holds when a launch over one instance has `rows` rows
int row_groups_per_cta(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy, int rows);
// largest n the in-shared-memory row kernel supports
int row_max_n();
// Rows whose sort does not fit in shared memory are decoded by a kernel with its sort
// scratch in global memory: launch_rows with kGlobalTile and RowLaunch::gscratch /
// gstride set (row_global_stride(max_n) bytes for each of the grid's CTAs).
constexpr RowTile kGlobalTile{0, 0};
int row_max_n_global();
bool row_needs_global(int n, int pts, int kind);
size_t row_global_stride(int max_n);
int row_global_grid(int rows, int max_n);
// whether a compiled kernel has this many threads a row and they cover n keys
bool tile_covers(int block, int n);
// one-time set-up for a tile / shared-memory size: raises the dynamic shared-memory limit
// and returns the resident CTAs per SM (0 if the tile cannot run with that much memory)
cudaError_t prepare_rows(const RowTile& tile, int kind, int groups_per_cta, size_t smem, int* per_sm);
// launch the fused row kernel (generation / init / evaluate / NSGA-II offspring) on
// `grid` CTAs (<= resident capacity); prepare_rows must have run for this tile and size
cudaError_t launch_rows(const RowLaunch& L, int kind, const RowTile& tile, int grid, cudaStream_t s);
// the same for rows whose sort does not fit in shared memory (kGlobalTile)
cudaError_t launch_rows_global(const RowLaunch& L, int kind, int grid, cudaStream_t s);
// convenience for one-off launches: prepare + launch with an occupancy-sized grid
cudaError_t launch_rows_auto(const RowLaunch& L, int kind, const RowTile& tile, cudaStream_t s);
// bytes of instance data a CTA stages; whether rows keep their keys in shared memory; groups of
// four keys a thread of a tile takes
size_t points_bytes(int max_points, int kind);
bool keep_keys(int kind);
int tile_groups(int block, int n);

// ---------------------------------------------------------------------------------------
// whole generations of one single-objective population in one launch (evolve.cu)
// ---------------------------------------------------------------------------------------
struct EvolvePlan {
    RowTile tile{};
    int groups = 0;    // row groups per CTA (0: the population is not run this way)
    int ctas = 0;
    bool stage = false, keep = false;
    size_t smem = 0;
    int gens = 0;      // generations of a launch at most
};
// whether populations of P rows of n keys of this kind run in evolve launches, and how
// (threads: per row, 0 = chosen by size; machines: of job scheduling; ls_count rows searched with
// ls_moves moves each)
bool evolve_plan(int kind, int n, int P, int machines, int ls_count, int ls_moves, int threads, EvolvePlan* out);
// `gens` generations of the population at desc (its rows ranked): rows, elite partition, and for
// TSPJ the local search of ls_count rows where due.  words: 3 P 64-bit words of device memory,
// zero before the first launch; step0: a number that no step of an earlier launch is past (a launch
// takes up to kEvolveSteps a generation, and one number more where they wrap).
constexpr uint32_t kEvolveSteps = 2;
cudaError_t launch_evolve(const EvolvePlan& p, int kind, int n, int max_points, PopDesc* desc, int gens, uint32_t step0,
                          int ls_count, int ls_moves, unsigned long long* words, int P, cudaStream_t s);

// raise the shared-memory limit of the sort kernels for populations of up to maxP rows
cudaError_t prepare_sort(int maxP);
// raise (never lower) the dynamic shared-memory limit of a kernel on the current device
cudaError_t raise_smem_limit(const void* fn, size_t smem);

// elite partition of raw fitness segments: sorted[seg*P + r]
cudaError_t launch_sort_raw(const float* fit, int P, int segments, int maximize, int32_t* sorted,
                            cudaStream_t s);
// re-rank after a local search pass: only populations for which it was due
cudaError_t launch_sort_pops_after_ls(PopDesc* descs, int npops, int maxP, cudaStream_t s);
// engine sort: for each population, sort fit[cur^flip]; when flip, swap buffers and gen++;
// history[gen] = best
cudaError_t launch_sort_pops(PopDesc* descs, int npops, int maxP, int flip, cudaStream_t s);
// ring migration between `k` consecutive island descriptors starting at first_pid, for
// `ninst` instances laid out back to back (island descriptors of one instance adjacent)
cudaError_t launch_migrate(PopDesc* descs, int ninst, int k, int migrants, int max_n, cudaStream_t s);

int device_sm_count();

// Launch with programmatic stream serialization: the kernel is scheduled as the one before
// it in the stream drains, and waits for it (dep_wait) before it touches global memory.
// Only kernels that call dep_wait before any global-memory access are launched this way.
template <typename... Args>
inline cudaError_t launch_dep(void (*fn)(Args...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                              Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, args...);
    if (e != cudaSuccess) cudaGetLastError();  // the status is returned, not left behind
    return e;
}

}  // namespace bk
