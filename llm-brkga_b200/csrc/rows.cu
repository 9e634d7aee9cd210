// rows.cu -- the fused row kernel of the generation hot path: build a chromosome row, store
// it, decode it (stable argsort) and score it.
//
// A CTA holds blockDim.x / T groups of T threads, each taking whole rows by itself: it
//   1. builds the row in registers: elite copy, biased crossover of two parent rows
//      (128-bit loads, Philox coins), mutant fill, or a load of given keys;
//   2. writes it to the next population buffer (128-bit stores);
//   3. decodes it: the argsort of row_group.cuh (ties to the lower index exactly like the
//      reference's std::sort over (key, index) pairs, configs/tsp_config.hpp:206-225);
//   4. scores the permutation.
// The groups of a CTA work on one population at a time and share its staged coordinates, so a
// row can have as few threads as its barriers and latency are worth while the SM still holds
// as many rows as its shared memory takes.
#include <algorithm>
#include <climits>
#include <map>
#include <mutex>
#include <tuple>

#include "kernels.h"
#include "row_body.cuh"

namespace bk {


size_t points_bytes(int max_points, int kind) {
    return row_align(max_points * (kind == BITSP_COORDS ? 16u : kind == JOBSCHED ? 4u : 8u));
}

// Whether a row's keys stay in shared memory between the histogram and the scatter (14 bytes
// a key instead of 10).  MO-VRP and TSPJ rows need them there (the sort values follow a hash
// of all keys; the local search moves keys about); other rows read them back from the row
// just written (L2): the same time at n = 1000, and more rows fit on an SM.
bool keep_keys(int kind) { return kind == MOVRP || kind == TSPJ; }

size_t row_smem_bytes(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy, int groups_per_cta) {
    const uint32_t r = groups_per_cta < 1 ? 1 : groups_per_cta;
    size_t b = row_align((uint32_t)sizeof(PopDesc)) + (size_t)r * row_slice_bytes(t.block, max_n, keep_keys(kind));
    if (stage_xy && has_points(kind)) b += points_bytes(max_points, kind);
    return b;
}

// One kernel per class of kinds: each holds only its own decode, so the instructions a row
// passes through stay close together and each class has the registers it needs.  A launch
// over several instances has one class (the batch and the server split their launches).
template <int T, int CLS>
__global__ void __launch_bounds__(T * max_groups(T), 1) row_kernel(RowLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int grab[2];

    const RowGroup<T> g;
    const int t = g.tid, groups = T < 1024 ? (int)blockDim.x / T : 1;
    // the descriptor, the groups' slices, the coordinates
    PopDesc& sd = *reinterpret_cast<PopDesc*>(smem_raw);
    unsigned char* base = smem_raw + row_align((uint32_t)sizeof(PopDesc));
    const uint32_t slice = row_slice_bytes(T, L.max_n, L.keep_keys != 0);
    const RowBuf s = row_carve(base + g.rg * slice, T, L.max_n, L.keep_keys != 0);
    float* pts = reinterpret_cast<float*>(base + groups * slice);
    if (CLS != ROWS_KEYS) zero_counters<T>(s, t);  // (that class sorts nothing)
    dep_wait();  // shared memory only above this line

    // Rows come in runs of one population: its descriptor and coordinates are staged once and
    // shared by the CTA's groups, which take the run's rows in turn.  Without a task list the
    // CTA's rows blockIdx, blockIdx + grid, ... are one run, so rows spread over the SMs
    // first.  With one, a CTA takes units of K consecutive tasks (K <= 32), statically or from
    // the work counter (L.work), which lets a CTA that drew short rows take more; a unit
    // splits where its population changes.
    const int K = L.task_group < 1 ? 1 : L.task_group;
    const bool dyn = L.work != nullptr;
    int cur_pid = -1, unit = blockIdx.x * K, used = 0, round = 0;
    Task mine{0, 0};  // task `unit + lane` of the unit
    if (dyn) {
        if (threadIdx.x == 0) grab[0] = atomicAdd(L.work, K);
        __syncthreads();
        unit = grab[0];
    }
    int next_unit = 0;
    for (bool first = true;; first = false) {
        int pid = 0, len = 0;
        if (!L.tasks) {
            if (!first) break;
            len = (L.ntasks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
        } else {
            if (used == K || first) {
                if (!first) {
                    if (dyn) {
                        ++round;
                        if (threadIdx.x == 0) grab[round & 1] = next_unit;
                        __syncthreads();
                        unit = grab[round & 1];
                    } else {
                        unit += gridDim.x * K;
                    }
                }
                if (unit >= L.ntasks) break;
                if (dyn && threadIdx.x == 0) next_unit = atomicAdd(L.work, K);  // used after this unit
                used = 0;
                const int lane = threadIdx.x & 31;
                mine = (lane < K && unit + lane < L.ntasks) ? L.tasks[unit + lane] : Task{-1, 0};
            }
            pid = __shfl_sync(0xffffffffu, mine.pid, used);
            if (pid < 0) {  // past the last task
                used = K;
                continue;
            }
            const unsigned same = __ballot_sync(0xffffffffu, mine.pid == pid) >> used;
            len = __ffs(~same) - 1;  // consecutive tasks of this population
            if (len < 0) len = 32 - used;
        }
        if (pid != cur_pid) {
            const uint32_t* from = reinterpret_cast<const uint32_t*>(L.descs ? L.descs + pid : &L.single);
            __syncthreads();
            for (int i = threadIdx.x; i < (int)(sizeof(PopDesc) / 4); i += blockDim.x)
                reinterpret_cast<uint32_t*>(&sd)[i] = from[i];
            __syncthreads();
            if (L.stage_xy && has_points(sd.kind)) {
                stage_points<CLS>(sd, pts);
                __syncthreads();
            }
            cur_pid = pid;
        }
        const int run0 = used;
        used += len;
    for (int q0 = g.rg; q0 < len; q0 += groups) {
        int r = L.tasks ? __shfl_sync(0xffffffffu, mine.row, run0 + q0) : (int)blockIdx.x + (int)gridDim.x * q0;
        if (!L.tasks && L.mode == MODE_GEN) r = row_of_task(sd, r);
        row_work<T, CLS, false>(L, sd, L.mode, r, nullptr, L.stage_xy ? pts : nullptr, s, g);
    }
    }
    if (dyn && threadIdx.x == 0 && atomicAdd(L.work + 1, 1) == (int)gridDim.x - 1) {
        // every CTA has taken its last unit: leave the counter zero for the next launch
        L.work[0] = 0;
        L.work[1] = 0;
    }
}

// ---------------------------------------------------------------------------------------
// tiles
// ---------------------------------------------------------------------------------------
// threads per row; a tile's second number is the groups of four keys a thread takes
#define BK_TILES(X) X(32) X(64) X(128) X(256) X(512) X(1024)

int tile_groups(int block, int n) { return (n + 4 * block - 1) / (4 * block); }

bool tile_covers(int block, int n) {
    bool compiled = false;
#define X(B) compiled = compiled || block == B;
    BK_TILES(X)
#undef X
    return compiled && tile_groups(block, n) <= kMaxTileGroups;
}

// every thread count that gives a thread 1 .. kMaxTileGroups groups of four keys, fewest threads
// first
int tile_candidates(int n, RowTile* out, int cap) {
    int c = 0;
    for (int b = 32; b <= 1024; b *= 2) {
        const int g = tile_groups(b, n);
        if (!tile_covers(b, n) || c >= cap) continue;
        out[c++] = RowTile{b, g};
        if (g == 1) break;
    }
    return c;
}

// the default: up to four groups a thread; one warp where a sum in index order takes most of
// the time, which more threads do not share (job scheduling, n = 1000, P = 2048: 18 us a
// generation's rows with 32 threads, 21 with 64, 36 with 128).  Few rows take more threads, up to
// one for four keys, while an SM's share of the rows takes three quarters of its threads at
// most: evaluations of n = 921, P = 104 took 11.5 us with 64 threads a row, 6.0 with 256; of TSPJ
// with 100 cities, P = 2000, 10.3 with 32 and 11.4 with the 64 that would take all.
RowTile pick_tile(int n, int kind, int rows) {
    if (n > row_max_n()) return RowTile{0, 0};
    if ((kind == JOBSCHED || kind == CONTINUOUS) && tile_covers(32, n)) return RowTile{32, tile_groups(32, n)};
    int b = 32;
    while (b < 1024 && tile_groups(b, n) > 4) b *= 2;
    const int sms = device_sm_count(), share = (rows + sms - 1) / sms;
    while (rows > 0 && b < 1024 && 2 * b * share <= (share == 1 ? kSmThreads : kSmThreads * 3 / 4) && 4 * b < n) b *= 2;
    return RowTile{b, tile_groups(b, n)};
}

int row_max_n() { return 4 * 1024 * 4; }

int row_max_n_global() { return 1 << 22; }

// The longest rows decoded in shared memory: a counter per key of the tile that covers n and
// 12 bytes a key, which is the line that callers of MO-VRP, batches and the server know.  (The
// slices above take less: up to 16 384 keys would fit.  Rows in between go to row_kernel_big.)
bool row_needs_global(int n, int pts, int kind) {
    (void)pts;
    // rows of an external-fitness problem are only built: the global kernel builds them
    // without a sort buffer in shared memory
    if (kind == EXTERNAL) return true;
    if (n > row_max_n()) return true;
    const size_t cap = n <= 8192 ? 8192 : (n <= 12288 ? 12288 : 16384);
    return cap * 4 + 16 + row_align(8u * n) + row_align(4u * n) > kRowSmemCap;
}

using RowFn = void (*)(RowLaunch);

static RowFn row_fn(const RowTile& t, int cls) {
#define X(B)                                                                                   \
    if (t.block == B)                                                                          \
        return cls == ROWS_MOVRP ? row_kernel<B, ROWS_MOVRP>                                   \
               : cls == ROWS_TSPJ ? row_kernel<B, ROWS_TSPJ>                                   \
               : cls == ROWS_KEYS ? row_kernel<B, ROWS_KEYS>                                   \
               : cls == ROWS_BITSP ? row_kernel<B, ROWS_BITSP> : row_kernel<B, ROWS_ORDER>;
    BK_TILES(X)
#undef X
    return nullptr;
}

int row_groups_per_cta(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy, int rows) {
    // an SM's share of the rows in as few rounds as shared memory and 1024 threads allow, in as
    // few CTAs as that takes: one CTA of 14 rows an SM against four of four (n = 1000,
    // P = 2048, 64 threads a row): 21.5 against 26.5 us a generation, since every SM then has
    // the same number of rows and stages the coordinates once
    const int sms = device_sm_count(), share = (rows + sms - 1) / sms;
    int best = 1, best_rounds = INT_MAX, best_ctas = 0;
    for (int r = std::min(max_groups(t.block), share); r >= 1; --r) {
        const size_t b = row_smem_bytes(t, max_n, max_points, kind, stage_xy, r);
        if (b > kRowSmemCap) continue;
        const int ctas = std::min<int>((int)(kSmSharedBytes / (b + 1024)), kSmThreads / (t.block * r));
        if (ctas < 1) continue;
        const int rounds = (share + ctas * r - 1) / (ctas * r);
        const int used = (share + r * rounds - 1) / (r * rounds);  // CTAs per SM that these rounds need
        if (rounds < best_rounds || (rounds == best_rounds && used <= best_ctas)) {
            best_rounds = rounds;
            best_ctas = used;
            best = r;  // the smallest r of the fewest CTAs: rows spread evenly
        }
    }
    return best;
}

// 512 threads a CTA, two CTAs an SM: 64 island instances of 100 .. 2000 cities took 102 ms for
// 250 generations, 106 ms with 256 threads, 146 ms with one row per CTA
int row_groups_shared(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy) {
    int r = std::max(1, std::min(max_groups(t.block), 512 / t.block));
    while (r > 1 && row_smem_bytes(t, max_n, max_points, kind, stage_xy, r) > kSmSharedBytes / 2 - 1024) --r;
    return r;
}

cudaError_t prepare_rows(const RowTile& tile, int kind, int groups_per_cta, size_t smem, int* per_sm) {
    RowFn fn = row_fn(tile, row_class(kind));
    if (!fn) return cudaErrorInvalidValue;
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(fn), smem);
    if (e != cudaSuccess) return e;
    // asked once per (kernel, CTA shape): the occupancy calculation costs microseconds of
    // host time, and operator calls make one launch each
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> known;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto key = std::make_tuple(dev, reinterpret_cast<const void*>(fn), groups_per_cta, smem);
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(key);
    if (it == known.end()) {
        int occ = 0;
        const cudaError_t o = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, tile.block * groups_per_cta, smem);
        if (o != cudaSuccess) return o;
        if (known.size() > 4096) known.clear();
        it = known.emplace(key, occ).first;
    }
    *per_sm = it->second;
    return cudaSuccess;
}

cudaError_t launch_rows(const RowLaunch& L, int kind, const RowTile& tile, int grid, cudaStream_t s) {
    if (tile.block == 0) return launch_rows_global(L, kind, grid, s);
    RowFn fn = row_fn(tile, row_class(kind));
    if (!fn || !tile_covers(tile.block, L.max_n)) return cudaErrorInvalidValue;
    if (L.ntasks <= 0 || grid <= 0) return cudaSuccess;
    const int groups = L.groups_per_cta < 1 ? 1 : L.groups_per_cta;
    const int unit = L.tasks ? (L.task_group < 1 ? 1 : L.task_group) : groups;
    const int ctas = (L.ntasks + unit - 1) / unit;
    if (grid > ctas) grid = ctas;
    const size_t smem = row_smem_bytes(tile, L.max_n, L.max_points, kind, L.stage_xy != 0, groups);
    RowLaunch A = L;
    A.keep_keys = keep_keys(kind) ? 1 : 0;
    return launch_dep(fn, dim3(grid), dim3(tile.block * groups), smem, s, A);
}

cudaError_t launch_rows_auto(const RowLaunch& L0, int kind, const RowTile& tile, cudaStream_t s) {
    RowLaunch L = L0;
    L.groups_per_cta = row_groups_per_cta(tile, L.max_n, L.max_points, kind, L.stage_xy != 0, L.ntasks);
    const size_t smem = row_smem_bytes(tile, L.max_n, L.max_points, kind, L.stage_xy != 0, L.groups_per_cta);
    int per_sm = 0;
    cudaError_t e = prepare_rows(tile, kind, L.groups_per_cta, smem, &per_sm);
    if (e != cudaSuccess) return e;
    if (per_sm <= 0) return cudaErrorInvalidConfiguration;
    return launch_rows(L, kind, tile, per_sm * device_sm_count(), s);
}

}  // namespace bk
