// evolve.cu -- whole generations of one single-objective population in one launch.
//
// A generation is two dependent steps: the rows, which read the ranks of the last
// generation, and the elite partition, which reads the fitness of every row.  As two
// launches each pays for its start and drain (about 2 us each, more than the work of a
// small population), loads the descriptor again, stages the coordinates again and starts
// with a chain of dependent loads.  Here the CTAs stay (a cooperative launch: all of them
// are resident): each keeps the descriptor, the coordinates and the parents' ranks of its
// own rows (drawn ahead; they depend on seed, row and generation only).
//
// Nor do they meet in barriers (a counter barrier over 148 CTAs took 3500 cycles, twice a
// generation).  What one CTA needs of another carries the number of the step it belongs to:
//   fwords[step & 1][row]  fitness key of a row and the step, published once the row is built
//   swords[rank]           row of that rank and the step
// A CTA waits for the words it reads: all fitness words before it ranks its own rows, the
// two parents' (or one elite's) rank words before it builds a row.  The fitness words order
// all else: a row's keys and fitness are written before its word (the group's threads meet,
// then one of them releases the word), and every CTA has seen every word of the step (acquire)
// before it reads any row of it; a buffer is overwritten two steps later, when every CTA has
// passed the step between.  The rank words carry nothing but their value: whoever reads one
// has ranked the step it belongs to, and so has acquired all of that step's rows.
//
// Results are those of the row and rank kernels: the same row code, the same order by
// (fitness, row).
#include <algorithm>
#include <climits>
#include <cmath>

#include "kernels.h"
#include "row_body.cuh"

namespace bk {

struct EvolveArgs {
    RowLaunch L;
    PopDesc* desc;
    unsigned long long* fwords;  // [2][P]
    unsigned long long* swords;  // [P]
    uint32_t step0;              // steps taken by earlier launches (two per generation at most)
    int gens, ls_count;
};

// Steps are numbered from 1 and wrap past 0, which is what words hold before their first step
// (and stands for "no step" below).  Neighbours differ in their lowest bit across the wrap too: it
// picks one of the two buffers of fitness words.
__host__ __device__ __forceinline__ uint32_t next_step(uint32_t step) { return step == 0xFFFFFFFFu ? 2u : step + 1u; }

__device__ __forceinline__ unsigned long long word_of(uint32_t step, uint32_t v) {
    return ((unsigned long long)step << 32) | v;
}

// the word's value once it carries `step`; 0 and *stuck set when the wait runs out
__device__ __forceinline__ uint32_t await(const unsigned long long* p, uint32_t step, uint32_t polls, int* stuck) {
    unsigned long long w;
    for (uint32_t n = 0; n < polls; ++n) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
        if ((uint32_t)(w >> 32) == step) return (uint32_t)w;
        if ((n & 255u) == 255u && *static_cast<volatile int*>(stuck)) break;  // the CTA has given up
    }
    *stuck = 1;
    return 0u;
}

template <int T, int CLS>
__global__ void __launch_bounds__(T * max_groups(T), 1) evolve_kernel(EvolveArgs A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int stuck;
    constexpr bool TSPJ_ROWS = CLS == ROWS_TSPJ;
    const RowLaunch& L = A.L;
    const RowGroup<T> g;
    const int groups = (int)blockDim.x / T, grid = gridDim.x, c0 = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;

    // the descriptor, the groups' slices, the coordinates, the population's order keys, the
    // parents' ranks and the ranks of this CTA's rows
    PopDesc& sd = *reinterpret_cast<PopDesc*>(smem_raw);
    unsigned char* base = smem_raw + row_align((uint32_t)sizeof(PopDesc));
    const uint32_t slice = row_slice_bytes(T, L.max_n, L.keep_keys != 0);
    const RowBuf s = row_carve(base + g.rg * slice, T, L.max_n, L.keep_keys != 0);
    base += groups * slice;
    float* pts = reinterpret_cast<float*>(base);
    if (L.stage_xy && has_points(L.single.kind)) base += row_align((uint32_t)(L.max_points * (CLS == ROWS_KEYS ? 4 : 8)));
    uint32_t* okeys = reinterpret_cast<uint32_t*>(base);
    base += row_align(4u * (uint32_t)(round_up(L.single.P, 4)));
    int2* par = reinterpret_cast<int2*>(base);
    int* rk = reinterpret_cast<int*>(par + (L.single.P + grid - 1) / grid);

    if (threadIdx.x == 0) stuck = 0;
    for (int i = threadIdx.x; i < (int)(sizeof(PopDesc) / 4); i += blockDim.x)
        reinterpret_cast<uint32_t*>(&sd)[i] = reinterpret_cast<const uint32_t*>(A.desc)[i];
    if (CLS != ROWS_KEYS) zero_counters<T>(s, g.tid);
    __syncthreads();
    if (sd.stuck) return;  // an earlier launch gave up a wait
    const bool staged = L.stage_xy && has_points(sd.kind);
    if (staged) stage_points<CLS>(sd, pts);
    const int P = sd.P, E = sd.E, M = sd.M, mx = sd.maximize;

    // parents' ranks of the children this CTA builds in generation gen (core/solver.hpp:1117-1118)
    auto draw_parents = [&](uint32_t gen) {
        for (int q = threadIdx.x; c0 + grid * q < P - E - M; q += blockDim.x) {
            const uint4 pr = draw4(sd.seed, 0u, (uint32_t)(E + c0 + grid * q), gen, (sd.island << 8) | TAG_PARENT);
            par[q] = make_int2((int)pick(pr.x, (uint32_t)E), E + (int)pick(pr.y, (uint32_t)(P - E)));
        }
    };
    draw_parents(sd.gen + 1u);
    __syncthreads();

    // rank(i) = elements before row i in (fitness key, row) order, for this CTA's rows: a warp per
    // row, four keys per 128-bit load; the keys are the fitness words of `step`
    auto rank_rows = [&](uint32_t step) {
        const unsigned long long* w = A.fwords + (size_t)(step & 1u) * P;
        for (int j = threadIdx.x; j < round_up(P, 4); j += blockDim.x)
            okeys[j] = (j < P) ? await(w + j, step, sd.wait_polls, &stuck) : 0xFFFFFFFFu;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        __syncthreads();
        for (int q = warp; c0 + grid * q < P; q += warps) {
            const int i = row_of_task(sd, c0 + grid * q);
            const uint32_t me = okeys[i];
            int before = 0;
            if (me != 0xFFFFFFFFu) {
                // equal keys of lower rows count too: one compare a key against me + 1 below row i
                for (int j = 4 * lane; j < P; j += 128) {
                    const uint4 k = *reinterpret_cast<const uint4*>(okeys + j);
                    const uint32_t bar = (j + 3 < i) ? me + 1u : me;
                    before += (k.x < bar) + (k.y < bar) + (k.z < bar) + (k.w < bar);
                    if ((j >> 2) == (i >> 2))  // row i's own four
                        before += (j < i && k.x == me) + (j + 1 < i && k.y == me) + (j + 2 < i && k.z == me);
                }
            } else {  // NaN: after every number
                for (int j = lane; j < P; j += 32) before += (okeys[j] != me || j < i) ? 1 : 0;
            }
            before = __reduce_add_sync(0xffffffffu, before);
            if (lane == 0) rk[q] = before;
        }
    };

    uint32_t step = A.step0, ranked = 0;  // ranked: the step whose rank words hold (0: the sorted array)
    for (int left = A.gens; left > 0; --left) {
        step = next_step(step);
        unsigned long long* fw = A.fwords + (size_t)(step & 1u) * P;
        for (int q = g.rg; c0 + grid * q < P; q += groups) {
            const int r = row_of_task(sd, c0 + grid * q);
            // the rows at the ranks this row is built from
            int2 from = make_int2(0, 0);
            if (r < P - M) {
                const int2 pk = (r < E) ? make_int2(r, r) : par[q];
                if (ranked == 0) {
                    from = make_int2(sd.sorted[pk.x], sd.sorted[pk.y]);
                } else if (T == 32 || g.tid < 32) {
                    from.x = (int)await(A.swords + ((lane & 1) ? pk.y : pk.x), ranked, sd.wait_polls, &stuck);
                    from.y = __shfl_sync(0xffffffffu, from.x, 1);
                    from.x = __shfl_sync(0xffffffffu, from.x, 0);
                }
                if (T > 32 && ranked != 0) {
                    if (g.tid == 0) *reinterpret_cast<int2*>(s.red) = from;
                    g.sync();
                    from = *reinterpret_cast<const int2*>(s.red);
                    g.sync();
                }
            }
            row_work<T, CLS, true>(L, sd, MODE_GEN, r, &from, staged ? pts : nullptr, s, g);
            if (g.tid == 0) {
                const unsigned long long w = word_of(step, fitkey(sd.fit[sd.cur ^ 1][r], mx));
                asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(fw + r), "l"(w) : "memory");
            }
        }
        __syncthreads();  // every group is done with the descriptor's state and the last keys
        if (stuck) break;
        draw_parents(sd.gen + 2u);  // while the other CTAs' fitness words arrive
        __syncthreads();
        if (threadIdx.x == 0) {
            sd.cur ^= 1;
            sd.gen += 1u;
        }
        rank_rows(step);
        __syncthreads();
        if (TSPJ_ROWS && A.ls_count > 0 && ls_due(sd)) {
            // the best rows searched, each by the CTA that built it, then ranked again
            // (core/solver.hpp:459-461)
            step = next_step(step);
            fw = A.fwords + (size_t)(step & 1u) * P;
            for (int q = g.rg; c0 + grid * q < P; q += groups) {
                const int r = row_of_task(sd, c0 + grid * q);
                if (rk[q] < A.ls_count) {
                    const int2 at = make_int2(r, rk[q]);
                    row_work<T, CLS, true>(L, sd, MODE_LSEARCH, rk[q], &at, staged ? pts : nullptr, s, g);
                }
                if (g.tid == 0) {
                    const unsigned long long w = word_of(step, fitkey(sd.fit[sd.cur][r], mx));
                    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(fw + r), "l"(w) : "memory");
                }
            }
            __syncthreads();
            rank_rows(step);
            __syncthreads();
        }
        // the rank words, and at the end the plain order
        for (int q = threadIdx.x; c0 + grid * q < P; q += blockDim.x) {
            const int r = row_of_task(sd, c0 + grid * q), k = rk[q];
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(A.swords + k), "l"(word_of(step, (uint32_t)r)) : "memory");
            if (left == 1) sd.sorted[k] = r;
            if (k == 0 && sd.history && (int)sd.gen < sd.hist_cap) sd.history[sd.gen] = sd.fit[sd.cur][r];
        }
        ranked = step;
        __syncthreads();  // the ranks and parents are read
    }
    if (c0 == 0 && threadIdx.x == 0) {
        A.desc->cur = sd.cur;
        A.desc->gen = sd.gen;
    }
    if (threadIdx.x == 0 && stuck) set_stuck(*A.desc);
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
using EvolveFn = void (*)(EvolveArgs);

static EvolveFn evolve_fn(int block, int cls) {
#define X(B)          \
    if (block == B)   \
        return cls == ROWS_TSPJ ? evolve_kernel<B, ROWS_TSPJ> : cls == ROWS_KEYS ? evolve_kernel<B, ROWS_KEYS> : evolve_kernel<B, ROWS_ORDER>;
    X(32) X(64) X(128) X(256) X(512)
#undef X
    return nullptr;
}

static size_t evolve_smem(const EvolvePlan& p, int kind, int n, int P) {
    const uint32_t rows = (P + p.ctas - 1) / p.ctas;
    return row_align((uint32_t)sizeof(PopDesc)) + (size_t)p.groups * row_slice_bytes(p.tile.block, n, p.keep) +
           (p.stage ? points_bytes(n, kind) : 0) + row_align(4u * (uint32_t)round_up(P, 4)) + row_align(12u * rows);
}

// An SM's cycles for a generation, roughly (3 a key, 1/12 a compare of the ranking, two exchanges;
// measured, P = 16 384: n = 20 140 K cycles, here 160 K; n = 3000 690 K, here 1.2 M).
static double generation_cycles(const EvolvePlan& p, int kind, int n, int P, int machines, int ls_count, int ls_moves) {
    const int T = p.tile.block, rows = (P + p.ctas - 1) / p.ctas;
    double row = 3.0 * n;
    if (kind == JOBSCHED)  // a thread passes all jobs for every T-th machine
        row = std::max(row, 2.0 * n * std::ceil((double)machines / T) * T / 32);
    double cycles = 10000.0 + rows * (row + P / 12.0);
    if (ls_count > 0)  // the searched rows may all lie in one CTA; its groups take one at a time
        cycles += std::ceil((double)std::min(ls_count, rows) / p.groups) * ls_moves * (300.0 + 5.0 * n / T);
    return cycles;
}

// Launches are bounded by their work: a launch that fills the SMs keeps the kernels of other streams
// waiting to its end.  A launch costs 4.5 us (n = 1000, P = 2048: 8 generations a launch 18.6 us
// each, 16 18.3, 128 18.0); with 128 of them (2.3 ms) a matrix product beside that solver took
// 868 us instead of 33 alone, six served requests 194 ms instead of 8, with 9 (0.16 ms) 165 us and
// 54 ms.  2^20 of the cycles above are 19 generations of 2048 rows of 1000 keys (0.34 ms), three of
// 2048 rows of 8000.  Populations on less than half the SMs leave the rest to others: 128.  A
// generation that alone takes 4.4 ms and more (a long local search, very many machines) could
// outlast the waits of a launch's CTAs, about a second, and gains nothing from sharing one: it
// goes row launch by row launch.
constexpr double kLaunchCycles = 1 << 20, kGenerationCycles = 1 << 23;
constexpr int kLaunchGens = 128;

bool evolve_plan(int kind, int n, int P, int machines, int ls_count, int ls_moves, int threads, EvolvePlan* out) {
    const int cls = row_class(kind);
    if (kind == EXTERNAL || (cls != ROWS_ORDER && cls != ROWS_TSPJ && cls != ROWS_KEYS)) return false;
    const int sms = device_sm_count(), share = (P + sms - 1) / sms;
    // Threads a row, from runs of 300 generations (us a generation; launches = row + rank kernels):
    // as many as let three quarters of an SM hold its share of the rows at once, up to one per
    // four keys (n = 200, P = 1000: 64 threads 7.0, 128 7.7, launches 10.2), at least one per 16
    // keys (n = 1500, P = 2048: 128 threads 26.5, 64 28.8, launches 30.0).  Not a whole SM, since a
    // launch starts only when all its CTAs fit beside what runs: eight engines of n = 2000, P = 256
    // at once take 52 us a generation of all with 256 threads a row, 80 with the 512 that fill the
    // SMs, and one alone 10.0 and 9.8 (n = 600, P = 1000: 57 and 91, alone 11.8 and 11.6); half an
    // SM cost one alone up to a third (n = 300, P = 600: 8.4, 6.3 with this rule).  Kinds without an
    // order take one warp up to 512 keys, as the sum in index order is most of their time.
    int T = threads;
    if (T == 0) {
        T = 512;
        while (T > 32 && T * share > kSmThreads * 3 / 4) T /= 2;
        while (T > 32 && T / 2 * 4 >= n) T /= 2;
        if (cls == ROWS_KEYS) T = 32;
        while (T < 512 && 16 * T < n) T *= 2;
    }
    // longer rows fill the GPU for long enough that two launches a generation cost nothing
    // (greedy knapsack n = 10 000, P = 1024: launches 110, here 134)
    if (!evolve_fn(T, cls) || n > 16 * T) return false;
    EvolvePlan p;
    p.tile = RowTile{T, tile_groups(T, n)};
    // one-warp rows: eight rows a CTA rather than one or two on every SM, so that fewer CTAs
    // exchange words (n = 52, P = 256: 32 CTAs 5.1, 148 5.7, launches 8.3)
    p.ctas = std::min(sms, T == 32 ? (P + 7) / 8 : P);
    p.stage = has_points(kind);
    // rows of the CTA in as few rounds as its shared memory and 1024 threads allow; the keys kept
    // on chip when that costs no round (a trip to L2 less per row)
    const int rows = (P + p.ctas - 1) / p.ctas;
    int best = INT_MAX;
    for (int keep = 1; keep >= (keep_keys(kind) ? 1 : 0); --keep) {
        EvolvePlan q = p;
        q.keep = keep != 0;
        for (q.groups = std::min(max_groups(T), rows); q.groups >= 1; --q.groups)
            if (evolve_smem(q, kind, n, P) <= kRowSmemCap) break;
        if (q.groups < 1) continue;
        const int rounds = (rows + q.groups - 1) / q.groups;
        if (rounds < best) {
            best = rounds;
            p = q;
        }
    }
    if (best == INT_MAX) return false;
    p.groups = (rows + best - 1) / best;
    p.smem = evolve_smem(p, kind, n, P);
    const double cycles = generation_cycles(p, kind, n, P, machines, ls_count, ls_moves);
    if (cycles > kGenerationCycles) return false;
    const double room = 2 * p.ctas < sms ? kGenerationCycles : kLaunchCycles;
    p.gens = std::max(1, std::min(kLaunchGens, (int)(room / cycles)));
    *out = p;
    return true;
}

cudaError_t launch_evolve(const EvolvePlan& p, int kind, int n, int max_points, PopDesc* desc, int gens, uint32_t step0,
                          int ls_count, int ls_moves, unsigned long long* words, int P, cudaStream_t s) {
    EvolveFn fn = evolve_fn(p.tile.block, row_class(kind));
    if (!fn || p.groups < 1) return cudaErrorInvalidValue;
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(fn), p.smem);
    if (e != cudaSuccess) return e;
    EvolveArgs a = {};
    a.L.mode = MODE_GEN;
    a.L.single.kind = kind;
    a.L.single.P = P;
    a.L.max_n = n;
    a.L.max_points = max_points;
    a.L.stage_xy = p.stage ? 1 : 0;
    a.L.keep_keys = p.keep ? 1 : 0;
    a.L.ls_moves = ls_moves;
    a.desc = desc;
    a.fwords = words;
    a.swords = words + 2 * (size_t)P;
    a.step0 = step0;
    a.gens = gens;
    a.ls_count = ls_count;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ctas);
    cfg.blockDim = dim3(p.tile.block * p.groups);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, fn, a);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace bk
