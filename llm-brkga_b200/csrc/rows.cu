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
#include "row_group.cuh"

namespace bk {

constexpr size_t kSmSharedBytes = 228 * 1024;  // per SM; each CTA takes 1 KB more than it asks for
constexpr size_t kRowSmemCap = 227 * 1024;  // opt-in dynamic shared memory per CTA

// instance data that a CTA stages in shared memory: coordinates, or job times
__host__ __device__ inline bool has_points(int kind) {
    return kind == TSP_COORDS || kind == BITSP_COORDS || kind == MOVRP || kind == JOBSCHED;
}

static size_t points_bytes(int max_points, int kind) {
    return row_align(max_points * (kind == BITSP_COORDS ? 16u : kind == JOBSCHED ? 4u : 8u));
}

// Whether a row's keys stay in shared memory between the histogram and the scatter (14 bytes
// a key instead of 10).  MO-VRP and TSPJ rows need them there (the sort values follow a hash
// of all keys; the local search moves keys about); other rows read them back from the row
// just written (L2): the same time at n = 1000, and more rows fit on an SM.
static bool keep_keys(int kind) { return kind == MOVRP || kind == TSPJ; }

size_t row_smem_bytes(const RowTile& t, int max_n, int max_points, int kind, bool stage_xy, int groups_per_cta) {
    const uint32_t r = groups_per_cta < 1 ? 1 : groups_per_cta;
    size_t b = row_align((uint32_t)sizeof(PopDesc)) + (size_t)r * row_slice_bytes(t.block, max_n, keep_keys(kind));
    if (stage_xy && has_points(kind)) b += points_bytes(max_points, kind);
    return b;
}

__device__ __forceinline__ int tourn(int i1, int i2, const int32_t* rank, const float* cd) {
    const int r1 = __ldg(rank + i1), r2 = __ldg(rank + i2);
    if (r1 < r2) return i1;
    if (r2 < r1) return i2;
    if (__ldg(cd + i1) > __ldg(cd + i2)) return i1;
    return i2;
}

// groups of a CTA at most: 1024 threads (64 registers each, so that an SM holds that many), and
// 15 barriers for groups of more than a warp
__host__ __device__ constexpr int max_groups(int T) { return T == 64 ? 15 : 1024 / T; }
constexpr int kSmThreads = 1024;

// One kernel per class of kinds: each holds only its own decode, so the instructions a row
// passes through stay close together and each class has the registers it needs.  A launch
// over several instances has one class (the batch and the server split their launches).
template <int T, int CLS>
__global__ void __launch_bounds__(T * max_groups(T), 1) row_kernel(RowLaunch L) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr bool VRP = CLS == ROWS_MOVRP, TSPJ_ROWS = CLS == ROWS_TSPJ, SORTS = CLS != ROWS_KEYS,
                   NSGA = VRP || CLS == ROWS_BITSP;
    __shared__ int grab[2];

    const RowGroup<T> g;
    const int t = g.tid, groups = T < 1024 ? (int)blockDim.x / T : 1;
    // the descriptor, the groups' slices, the coordinates
    PopDesc& sd = *reinterpret_cast<PopDesc*>(smem_raw);
    unsigned char* base = smem_raw + row_align((uint32_t)sizeof(PopDesc));
    const uint32_t slice = row_slice_bytes(T, L.max_n, L.keep_keys != 0);
    const RowBuf s = row_carve(base + g.rg * slice, T, L.max_n, L.keep_keys != 0);
    float* pts = reinterpret_cast<float*>(base + groups * slice);
    zero_counters<T>(s, t);
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
            if (CLS == ROWS_KEYS) {
                if (L.stage_xy && sd.kind == JOBSCHED) {
                    for (int i = threadIdx.x; i < sd.n; i += blockDim.x) pts[i] = sd.jt[i];
                    __syncthreads();
                }
            } else if (L.stage_xy && has_points(sd.kind)) {
                const int npts = (sd.kind == TSP_COORDS) ? sd.n : sd.n + 1;
                const float2* g0 = reinterpret_cast<const float2*>(sd.xy);
                float2* d0 = reinterpret_cast<float2*>(pts);
                for (int i = threadIdx.x; i < npts; i += blockDim.x) d0[i] = g0[i];
                if (sd.kind == BITSP_COORDS) {
                    const float2* g1 = reinterpret_cast<const float2*>(sd.xy2);
                    for (int i = threadIdx.x; i < npts; i += blockDim.x) d0[npts + i] = g1[i];
                }
                __syncthreads();
            }
            cur_pid = pid;
        }
        const int run0 = used;
        used += len;
    for (int q0 = g.rg; q0 < len; q0 += groups) {
        const int task = L.tasks ? q0 : (int)blockIdx.x + (int)gridDim.x * q0;
        int r = L.tasks ? __shfl_sync(0xffffffffu, mine.row, run0 + q0) : task;
        const int n = sd.n, ld = sd.ld, P = sd.P, E = sd.E, M = sd.M, m = sd.m;
        const int cur = sd.cur;
        if ((L.mode == MODE_GEN || L.mode == MODE_NSGA_OFF) && at_limit(sd)) continue;
        if (NSGA && L.mode == MODE_NSGA_REFILL && !sd.advanced) continue;
        if (!L.tasks && L.mode == MODE_GEN) r = (task < P - E) ? E + task : task - (P - E);
        // local search: task = rank q; the row is the q-th best (the operator form works on
        // rows in rank order already)
        const int lsq = r;
        if (TSPJ_ROWS && L.mode == MODE_LSEARCH) {
            if (!L.ls_force && (!ls_due(sd) || at_limit(sd))) continue;
            if (!L.ls_force) r = __ldg(sd.sorted + lsq);
        }

        float* dst = nullptr;
        int fbuf = cur, frow = r;  // where the fitness goes: buffer, row
        const uint32_t isl = sd.island << 8;
        // how the row is built: BUILD_LOAD (given keys), BUILD_COPY (elite), BUILD_RANDOM
        // (fresh keys from one stream), BUILD_CROSS (biased crossover), BUILD_NSGA
        // (uniform crossover + per-gene reset)
        enum { BUILD_LOAD, BUILD_COPY, BUILD_RANDOM, BUILD_CROSS, BUILD_NSGA };
        int build = BUILD_LOAD;
        uint32_t gdraw = 0, tag0 = 0;
        const float* src = sd.keys[cur];
        int pa = 0, pb = 0;
        if (!NSGA && L.mode == MODE_GEN) {
            dst = sd.keys[cur ^ 1];
            fbuf = cur ^ 1;
            gdraw = sd.gen + 1;
            if (r < E) {
                build = BUILD_COPY;
            } else if (r < P - M) {
                // biased crossover (core/solver.hpp:1109-1135; core/cuda_kernels.cuh:120-134)
                build = BUILD_CROSS;
                tag0 = isl | TAG_COIN;
                int2 prk;
                if (sd.parents) {
                    prk = sd.parents[r];
                } else {
                    const uint4 pr = draw4(sd.seed, 0u, (uint32_t)r, gdraw, isl | TAG_PARENT);
                    prk = make_int2((int)pick(pr.x, (uint32_t)E), E + (int)pick(pr.y, (uint32_t)(P - E)));
                }
                pa = __ldg(sd.sorted + prk.x);
                pb = __ldg(sd.sorted + prk.y);
            } else {
                build = BUILD_RANDOM;  // mutant (core/solver.hpp:1244-1258)
                tag0 = isl | TAG_MUTANT;
            }
        } else if (L.mode == MODE_INIT) {
            // Population::initialize keys (core/population.hpp:107-110)
            dst = sd.keys[cur];
            build = BUILD_RANDOM;
            tag0 = isl | TAG_INIT;
        } else if (NSGA && L.mode == MODE_NSGA_OFF) {
            // NSGA-II offspring (core/solver.hpp:1019-1091): pool rows [P, 2P) of keys[cur]
            dst = sd.keys[cur] + (size_t)P * ld;
            frow = P + r;
            gdraw = sd.gen + 1;
            if (r >= P - sd.Mn) {
                build = BUILD_RANDOM;
                tag0 = TAG_MUTANT;
            } else {
                build = BUILD_NSGA;
                tag0 = TAG_NSGA_COIN;
                const uint4 pk = draw4(sd.seed, 0u, (uint32_t)r, gdraw, TAG_NSGA_TOUR);
                pa = tourn(pick(pk.x, P), pick(pk.y, P), sd.nrank, sd.ncd);
                pb = tourn(pick(pk.z, P), pick(pk.w, P), sd.nrank, sd.ncd);
            }
        } else if (NSGA && L.mode == MODE_NSGA_REFILL) {
            // ensure_minimum_diversity refill (core/population.hpp:166-171): rows from the
            // unique count on are replaced by fresh random keys of generation sd.gen
            if (r < __ldg(sd.nu)) continue;
            dst = sd.keys[cur];
            gdraw = sd.gen;
            build = BUILD_RANDOM;
            tag0 = TAG_NSGA_REFILL;
        } else if (TSPJ_ROWS && L.mode == MODE_LSEARCH) {
            // random 2-opt (core/cuda_kernels.cuh:166-246): the row is rewritten in place, and
            // only when the search improved it
        }  // MODE_EVAL: given keys

        if (!NSGA && build == BUILD_COPY) {
            // elite copy (core/population.hpp:700-714), fitness kept
            const int sr = __ldg(sd.sorted + r);
            const float4* a = reinterpret_cast<const float4*>(src + (size_t)sr * ld);
            float4* o = reinterpret_cast<float4*>(dst + (size_t)r * ld);
            for (int q = t; q < ld / 4; q += T) o[q] = __ldg(a + q);
            if (t < m) sd.fit[fbuf][(size_t)r * m + t] = __ldg(sd.fit[cur] + (size_t)sr * m + t);
            continue;
        }

        const float* given = src + (size_t)(build == BUILD_LOAD ? r : pa) * ld;  // the given row, or parent a
        const bool vec = ((ld & 3) == 0) && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
        auto given_keys = [&](int q) {
            float4 k;
            if (vec) {
                k = *(reinterpret_cast<const float4*>(given) + q);
            } else {
                k.x = given[4 * q];
                k.y = (4 * q + 1 < n) ? given[4 * q + 1] : 0.0f;
                k.z = (4 * q + 2 < n) ? given[4 * q + 2] : 0.0f;
                k.w = (4 * q + 3 < n) ? given[4 * q + 3] : 0.0f;
            }
            return k;
        };
        auto pad = [&](float4& k, int q, float v) {
            if (4 * q + 3 >= n) {
                if (4 * q + 1 >= n) k.y = v;
                if (4 * q + 2 >= n) k.z = v;
                if (4 * q + 3 >= n) k.w = v;
            }
        };
        const float kNaN = __int_as_float(0x7FFFFFFF);
        const int n4 = round_up(n, 4);
        const int kind = sd.kind;
        const bool lsearch = TSPJ_ROWS && L.mode == MODE_LSEARCH;
        const int split = TSPJ_ROWS ? n / 2 : n;
        auto plain = [](float v, int nb) { return key_bucket(v, (float)nb, nb); };

        // the row's keys, four at a time: built, stored, and handed to the decode's first pass
        long long tw = 0, tv = 0;
        const float4* Bv = reinterpret_cast<const float4*>(src + (size_t)pb * ld);
        float4* o = reinterpret_cast<float4*>(dst + (size_t)r * ld);
#pragma unroll 1
        for (int q = t; 4 * q < n; q += T) {
            float4 k;
            if (build == BUILD_LOAD) {
                k = given_keys(q);
            } else {
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                if (build != BUILD_RANDOM) {
                    a = __ldg(reinterpret_cast<const float4*>(given) + q);
                    b = __ldg(Bv + q);
                }
                // one Philox call site for every way a row is built
                const uint4 x = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, tag0);
                if (build == BUILD_RANDOM) {
                    k.x = u24(x.x);
                    k.y = u24(x.y);
                    k.z = u24(x.z);
                    k.w = u24(x.w);
                } else {
                    const uint32_t Th = sd.rhoT;
                    k.x = ((x.x >> 8) < Th) ? a.x : b.x;
                    k.y = ((x.y >> 8) < Th) ? a.y : b.y;
                    k.z = ((x.z >> 8) < Th) ? a.z : b.z;
                    k.w = ((x.w >> 8) < Th) ? a.w : b.w;
                }
                if (NSGA && build == BUILD_NSGA) {
                    const uint4 mp = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, TAG_NSGA_MUTP);
                    const uint32_t Th = sd.mutT;
                    const bool m0 = (mp.x >> 8) < Th, m1 = (mp.y >> 8) < Th, m2 = (mp.z >> 8) < Th, m3 = (mp.w >> 8) < Th;
                    if (m0 || m1 || m2 || m3) {
                        const uint4 mk = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, TAG_NSGA_MUTK);
                        if (m0) k.x = u24(mk.x);
                        if (m1) k.y = u24(mk.y);
                        if (m2) k.z = u24(mk.z);
                        if (m3) k.w = u24(mk.w);
                    }
                }
                pad(k, q, 0.0f);  // padding lanes (>= n) are zero
                o[q] = k;
            }
            if (VRP || lsearch) {
                reinterpret_cast<float4*>(s.kin)[q] = k;
            } else if (SORTS) {
                pad(k, q, kNaN);
                if (L.keep_keys) reinterpret_cast<float4*>(s.kin)[q] = k;
                count_keys<TSPJ_ROWS>(k, q, split, s, plain);
            } else if (kind == CONTINUOUS) {
                reinterpret_cast<float4*>(s.sk)[q] = k;
            } else if (kind == JOBSCHED) {
                const float mf = (float)sd.machines;
                auto machine = [&](float v) {
                    const int mm = (int)__fmul_rn(v, mf);
                    return mm >= sd.machines ? sd.machines - 1 : (mm < 0 ? 0 : mm);
                };
                reinterpret_cast<int4*>(s.sk)[q] = make_int4(machine(k.x), machine(k.y), machine(k.z), machine(k.w));
            } else {  // KNAP_THRESHOLD: (weight, value) of the items taken
                auto take = [&](float v, int i) {
                    if (i < n && v > 0.5f) {
                        const int2 x = __ldg(sd.wv + i);
                        tw += x.x;
                        tv += x.y;
                    }
                };
                take(k.x, 4 * q);
                take(k.y, 4 * q + 1);
                take(k.z, 4 * q + 2);
                take(k.w, 4 * q + 3);
            }
        }
        // rows whose stride has more padding than the last four keys
        if (build != BUILD_LOAD)
            for (int q = n4 / 4 + t; q < ld / 4; q += T) o[q] = make_float4(0.f, 0.f, 0.f, 0.f);

        if (lsearch) {
            // reverse random segments [i, j] of the city keys (the first n/2 genes), as the
            // reference's random_2opt_kernel: i, j uniform over the cities, ordered, skipped
            // when j - i < 2
            const int c = n / 2;
            float* sk = s.kin;
            g.sync();
            for (int mv = 0; mv < L.ls_moves; ++mv) {
                const uint4 x = draw4(sd.seed, (uint32_t)mv, (uint32_t)lsq, sd.gen, isl | TAG_LS);
                int i = (int)pick(x.x, (uint32_t)c), j = (int)pick(x.y, (uint32_t)c);
                if (i > j) {
                    const int tmp = i;
                    i = j;
                    j = tmp;
                }
                if (j - i >= 2)
                    for (int p = t; p < (j - i + 1) / 2; p += T) {
                        const float u = sk[i + p];
                        sk[i + p] = sk[j - p];
                        sk[j - p] = u;
                    }
                g.sync();
            }
            for (int q = t; 4 * q < n; q += T) {
                float4 k = reinterpret_cast<const float4*>(sk)[q];
                pad(k, q, kNaN);
                reinterpret_cast<float4*>(sk)[q] = k;
                count_keys<true>(k, q, split, s, plain);
            }
        }

        float res[2] = {0.0f, 0.0f};
        // the keys again, for the scatter
        auto keys_again = [&](int q) {
            if (L.keep_keys) return reinterpret_cast<const float4*>(s.kin)[q];
            float4 k;
            if (build == BUILD_LOAD) k = given_keys(q);
            else k = o[q];
            pad(k, q, kNaN);
            return k;
        };
        auto write_perm = [&]() {
            if (L.perm_out) {
                int32_t* po = L.perm_out + (size_t)r * n;
                for (int i = t; i < n; i += T) po[i] = s.perm[i];
            }
        };
        float* ed = reinterpret_cast<float*>(s.sk);
        if constexpr (VRP) {
            // 1. h = the FP32 sum of key_i * (i + 1) in index order; the sort value of gene i
            //    is key_i + (i * 1e-5 + h * 1e-5)  (configs/multi_objective_vrp_config.hpp:219-230)
            float4* kin = reinterpret_cast<float4*>(s.kin);
            for (int q = t; 4 * q < n; q += T) {
                const float4 k = kin[q];
                const float f = (float)(4 * q);
                reinterpret_cast<float4*>(s.sk)[q] = make_float4(__fmul_rn(k.x, f + 1.0f), __fmul_rn(k.y, f + 2.0f),
                                                                 __fmul_rn(k.z, f + 3.0f), __fmul_rn(k.w, f + 4.0f));
            }
            g.sync();
            float h = 0.0f;
            int i = 0;
#pragma unroll 2
            for (; i + 4 <= n; i += 4) {
                const float4 q = *reinterpret_cast<const float4*>(ed + i);
                h = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(h, q.x), q.y), q.z), q.w);
            }
            for (; i < n; ++i) h = __fadd_rn(h, ed[i]);
            const float hb = __fmul_rn(h, 1.0e-5f);
            // 2. the visiting order: values span about [hb, hb + 1 + n * 1e-5], and any
            //    non-decreasing bucket map gives the same (value, index) order
            const float inv = __frcp_rn(__fadd_rn(1.0f, __fmul_rn((float)n, 1.0e-5f)));
            auto shifted = [&](float v, int nb) { return key_bucket(__fmul_rn(__fsub_rn(v, hb), inv), (float)nb, nb); };
            for (int q = t; 4 * q < n; q += T) {
                float4 k = kin[q];
                const float f = (float)(4 * q);
                k.x = __fadd_rn(k.x, __fadd_rn(__fmul_rn(f, 1.0e-5f), hb));
                k.y = __fadd_rn(k.y, __fadd_rn(__fmul_rn(f + 1.0f, 1.0e-5f), hb));
                k.z = __fadd_rn(k.z, __fadd_rn(__fmul_rn(f + 2.0f, 1.0e-5f), hb));
                k.w = __fadd_rn(k.w, __fadd_rn(__fmul_rn(f + 3.0f, 1.0e-5f), hb));
                pad(k, q, kNaN);
                kin[q] = k;
                count_keys<false>(k, q, n, s, shifted);
            }
            sort_row<T, false>(n4, n4, s, g, shifted, keys_again);
            write_perm();
            // 3. routes and objectives
            movrp_objectives<T>(n, L.stage_xy ? pts : sd.xy, sd.w, (int)sd.capi, sd.machines, s, g, res);
            g.sync();
            zero_counters<T>(s, t);
        } else if constexpr (!SORTS) {
            if (kind == KNAP_THRESHOLD) {
                // configs/knapsack_config.hpp:43-62 (integer sums are exact as floats below 2^24)
                tw = group_sum_ll<T>(tw, s, g);
                tv = group_sum_ll<T>(tv, s, g);
                const float twf = (float)tw, tvf = (float)tv;
                res[0] = (twf > sd.cap) ? __fsub_rn(tvf, __fmul_rn(__fsub_rn(twf, sd.cap), 1000.0f)) : tvf;
            } else if (kind == CONTINUOUS) {
                g.sync();
                res[0] = continuous_fitness<T>(n, sd.function, sd.lo, sd.hi, s, g);
                g.sync();
                zero_counters<T>(s, t);  // the terms lay over them
            } else {
                g.sync();
                res[0] = jobsched_makespan<T>(n, L.stage_xy ? pts : sd.jt, sd.machines, s, g);
            }
        } else if constexpr (TSPJ_ROWS) {
            sort_row<T, true>(n4, split, s, g, plain, keys_again);
            write_perm();
            res[0] = tspj_makespan<T>(n / 2, sd.mat, sd.mat2, s, g);
            zero_counters<T>(s, t);
        } else {
            sort_row<T, false>(n4, n4, s, g, plain, keys_again);
            write_perm();
            if constexpr (CLS == ROWS_BITSP) {  // bi-objective TSP: from the depot (point 0) through the cities and back
#pragma unroll 1
                for (int ob = 0; ob < 2; ++ob) {
                    if (kind == BITSP_COORDS) {
                        const float2* xy = reinterpret_cast<const float2*>(L.stage_xy ? pts + (size_t)ob * 2 * (n + 1)
                                                                                      : (ob ? sd.xy2 : sd.xy));
                        tour_edges<T, false>(n, ed, s.perm, [&](const int* id, float* d) {
                            float2 p[5];
#pragma unroll
                            for (int i = 0; i < 5; ++i) p[i] = xy[id[i]];
#pragma unroll
                            for (int i = 0; i < 4; ++i) d[i] = edge_pts(p[i], p[i + 1]);
                        }, g);
                    } else {
                        const float* mat = ob ? sd.mat2 : sd.mat;
                        tour_edges<T, false>(n, ed, s.perm, [&](const int* id, float* d) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) d[i] = __ldg(mat + (size_t)id[i] * (n + 1) + id[i + 1]);
                        }, g);
                    }
                    g.sync();
                    if (ob == 1) zero_counters<T>(s, t);
                    const float v = canon_terms<T>(ed, n + 1, s, g);
                    if (ob == 0) res[0] = v;
                    else res[1] = v;
                    g.sync();
                }
            } else if (kind == TSP_COORDS || kind == TSP_MATRIX) {
                if (kind == TSP_COORDS) {
                    const float2* xy = reinterpret_cast<const float2*>(L.stage_xy ? pts : sd.xy);
                    tour_edges<T, true>(n, ed, s.perm, [&](const int* id, float* d) {
                        float2 p[5];
#pragma unroll
                        for (int i = 0; i < 5; ++i) p[i] = xy[id[i]];
#pragma unroll
                        for (int i = 0; i < 4; ++i) d[i] = edge_pts(p[i], p[i + 1]);
                    }, g);
                } else {
                    const float* mat = sd.mat;
                    tour_edges<T, true>(n, ed, s.perm, [&](const int* id, float* d) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) d[i] = __ldg(mat + (size_t)id[i] * n + id[i + 1]);
                    }, g);
                }
                g.sync();
                zero_counters<T>(s, t);  // the permutation is dead
                res[0] = canon_terms<T>(ed, n, s, g);
            } else if (kind == KNAP_GREEDY) {
                res[0] = knap_greedy<T>(n, sd.wv, sd.capi, s, g);
                g.sync();
                zero_counters<T>(s, t);
            }
        }
        if (lsearch) {
            // keep the searched row only if it is better (restore_if_worse_kernel); thread 0
            // holds the makespan
            if (t == 0) {
                float* dfit = sd.fit[fbuf] + (size_t)r * m;
                const float old = *dfit;
                const int better = sd.maximize ? (res[0] > old) : (res[0] < old);
                if (better) *dfit = res[0];
                *reinterpret_cast<int*>(s.red) = better;
            }
            g.sync();
            if (*reinterpret_cast<const int*>(s.red)) {
                o = reinterpret_cast<float4*>(sd.keys[cur] + (size_t)r * ld);
                for (int q = t; 4 * q < n; q += T) {
                    float4 k = reinterpret_cast<const float4*>(s.kin)[q];
                    pad(k, q, 0.0f);
                    o[q] = k;
                }
            }
        } else if (t == 0) {
            float* dfit = sd.fit[fbuf] + (size_t)frow * m;
            dfit[0] = res[0];
            if (m > 1) dfit[1] = res[1];
        }
        g.sync();
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

static int tile_groups(int block, int n) { return (n + 4 * block - 1) / (4 * block); }

// every thread count that gives a thread 1 .. 16 groups of four keys, fewest threads first
int tile_candidates(int n, RowTile* out, int cap) {
    int c = 0;
    for (int b = 32; b <= 1024; b *= 2) {
        const int g = tile_groups(b, n);
        if (g > 16 || c >= cap) continue;
        out[c++] = RowTile{b, g};
        if (g == 1) break;
    }
    return c;
}

// the default: up to four groups a thread; one warp where a sum in index order takes most of
// the time, which more threads do not share (job scheduling, n = 1000, P = 2048: 18 us a
// generation's rows with 32 threads, 21 with 64, 36 with 128)
RowTile pick_tile(int n, int kind) {
    if (n > row_max_n()) return RowTile{0, 0};
    if ((kind == JOBSCHED || kind == CONTINUOUS) && tile_groups(32, n) <= 16) return RowTile{32, tile_groups(32, n)};
    for (int b = 32; b < 1024; b *= 2)
        if (tile_groups(b, n) <= 4) return RowTile{b, tile_groups(b, n)};
    return RowTile{1024, tile_groups(1024, n)};
}

int row_max_n() { return 4 * 1024 * 4; }

int row_max_n_global() { return 1 << 22; }

// The longest rows decoded in shared memory: a counter per key of the tile that covers n and
// 12 bytes a key.  (The slices above take less; rows in between are long enough for the
// kernels that spread a row over several CTAs.)
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
    if (!fn) return cudaErrorInvalidValue;
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
