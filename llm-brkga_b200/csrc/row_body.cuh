// row_body.cuh -- one chromosome row by one thread group: build, store, decode, score.
// Shared by the row kernel (one launch per step) and the evolve kernel (whole generations).
#pragma once

#include "row_group.cuh"

namespace bk {

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

constexpr size_t kRowSmemCap = 227 * 1024;  // opt-in dynamic shared memory per CTA
constexpr size_t kSmSharedBytes = 228 * 1024;  // per SM; each CTA takes 1 KB more than it asks for

// instance data that a CTA stages in shared memory: coordinates, or job times
__host__ __device__ inline bool has_points(int kind) {
    return kind == TSP_COORDS || kind == BITSP_COORDS || kind == MOVRP || kind == JOBSCHED;
}

template <int CLS>
__device__ __forceinline__ void stage_points(const PopDesc& sd, float* pts) {
    if (CLS == ROWS_KEYS) {
        for (int i = threadIdx.x; i < sd.n; i += blockDim.x) pts[i] = sd.jt[i];
        return;
    }
    const int npts = (sd.kind == TSP_COORDS) ? sd.n : sd.n + 1;
    const float2* g0 = reinterpret_cast<const float2*>(sd.xy);
    float2* d0 = reinterpret_cast<float2*>(pts);
    for (int i = threadIdx.x; i < npts; i += blockDim.x) d0[i] = g0[i];
    if (sd.kind == BITSP_COORDS) {
        const float2* g1 = reinterpret_cast<const float2*>(sd.xy2);
        for (int i = threadIdx.x; i < npts; i += blockDim.x) d0[npts + i] = g1[i];
    }
}

// Loads of the population's state.  A launch that lasts one step reads what earlier launches
// wrote (read-only path); one that lasts several generations (COH) reads what other SMs wrote
// meanwhile, past its L1.
template <bool COH, typename V>
__device__ __forceinline__ V row_ld(const V* p) {
    return COH ? __ldcg(p) : __ldg(p);
}

// the row that task `task` of a generation builds: children and mutants (costly) first, the
// elite copies last
__device__ __forceinline__ int row_of_task(const PopDesc& sd, int task) {
    return task < sd.P - sd.E ? sd.E + task : task - (sd.P - sd.E);
}

// Row r of population sd (MODE_LSEARCH: the r-th best row).  from: the rows it is built from
// (parents, the elite row copied, the searched row) where the caller has resolved them; pts:
// the instance data staged in shared memory, or null.  Where a row was written, the group's threads have met (g.sync) when this
// returns: any one of them may then publish the row for all.
template <int T, int CLS, bool COH>
__device__ __forceinline__ void row_work(const RowLaunch& L, const PopDesc& sd, int mode, int r, const int2* from,
                                         float* pts, const RowBuf& s, const RowGroup<T>& g) {
    constexpr bool VRP = CLS == ROWS_MOVRP, TSPJ_ROWS = CLS == ROWS_TSPJ, SORTS = CLS != ROWS_KEYS,
                   NSGA = VRP || CLS == ROWS_BITSP;
    const int t = g.tid;
    const int n = sd.n, ld = sd.ld, P = sd.P, E = sd.E, M = sd.M, m = sd.m;
    const int cur = sd.cur;
    if ((mode == MODE_GEN || mode == MODE_NSGA_OFF) && at_limit(sd)) return;
    if (NSGA && mode == MODE_NSGA_REFILL && !sd.advanced) return;
    // local search: task = rank q; the row is the q-th best (the operator form works on
    // rows in rank order already)
    const int lsq = r;
    if (TSPJ_ROWS && mode == MODE_LSEARCH) {
        if (!L.ls_force && (!ls_due(sd) || at_limit(sd))) return;
        if (from) r = from->x;
        else if (!L.ls_force) r = row_ld<COH>(sd.sorted + lsq);
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
    if (!NSGA && mode == MODE_GEN) {
        dst = sd.keys[cur ^ 1];
        fbuf = cur ^ 1;
        gdraw = sd.gen + 1;
        if (r < E) {
            build = BUILD_COPY;
        } else if (r < P - M) {
            // biased crossover (core/solver.hpp:1109-1135; core/cuda_kernels.cuh:120-134)
            build = BUILD_CROSS;
            tag0 = isl | TAG_COIN;
            if (from) {
                pa = from->x;
                pb = from->y;
            } else {
                int2 prk;
                if (sd.parents) {
                    prk = sd.parents[r];
                } else {
                    const uint4 pr = draw4(sd.seed, 0u, (uint32_t)r, gdraw, isl | TAG_PARENT);
                    prk = make_int2((int)pick(pr.x, (uint32_t)E), E + (int)pick(pr.y, (uint32_t)(P - E)));
                }
                pa = row_ld<COH>(sd.sorted + prk.x);
                pb = row_ld<COH>(sd.sorted + prk.y);
            }
        } else {
            build = BUILD_RANDOM;  // mutant (core/solver.hpp:1244-1258)
            tag0 = isl | TAG_MUTANT;
        }
    } else if (mode == MODE_INIT) {
        // Population::initialize keys (core/population.hpp:107-110)
        dst = sd.keys[cur];
        build = BUILD_RANDOM;
        tag0 = isl | TAG_INIT;
    } else if (NSGA && mode == MODE_NSGA_OFF) {
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
    } else if (NSGA && mode == MODE_NSGA_REFILL) {
        // ensure_minimum_diversity refill (core/population.hpp:166-171): rows from the
        // unique count on are replaced by fresh random keys of generation sd.gen
        if (r < __ldg(sd.nu)) return;
        dst = sd.keys[cur];
        gdraw = sd.gen;
        build = BUILD_RANDOM;
        tag0 = TAG_NSGA_REFILL;
    } else if (TSPJ_ROWS && mode == MODE_LSEARCH) {
        // random 2-opt (core/cuda_kernels.cuh:166-246): the row is rewritten in place, and
        // only when the search improved it
    }  // MODE_EVAL: given keys

    if (!NSGA && build == BUILD_COPY) {
        // elite copy (core/population.hpp:700-714), fitness kept
        const int sr = from ? from->x : row_ld<COH>(sd.sorted + r);
        const float4* a = reinterpret_cast<const float4*>(src + (size_t)sr * ld);
        float4* o = reinterpret_cast<float4*>(dst + (size_t)r * ld);
        for (int q = t; q < ld / 4; q += T) o[q] = row_ld<COH>(a + q);
        if (t < m) sd.fit[fbuf][(size_t)r * m + t] = row_ld<COH>(sd.fit[cur] + (size_t)sr * m + t);
        g.sync();
        return;
    }

    const float* given = src + (size_t)(build == BUILD_LOAD ? r : pa) * ld;  // the given row, or parent a
    const bool vec = ((ld & 3) == 0) && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
    auto given_keys = [&](int q) {
        float4 k;
        if (vec) {
            k = row_ld<COH>(reinterpret_cast<const float4*>(given) + q);
        } else {
            k.x = row_ld<COH>(given + 4 * q);
            k.y = (4 * q + 1 < n) ? row_ld<COH>(given + 4 * q + 1) : 0.0f;
            k.z = (4 * q + 2 < n) ? row_ld<COH>(given + 4 * q + 2) : 0.0f;
            k.w = (4 * q + 3 < n) ? row_ld<COH>(given + 4 * q + 3) : 0.0f;
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
    const bool lsearch = TSPJ_ROWS && mode == MODE_LSEARCH;
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
                a = row_ld<COH>(reinterpret_cast<const float4*>(given) + q);
                b = row_ld<COH>(Bv + q);
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
            if (4 * q + 3 < n) {  // four items by two loads that wait for no key
                const int4 a = __ldg(reinterpret_cast<const int4*>(sd.wv) + 2 * q);
                const int4 b = __ldg(reinterpret_cast<const int4*>(sd.wv) + 2 * q + 1);
                tw += (long long)(k.x > 0.5f ? a.x : 0) + (k.y > 0.5f ? a.z : 0) + (k.z > 0.5f ? b.x : 0) + (k.w > 0.5f ? b.z : 0);
                tv += (long long)(k.x > 0.5f ? a.y : 0) + (k.y > 0.5f ? a.w : 0) + (k.z > 0.5f ? b.y : 0) + (k.w > 0.5f ? b.w : 0);
            } else {
                take(k.x, 4 * q);
                take(k.y, 4 * q + 1);
                take(k.z, 4 * q + 2);
            }
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
        auto shifted = [hb, inv](float v, int nb) { return key_bucket(__fmul_rn(__fsub_rn(v, hb), inv), (float)nb, nb); };
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
        movrp_objectives<T>(n, pts ? pts : sd.xy, sd.w, (int)sd.capi, sd.machines, s, g, res);
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
        } else {
            g.sync();
            res[0] = jobsched_makespan<T>(n, pts ? pts : sd.jt, sd.machines, s, g);
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
                    const float2* xy = reinterpret_cast<const float2*>(pts ? pts + (size_t)ob * 2 * (n + 1)
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
                const float2* xy = reinterpret_cast<const float2*>(pts ? pts : sd.xy);
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
            const float old = row_ld<COH>(dfit);
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

}  // namespace bk
