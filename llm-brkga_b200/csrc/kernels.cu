// kernels.cu -- rows beyond shared memory (row_kernel_big), the elite partition (rank_kernel)
// and island migration.  The fused row kernel is in rows.cu, whole generations in one launch
// in evolve.cu.  The elite partition ranks (fitness key, row) composites by exact counting
// across the grid.
#include <algorithm>
#include <climits>
#include <cstdio>
#include <map>
#include <mutex>
#include <utility>

#include "kernels.h"
#include "row_group.cuh"

namespace bk {

__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Ascending sort of a[0, n) (shared or global memory) by the whole block, any n: the
// bitonic network in its one-direction form (each merge of size k first compares i with
// its mirror inside the k-block, then half-cleaners of stride k/4 .. 1), with a[i] for
// i >= n taken as +infinity.  Such an element is always the higher index of its pair and
// would stay put, so pairs that reach past n are skipped and nothing is padded.
template <int BLOCK>
__device__ void block_sort_u64(unsigned long long* a, int n) {
    const int t = threadIdx.x;
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    const int half = n2 >> 1;
    for (int k = 2; k <= n2; k <<= 1) {
        const int hk = k >> 1;
        for (int p = t; p < half; p += BLOCK) {
            const int base = (p / hk) * k, x = p % hk;
            const int i = base + x, j = base + k - 1 - x;
            if (j < n) {
                const unsigned long long u = a[i], v = a[j];
                if (v < u) {
                    a[i] = v;
                    a[j] = u;
                }
            }
        }
        __syncthreads();
        for (int st = k >> 2; st > 0; st >>= 1) {
            for (int p = t; p < half; p += BLOCK) {
                const int i = ((p & ~(st - 1)) << 1) | (p & (st - 1));
                const int j = i + st;
                if (j < n) {
                    const unsigned long long u = a[i], v = a[j];
                    if (v < u) {
                        a[i] = v;
                        a[j] = u;
                    }
                }
            }
            __syncthreads();
        }
    }
}

// the permutation of a heavy row: each segment's composites sorted, then their indices;
// called rather than inlined, so the kernel keeps its registers for the common path
template <int BLOCK>
__device__ __noinline__ void heavy_row_perm(unsigned long long* sc, int32_t* perm, int n, int split) {
    block_sort_u64<BLOCK>(sc, split);
    if (split < n) block_sort_u64<BLOCK>(sc + split, n - split);
    for (int p = threadIdx.x; p < n; p += BLOCK) perm[p] = (int32_t)(uint32_t)sc[p];
    __syncthreads();
}

// ---------------------------------------------------------------------------------------
// fitness
// ---------------------------------------------------------------------------------------
// exclusive block scan of two 64-bit values at once (red: 64 entries)
template <int BLOCK>
__device__ __forceinline__ void block_excl_scan_ll2(long long a, long long b, long long* red, long long* ea,
                                                    long long* eb, long long* ta, long long* tb) {
    constexpr int NW = BLOCK / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    long long x = a, y = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long xu = __shfl_up_sync(0xffffffffu, x, o);
        const long long yu = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) {
            x += xu;
            y += yu;
        }
    }
    if (lane == 31) {
        red[w] = x;
        red[32 + w] = y;
    }
    __syncthreads();
    if (w == 0) {
        long long sx = (lane < NW) ? red[lane] : 0ll, sy = (lane < NW) ? red[32 + lane] : 0ll;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long xu = __shfl_up_sync(0xffffffffu, sx, o);
            const long long yu = __shfl_up_sync(0xffffffffu, sy, o);
            if (lane >= o) {
                sx += xu;
                sy += yu;
            }
        }
        if (lane < NW) {
            red[lane] = sx;
            red[32 + lane] = sy;
        }
    }
    __syncthreads();
    *ea = ((w > 0) ? red[w - 1] : 0ll) + x - a;
    *eb = ((w > 0) ? red[32 + w - 1] : 0ll) + y - b;
    *ta = red[NW - 1];
    *tb = red[32 + NW - 1];
    __syncthreads();
}

// knapsack greedy in key order: prefix of the sorted items that fits, then a
// first-fit scan of the rest by warp 0 (weights must be >= 0).  The items' (weight, value)
// pairs are first gathered in key order into wv ([n], free scratch after the argsort) by
// the whole block, so the scans read on-chip data instead of one dependent round of loads
// per 32 items.
template <int BLOCK>
__device__ float knap_greedy(const int32_t* perm, int n, const int2* __restrict__ items, long long C,
                             long long* red, long long* shared_misc, int2* wv) {
    const int t = threadIdx.x;
    // one 8-byte load per item from the interleaved (weight, value) table: an item's pair
    // sits in one cache line, so the random gather touches half the lines of two tables
    for (int p = t; p < n; p += BLOCK) wv[p] = __ldg(items + perm[p]);
    __syncthreads();
    const int ch = (n + BLOCK - 1) / BLOCK;
    const int p0 = t * ch, p1 = min(n, p0 + ch);
    long long ws = 0, vs = 0;
    for (int p = p0; p < p1; ++p) {
        const int2 x = wv[p];
        ws += x.x;
        vs += x.y;
    }
    long long S, V, totw, totv;
    block_excl_scan_ll2<BLOCK>(ws, vs, red, &S, &V, &totw, &totv);
    // the prefix: positions whose inclusive prefix weight stays <= C.  Weights are >= 0, so
    // the prefix weight only grows and exactly one position breaks it (none when every item
    // fits); the thread holding it records the prefix's weight, length and value
    if (t == 0 && totw <= C) {
        shared_misc[0] = totw;
        shared_misc[1] = n;
        shared_misc[2] = totv;
    }
    for (int p = p0; p < p1; ++p) {
        const int2 x = wv[p];
        if (S <= C && S + x.x > C) {
            shared_misc[0] = S;
            shared_misc[1] = p;
            shared_misc[2] = V;
        }
        S += x.x;
        V += x.y;
    }
    __syncthreads();
    const long long f = shared_misc[1], v0 = shared_misc[2];
    long long vt = 0;
    if (t < 32 && f < n) {
        // the spare capacity left by the prefix is below the weight of the item that broke
        // it, so it fits in 32 bits from here on; four chunks of 32 items are loaded before
        // they are walked, so the walk waits for one load round per 128 items
        int r = (int)(C - shared_misc[0]);
        for (int b0 = (int)f + 1; b0 < n; b0 += 128) {
            int2 x[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int pos = b0 + 32 * c + t;
                x[c] = (pos < n) ? wv[pos] : make_int2(INT_MAX, 0);
            }
            // one vote for the 128 items: once the spare capacity is small most groups hold
            // no item that fits, and the walk passes them without stepping chunk by chunk
            if (!__any_sync(0xffffffffu, x[0].x <= r || x[1].x <= r || x[2].x <= r || x[3].x <= r)) continue;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                int cur = 0;
                for (;;) {
                    const unsigned mask = __ballot_sync(0xffffffffu, t >= cur && x[c].x <= r);
                    if (!mask) break;
                    const int j = __ffs(mask) - 1;
                    r -= __shfl_sync(0xffffffffu, x[c].x, j);
                    vt += __shfl_sync(0xffffffffu, x[c].y, j);
                    cur = j + 1;
                }
            }
        }
    }
    __syncthreads();
    return (float)(v0 + vt);
}

// TSPJ makespan (configs/tspj_config.hpp:555-585): the city tour from the depot (node 0)
// and back; at each position the arrival time plus the duration of the job type assigned
// to that position; the larger of the tour length and the latest job completion.  perm[0,
// c) is the city order (cities perm+1), perm[c, 2c) the job order (types perm-c+1).  One
// warp adds in the reference's own sequential order, so the value equals the reference's
// fitness function bit for bit.
template <int BLOCK>
__device__ float tspj_makespan(const int32_t* perm, int nc, const float* __restrict__ travel,
                               const float* __restrict__ jobs, float* red) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const size_t D = (size_t)nc + 1;
        float run = 0.0f, mjc = 0.0f;
        for (int c0 = 0; c0 < nc; c0 += 32) {
            const int i = c0 + lane;
            float e = 0.0f, jd = 0.0f;
            if (i < nc) {
                const int city = perm[i] + 1;
                const int prev = (i == 0) ? 0 : perm[i - 1] + 1;
                const int job = perm[nc + i] - nc + 1;
                e = __ldg(travel + (size_t)prev * D + city);
                jd = __ldg(jobs + (size_t)city * D + job);
            }
            const int cnt = min(32, nc - c0);
            for (int q = 0; q < cnt; ++q) {
                run = __fadd_rn(run, __shfl_sync(0xffffffffu, e, q));
                const float jc = __fadd_rn(run, __shfl_sync(0xffffffffu, jd, q));
                mjc = (mjc < jc) ? jc : mjc;
            }
        }
        const float tt = __fadd_rn(run, __ldg(travel + (size_t)(perm[nc - 1] + 1) * D));
        if (lane == 0) red[0] = (tt < mjc) ? mjc : tt;
    }
    __syncthreads();
    const float v = red[0];
    __syncthreads();
    return v;
}

// ContinuousOptGPUConfig (configs/continuous_opt_gpu_config.hpp:114-173): x = key * (upper -
// lower) + lower; sphere sum x^2; Rastrigin 10 n + sum (x^2 - 10 cos(2 pi x)); Rosenbrock
// sum 100 (x_{i+1} - x_i^2)^2 + (1 - x_i)^2.  keys in index order (shared or global memory).
// One warp adds the terms in the reference's sequential order, so sphere and Rosenbrock
// equal the reference's values bit for bit; Rastrigin goes through the device cosf.
template <int BLOCK>
__device__ float continuous_fitness(const float* keys, int n, int fn, float lo, float hi, float* red) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const float range = __fsub_rn(hi, lo);
        const float two_pi = __fmul_rn(2.0f, 3.14159265358979323846f);
        float sum = (fn == FN_RASTRIGIN) ? __fmul_rn(10.0f, (float)n) : 0.0f;
        const int terms = (fn == FN_ROSENBROCK) ? n - 1 : n;
        for (int c0 = 0; c0 < terms; c0 += 32) {
            const int i = c0 + lane;
            float term = 0.0f;
            if (i < terms) {
                const float x = __fadd_rn(__fmul_rn(keys[i], range), lo);
                if (fn == FN_SPHERE) {
                    term = __fmul_rn(x, x);
                } else if (fn == FN_RASTRIGIN) {
                    term = __fsub_rn(__fmul_rn(x, x), __fmul_rn(10.0f, cosf(__fmul_rn(two_pi, x))));
                } else {
                    const float xn = __fadd_rn(__fmul_rn(keys[i + 1], range), lo);
                    const float t1 = __fsub_rn(xn, __fmul_rn(x, x));
                    const float t2 = __fsub_rn(1.0f, x);
                    term = __fadd_rn(__fmul_rn(__fmul_rn(100.0f, t1), t1), __fmul_rn(t2, t2));
                }
            }
            const int cnt = min(32, terms - c0);
            for (int q = 0; q < cnt; ++q) sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, term, q));
        }
        if (lane == 0) red[0] = sum;
    }
    __syncthreads();
    const float v = red[0];
    __syncthreads();
    return v;
}

// JobSchedulingGPUConfig (configs/job_scheduling_gpu_config.hpp:132-148): job i goes to
// machine (int)(key_i * machines), capped at machines - 1; each machine's load adds its
// jobs in index order; the makespan is the largest load.  Lane l of warp w keeps machine
// 32 w + l (and every BLOCK-th after it) and adds the jobs of each 32-job chunk in order,
// so every load equals the reference's sequential float sum bit for bit.
template <int BLOCK>
__device__ float jobsched_makespan(const float* keys, int n, const float* __restrict__ jt, int M, float* red) {
    constexpr int NW = BLOCK / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float mf = (float)M;
    float best = -INFINITY;
    for (int m0 = warp * 32; m0 < M; m0 += BLOCK) {
        float load = 0.0f;
        for (int c0 = 0; c0 < n; c0 += 32) {
            const int i = c0 + lane;
            int mid = -1;
            float v = 0.0f;
            if (i < n) {
                int mm = (int)__fmul_rn(keys[i], mf);
                mid = mm >= M ? M - 1 : (mm < 0 ? 0 : mm);
                v = __ldg(jt + i);
            }
            const int cnt = min(32, n - c0);
            for (int q = 0; q < cnt; ++q) {
                const int mq = __shfl_sync(0xffffffffu, mid, q);
                const float vq = __shfl_sync(0xffffffffu, v, q);
                if (mq == m0 + lane) load = __fadd_rn(load, vq);
            }
        }
        if (m0 + lane < M) best = (best < load) ? load : best;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, best, o);
        best = (best < other) ? other : best;
    }
    if (lane == 0) red[warp] = best;
    __syncthreads();
    float r = red[0];
    for (int w = 1; w < NW; ++w) r = (r < red[w]) ? red[w] : r;
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------------------
// the fused row kernel
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ int tourn(int i1, int i2, const int32_t* rank, const float* cd) {
    const int r1 = __ldg(rank + i1), r2 = __ldg(rank + i2);
    if (r1 < r2) return i1;
    if (r2 < r1) return i2;
    if (__ldg(cd + i1) > __ldg(cd + i2)) return i1;
    return i2;
}

// ---------------------------------------------------------------------------------------
// rows beyond shared memory: the same build and canonical sums, one CTA per row.  The argsort
// takes two levels: the row's keys are dealt to 4096 bins of the key range (a histogram and
// cursors in shared memory; (key, gene) pairs to global scratch, L2-resident), and runs of
// bins of up to kBigChunk keys are sorted in shared memory by the row kernel's argsort, one
// after the other.  Equal keys go by gene, so results equal the other kernel's bit for bit.
// Tours over coordinates are summed chunk by chunk: a point is fetched once, its edges are
// formed from shared memory, and the 256 virtual lanes carry their sums from chunk to chunk.
// With every counter, slot and composite of the row in global scratch instead, n = 65 536,
// P = 512 took 3.2 ms (a dependent L2 round trip per key and step).  One CTA an SM at a time: two of
// half the size put 230 MB of scratch in flight, past L2, and took 1.3 ms.
// ---------------------------------------------------------------------------------------
constexpr int kBigBlock = 1024;
constexpr int kBigBins = 4096;    // four a thread
constexpr int kBigChunk = 10240;  // 18 bytes a key and a counter for each: 218 KB with the bins
constexpr int kBigEdges = 8192;   // edge terms between two sums where the order comes from perm

__host__ __device__ inline size_t big_perm_bytes(int max_n) { return align_up((size_t)max_n * 4, 256); }

size_t row_global_stride(int max_n) { return big_perm_bytes(max_n) + align_up((size_t)max_n * 8, 256); }

// the row slice (its kept keys widened to (key, gene) pairs), bins, first bin of each chunk
__host__ __device__ inline uint32_t big_slice_bytes() { return row_slice_bytes(kBigBlock, kBigChunk, false); }
static size_t big_smem_bytes() { return big_slice_bytes() + kBigChunk * 8 + kBigBins * 4 + kBigBins * 2; }

// f(key, index) for every key of key[0, n) by a block of T threads: 128-bit loads, two of a thread
// in flight ahead of the keys it works on, where the row is aligned
template <int T, typename F>
__device__ __forceinline__ void for_keys(const float* key, int n, int t, F f) {
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(key) & 15) == 0) {
        const float4* k4 = reinterpret_cast<const float4*>(key);
        const int n4 = n / 4, rounds = n4 / T;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (rounds > 0) a = k4[t];
        if (rounds > 1) b = k4[t + T];
        for (int r = 0; r < rounds; ++r) {
            const float4 k = a;
            const int i = 4 * (t + r * T);
            a = b;
            if (r + 2 < rounds) b = k4[t + (r + 2) * T];
            f(k.x, i);
            f(k.y, i + 1);
            f(k.z, i + 2);
            f(k.w, i + 3);
        }
        done = 4 * rounds * T;
    }
    for (int i = done + t; i < n; i += T) f(key[i], i);
}

// Stable argsort of key[0, n): done(p0, m) is called for each chunk in turn, by the whole block,
// positions [p0, p0 + m) holding indices kin[s.perm[p - p0]].y (s.perm and kin are the chunk's;
// the scratch behind s.perm is free).  False, before any call, when a bin holds more than half
// a chunk, as equal or extreme keys do.
template <typename DoneF>
__device__ __forceinline__ bool long_argsort(const float* key, int n, uint2* sc, const RowBuf& s, uint2* kin,
                                             uint32_t* bins, uint16_t* first_bin, const RowGroup<kBigBlock>& g,
                                             DoneF done) {
    constexpr int T = kBigBlock;
    const int t = g.tid, lane = t & 31, warp = t >> 5;
    uint4* b4 = reinterpret_cast<uint4*>(bins);
    b4[t] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for_keys<T>(key, n, t, [&](float k, int) { atomicAdd(&bins[key_bucket(k, (float)kBigBins, kBigBins)], 1u); });
    __syncthreads();
    uint32_t* red = reinterpret_cast<uint32_t*>(s.red);
    const uint4 c = b4[t];
    const uint32_t sum = c.x + c.y + c.z + c.w;
    uint32_t x = sum, big = __reduce_max_sync(0xffffffffu, max(max(c.x, c.y), max(c.z, c.w)));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) {
        red[warp] = x;
        red[32 + warp] = big;
    }
    __syncthreads();
    const uint32_t v = (lane < T / 32) ? red[lane] : 0u;
    const uint32_t start = x - sum + __reduce_add_sync(0xffffffffu, (lane < warp) ? v : 0u);
    big = __reduce_max_sync(0xffffffffu, (lane < T / 32) ? red[32 + lane] : 0u);
    if (big > kBigChunk / 2) {
        __syncthreads();
        return false;
    }
    const uint4 o = make_uint4(start, start + c.x, start + c.x + c.y, start + c.x + c.y + c.z);
    b4[t] = o;
    __syncthreads();
    // chunk of a bin: its start over (kBigChunk - the largest bin), so a chunk's bins hold at
    // most kBigChunk keys; starts grow by less than that, so every chunk has a first bin
    const uint32_t span = kBigChunk - big;
    {
        const uint32_t st[4] = {o.x, o.y, o.z, o.w};
        uint32_t before = t ? bins[4 * t - 1] / span : 0xFFFFFFFFu;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint32_t id = st[l] / span;
            if (id != before) first_bin[id] = (uint16_t)(4 * t + l);
            before = id;
        }
        if (t == T - 1) red[0] = before + 1u;
    }
    __syncthreads();
    const int chunks = (int)red[0];
    // Few chunks: each picks its keys out of the row, read again (L2, coalesced).  Many: the
    // (key, gene) pairs are dealt to their bins in global scratch first, a 32-byte sector for
    // each.  (n = 65 536, 7 chunks: dealing took 90 K cycles a row, 250 K with the scratch not in
    // L2, and 50 K to read back; the seven passes take 154 K whatever is in L2.  Evaluations of 148
    // and 512 rows, passes and dealing: n = 130 000 647, 777 and 2547, 2657 us; n = 170 000, 17
    // chunks, 981, 1029 and 3900, 3569; n = 250 000 1940, 1542 and 7282, 5397.)
    const bool deal = chunks > 15;
    if (deal) {
        for_keys<T>(key, n, t, [&](float k, int i) {
            sc[atomicAdd(&bins[key_bucket(k, (float)kBigBins, kBigBins)], 1u)] =
                make_uint2(__float_as_uint(k), (uint32_t)i);
        });
        __syncthreads();  // a bin's cursor now stands at the next bin's start
    }
    for (int ch = 0; ch < chunks; ++ch) {
        const int b0 = first_bin[ch], b1 = (ch + 1 < chunks) ? first_bin[ch + 1] : kBigBins;
        int p0, p1;
        if (deal) {
            p0 = b0 ? (int)bins[b0 - 1] : 0;
            p1 = (int)bins[b1 - 1];
        } else {
            p0 = (int)bins[b0];  // the starts: without dealing no cursor moves
            p1 = (b1 < kBigBins) ? (int)bins[b1] : n;
        }
        const int m = p1 - p0, m4 = round_up(m, 4);
        if (m == 0) continue;
        const float lo = (float)b0, scale = __fdiv_rn((float)s.nb, (float)(b1 - b0));
        // monotone over the chunk's key range
        auto bucket = [lo, scale](float k, int nb) {
            const float f = __fmul_rn(__fsub_rn(__fmul_rn(k, (float)kBigBins), lo), scale);
            return max((int)fminf(f, (float)nb - 1.0f), 0);
        };
        zero_counters<T>(s, t);
        if (t == 0) red[64] = 0u;
        __syncthreads();
        if (deal) {
            const uint2* part = sc + p0;
            for (int p = t; p < m; p += T) kin[p] = part[p];
        } else {
            // bins are powers of two wide, so a chunk's keys are those between two exact bounds; NaN
            // belongs to the last.  A thread counts its keys of the round, the warp adds up and takes
            // its places with one atomic: a shared atomic takes the SM about eight cycles whatever
            // its lanes, so one per key and pass (a bin's cursor) took 25 K cycles a pass
            const float from = b0 ? (float)b0 / (float)kBigBins : -INFINITY;
            const float to = (float)b1 / (float)kBigBins;
            const bool last = b1 == kBigBins;
            auto mine = [&](float k) { return !(k < from) && (last || k < to); };
            constexpr int U = 8;  // keys a thread and round
            float ahead[U];       // the next round's keys are on their way
            const int rounds = (n + U * T - 1) / (U * T);
            auto fetch = [&](int i0) {
#pragma unroll
                for (int u = 0; u < U; ++u) ahead[u] = (i0 + u * T < n) ? key[i0 + u * T] : 0.0f;
            };
            fetch(t);
            for (int r = 0; r < rounds; ++r) {
                const int i0 = t + r * U * T;
                float k[U];
                int c = 0;
#pragma unroll
                for (int u = 0; u < U; ++u) k[u] = ahead[u];
                if (r + 1 < rounds) fetch(i0 + U * T);
                const bool whole = (r + 1) * U * T <= n;
#pragma unroll
                for (int u = 0; u < U; ++u) c += (mine(k[u]) && (whole || i0 + u * T < n)) ? 1 : 0;
                int x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                uint32_t at = 0u;
                if (lane == 31 && x) at = atomicAdd(&red[64], (uint32_t)x);
                at = __shfl_sync(0xffffffffu, at, 31) + (uint32_t)(x - c);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (mine(k[u]) && (whole || i0 + u * T < n))
                        kin[at++] = make_uint2(__float_as_uint(k[u]), (uint32_t)(i0 + u * T));
            }
        }
        if (t < m4 - m) kin[m + t] = make_uint2(0x7FFFFFFFu, 0xFFFFFFFFu);
        __syncthreads();
        auto keys = [&](int q) {
            const uint4 u = reinterpret_cast<const uint4*>(kin)[2 * q], v = reinterpret_cast<const uint4*>(kin)[2 * q + 1];
            return make_float4(__uint_as_float(u.x), __uint_as_float(u.z), __uint_as_float(v.x), __uint_as_float(v.z));
        };
        for (int q = t; 4 * q < m; q += T) count_keys<false>(keys(q), q, m4, s, bucket);
        sort_row<T, false>(m4, m4, s, g, bucket, keys, kin, m);
        done(p0, m);
        __syncthreads();
    }
    return true;
}

// the sums of the 256 virtual lanes (threads 0 .. 255) in the canonical order: butterflies in
// groups of 32, a fixed tree over the groups
__device__ float lane_tree(float acc, float* red, int t) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    if (t < 256 && (t & 31) == 0) red[t >> 5] = acc;
    __syncthreads();
    const float v = __fadd_rn(__fadd_rn(__fadd_rn(red[0], red[1]), __fadd_rn(red[2], red[3])),
                              __fadd_rn(__fadd_rn(red[4], red[5]), __fadd_rn(red[6], red[7])));
    __syncthreads();
    return v;
}

// canonical sum of a tour's edges in perm (global): every thread forms edge terms, kBigEdges at a
// time in shared memory, then the 256 virtual lanes add theirs in order.  CLOSED as in tour_edges.
template <bool CLOSED, typename EdgeF>
__device__ float long_tour(int m, const int32_t* perm, EdgeF edge, float* ed, float* red, int t) {
    constexpr int T = kBigBlock;
    const int edges = CLOSED ? m : m + 1;
    auto stop = [&](int j) {  // the j-th stop of the tour: edge e joins stops e and e + 1
        if (CLOSED) return perm[j < m ? j : 0];
        return (j == 0 || j > m) ? 0 : perm[j - 1] + 1;
    };
    float acc = 0.0f;
    for (int e0 = 0; e0 < edges; e0 += kBigEdges) {
        const int cnt = min(kBigEdges, edges - e0);
        for (int c = t; 4 * c < cnt; c += T) {
            int id[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) id[i] = stop(min(e0 + 4 * c + i, edges));
            float4 d;
            edge(id, &d.x);
            reinterpret_cast<float4*>(ed)[c] = d;
        }
        __syncthreads();
        if (t < 256)
            for (int e = t; e < cnt; e += 256) acc = __fadd_rn(acc, ed[e]);
        __syncthreads();
    }
    return lane_tree(acc, red, t);
}

// (Rows of an external-fitness problem are only built: as many threads as a row has groups of four
// keys, and no shared memory.)
__global__ void __launch_bounds__(kBigBlock, 1) row_kernel_big(RowLaunch L) {
    constexpr int BLOCK = kBigBlock;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ PopDesc sd;
    __shared__ long long red_ll[64];
    __shared__ float red_f[32];
    __shared__ long long misc[4];
    const int t = threadIdx.x;
    const RowGroup<BLOCK> g;
    const RowBuf s = row_carve(smem_raw, BLOCK, kBigChunk, false);
    uint2* kin = reinterpret_cast<uint2*>(smem_raw + big_slice_bytes());
    uint32_t* bins = reinterpret_cast<uint32_t*>(kin + kBigChunk);
    uint16_t* first_bin = reinterpret_cast<uint16_t*>(bins + kBigBins);
    float* ed = reinterpret_cast<float*>(smem_raw);
    unsigned char* base = static_cast<unsigned char*>(L.gscratch) + (size_t)blockIdx.x * L.gstride;
    int32_t* perm = reinterpret_cast<int32_t*>(base);
    unsigned long long* sc = reinterpret_cast<unsigned long long*>(base + big_perm_bytes(L.max_n));
    int cur_pid = -1;

    for (int task = blockIdx.x; task < L.ntasks; task += gridDim.x) {
        int pid = 0, r = task;
        if (L.tasks) {
            const Task tk = L.tasks[task];
            pid = tk.pid;
            r = tk.row;
        }
        if (pid != cur_pid) {
            __syncthreads();
            if (t == 0) sd = L.descs ? L.descs[pid] : L.single;
            __syncthreads();
            cur_pid = pid;
        }
        const int n = sd.n, ld = sd.ld, P = sd.P, E = sd.E, M = sd.M, m = sd.m;
        const int cur = sd.cur;
        if ((L.mode == MODE_GEN || L.mode == MODE_NSGA_OFF) && at_limit(sd)) continue;
        if (L.mode == MODE_NSGA_REFILL && !sd.advanced) continue;
        if (!L.tasks && L.mode == MODE_GEN) r = (task < P - E) ? E + task : task - (P - E);
        // local search: task = rank q; the row is the q-th best (the operator form works on
        // rows in rank order already)
        const int lsq = r;
        if (L.mode == MODE_LSEARCH) {
            if (!L.ls_force && (!ls_due(sd) || at_limit(sd))) continue;
            if (!L.ls_force) r = __ldg(sd.sorted + lsq);
        }

        enum { BUILD_LOAD, BUILD_COPY, BUILD_RANDOM, BUILD_CROSS, BUILD_NSGA };
        int build = BUILD_LOAD;
        float* dst = nullptr;
        float* dfit = nullptr;
        bool store = true;
        const uint32_t isl = sd.island << 8;
        uint32_t gdraw = 0, tag0 = 0;
        const float* src = sd.keys[cur];
        int pa = 0, pb = 0;
        if (L.mode == MODE_GEN) {
            dst = sd.keys[cur ^ 1];
            dfit = sd.fit[cur ^ 1];
            gdraw = sd.gen + 1;
            if (r < E) {
                build = BUILD_COPY;
            } else if (r < P - M) {
                build = BUILD_CROSS;  // core/solver.hpp:1109-1135
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
                build = BUILD_RANDOM;  // core/solver.hpp:1244-1258
                tag0 = isl | TAG_MUTANT;
            }
        } else if (L.mode == MODE_INIT) {
            dst = sd.keys[cur];
            dfit = sd.fit[cur];
            build = BUILD_RANDOM;
            tag0 = isl | TAG_INIT;
        } else if (L.mode == MODE_NSGA_OFF) {
            dst = sd.keys[cur] + (size_t)P * ld;
            dfit = sd.fit[cur] + (size_t)P * m;
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
        } else if (L.mode == MODE_NSGA_REFILL) {
            if (r < __ldg(sd.nu)) continue;
            dst = sd.keys[cur];
            dfit = sd.fit[cur];
            gdraw = sd.gen;
            build = BUILD_RANDOM;
            tag0 = TAG_NSGA_REFILL;
        } else {
            dfit = sd.fit[cur];
            store = false;
        }

        if (build == BUILD_COPY) {
            const int sr = __ldg(sd.sorted + r);
            const float4* a = reinterpret_cast<const float4*>(src + (size_t)sr * ld);
            float4* o = reinterpret_cast<float4*>(dst + (size_t)r * ld);
            for (int q = t; q < ld / 4; q += blockDim.x) o[q] = __ldg(a + q);
            if (t < m) dfit[(size_t)r * m + t] = __ldg(sd.fit[cur] + (size_t)sr * m + t);
            __syncthreads();
            continue;
        }
        const float* row = src + (size_t)r * ld;
        if (store) {
            const float4* A = reinterpret_cast<const float4*>(src + (size_t)pa * ld);
            const float4* Bv = reinterpret_cast<const float4*>(src + (size_t)pb * ld);
            float4* o = reinterpret_cast<float4*>(dst + (size_t)r * ld);
            for (int q = t; q < ld / 4; q += blockDim.x) {
                float k[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (4 * q < n) {
                    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                    if (build != BUILD_RANDOM) {
                        a = __ldg(A + q);
                        b = __ldg(Bv + q);
                    }
                    const uint4 x = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, tag0);
                    if (build == BUILD_RANDOM) {
                        k[0] = u24(x.x);
                        k[1] = u24(x.y);
                        k[2] = u24(x.z);
                        k[3] = u24(x.w);
                    } else {
                        const uint32_t T = sd.rhoT;
                        k[0] = ((x.x >> 8) < T) ? a.x : b.x;
                        k[1] = ((x.y >> 8) < T) ? a.y : b.y;
                        k[2] = ((x.z >> 8) < T) ? a.z : b.z;
                        k[3] = ((x.w >> 8) < T) ? a.w : b.w;
                    }
                    if (build == BUILD_NSGA) {
                        const uint4 mp = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, TAG_NSGA_MUTP);
                        const uint4 mk = draw4(sd.seed, (uint32_t)q, (uint32_t)r, gdraw, TAG_NSGA_MUTK);
                        const uint32_t T = sd.mutT;
                        if ((mp.x >> 8) < T) k[0] = u24(mk.x);
                        if ((mp.y >> 8) < T) k[1] = u24(mk.y);
                        if ((mp.z >> 8) < T) k[2] = u24(mk.z);
                        if ((mp.w >> 8) < T) k[3] = u24(mk.w);
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l)
                        if (4 * q + l >= n) k[l] = 0.0f;
                }
                o[q] = make_float4(k[0], k[1], k[2], k[3]);
            }
            row = dst + (size_t)r * ld;
        }
        __syncthreads();  // the row's keys are visible to the whole block
        if (sd.kind == EXTERNAL) continue;  // the caller computes the fitness

        float res[2] = {0.0f, 0.0f};
        const int kind = sd.kind;
        if (kind == KNAP_THRESHOLD) {
            long long tw = 0, tv = 0;
            for (int i = t; i < n; i += BLOCK)
                if (row[i] > 0.5f) {
                    tw += __ldg(sd.w + i);
                    tv += __ldg(&sd.wv[i].y);
                }
            tw = block_sum_ll<BLOCK>(tw, red_ll);
            tv = block_sum_ll<BLOCK>(tv, red_ll);
            const float twf = (float)tw, tvf = (float)tv;
            res[0] = (twf > sd.cap) ? __fsub_rn(tvf, __fmul_rn(__fsub_rn(twf, sd.cap), 1000.0f)) : tvf;
        } else if (kind == CONTINUOUS) {
            res[0] = continuous_fitness<BLOCK>(row, n, sd.function, sd.lo, sd.hi, red_f);
        } else if (kind == JOBSCHED) {
            res[0] = jobsched_makespan<BLOCK>(row, n, sd.jt, sd.machines, red_f);
        } else {
            // stable argsort; TSPJ's two segments one after the other
            const int split = (kind == TSPJ) ? n / 2 : n;
            const bool points = kind == TSP_COORDS || kind == BITSP_COORDS;
            const bool want_perm = !points || L.perm_out;
            bool sorted = true, summed = false;
            if (points) {
                // the tour's edges chunk by chunk.  TSP: edge e joins stops e and e + 1, the last the
                // first; bi-objective: from the depot (point 0), edge e joins stops e - 1 and e, back to
                // the depot
                const bool open = kind == BITSP_COORDS;
                const int objs = open ? 2 : 1;
                float acc[2] = {0.0f, 0.0f};
                float2 head[2], last[2];
                float2* pt = reinterpret_cast<float2*>(row_scratch(s, kBigChunk));
                auto chunk = [&](int p0, int m) {
                    if (want_perm)
                        for (int p = t; p < m; p += BLOCK) perm[p0 + p] = (int)kin[s.perm[p]].y;
                    for (int ob = 0; ob < objs; ++ob) {
                        const float2* xy = reinterpret_cast<const float2*>(ob ? sd.xy2 : sd.xy);
                        // the points by local index, all of a thread's fetches in flight
                        constexpr int U = kBigChunk / BLOCK;
                        {
                            float2 f[U];
#pragma unroll
                            for (int u = 0; u < U; ++u) {
                                const int x = t + u * BLOCK;
                                if (x < m) f[u] = __ldg(xy + kin[x].y + (open ? 1 : 0));
                            }
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                if (t + u * BLOCK < m) pt[t + u * BLOCK] = f[u];
                        }
                        __syncthreads();
                        if (p0 == 0) {
                            head[ob] = open ? __ldg(xy) : pt[s.perm[0]];
                            last[ob] = head[ob];
                        }
                        const float2 before = last[ob];
                        last[ob] = pt[s.perm[m - 1]];
                        // the edge into position p0 + p: number p0 + p (open) or p0 + p - 1; the terms take
                        // the places of the sorted keys
                        const int e0 = p0 - (open ? 0 : 1);
#pragma unroll 2
                        for (int p = t; p < m; p += BLOCK)
                            kin[p].x = __float_as_uint(edge_pts(p ? pt[s.perm[p - 1]] : before, pt[s.perm[p]]));
                        __syncthreads();
                        if (t < 256) {
                            // lane t adds the terms whose number is t modulo 256, in order
                            int p = (t - e0) & 255;
                            for (; p < m; p += 256)
                                if (e0 + p >= 0) acc[ob] = __fadd_rn(acc[ob], __uint_as_float(kin[p].x));
                        }
                        __syncthreads();
                    }
                };
                sorted = long_argsort(row, n, reinterpret_cast<uint2*>(sc), s, kin, bins, first_bin, g, chunk);
                if (sorted) {
                    summed = true;
                    for (int ob = 0; ob < objs; ++ob) {
                        const int e = open ? n : n - 1;  // the edge back to the start
                        if (t == (e & 255)) acc[ob] = __fadd_rn(acc[ob], edge_pts(last[ob], head[ob]));
                        res[ob] = lane_tree(acc[ob], red_f, t);
                    }
                }
            } else {
                for (int i0 = 0; i0 < n && sorted; i0 += split) {
                    const int m0 = (i0 == 0) ? split : n - split;
                    sorted = long_argsort(row + i0, m0, reinterpret_cast<uint2*>(sc), s, kin, bins, first_bin, g,
                                          [&](int p0, int m) {
                                              for (int p = t; p < m; p += BLOCK)
                                                  perm[i0 + p0 + p] = i0 + (int)kin[s.perm[p]].y;
                                          });
                }
            }
            if (!sorted) {
                // equal or extreme keys in few bins: the row's composites sorted in place
                for (int i = t; i < n; i += BLOCK) sc[i] = ((unsigned long long)okey(row[i]) << 32) | (uint32_t)i;
                __syncthreads();
                heavy_row_perm<BLOCK>(sc, perm, n, split);
            }
            __syncthreads();
            if (summed) {
                // done with the order
            } else if (kind == TSP_COORDS) {
                const float2* xy = reinterpret_cast<const float2*>(sd.xy);
                res[0] = long_tour<true>(n, perm, [&](const int* id, float* d) {
                    float2 p[5];
#pragma unroll
                    for (int i = 0; i < 5; ++i) p[i] = __ldg(xy + id[i]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) d[i] = edge_pts(p[i], p[i + 1]);
                }, ed, red_f, t);
            } else if (kind == TSP_MATRIX) {
                const float* mat = sd.mat;
                res[0] = long_tour<true>(n, perm, [&](const int* id, float* d) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) d[i] = __ldg(mat + (size_t)id[i] * n + id[i + 1]);
                }, ed, red_f, t);
            } else if (kind == BITSP_COORDS || kind == BITSP_MATRIX) {
                for (int ob = 0; ob < 2; ++ob) {
                    const float2* xy = reinterpret_cast<const float2*>(ob ? sd.xy2 : sd.xy);
                    const float* mat = ob ? sd.mat2 : sd.mat;
                    res[ob] = long_tour<false>(n, perm, [&](const int* id, float* d) {
                        if (kind == BITSP_COORDS) {
                            float2 p[5];
#pragma unroll
                            for (int i = 0; i < 5; ++i) p[i] = __ldg(xy + id[i]);
#pragma unroll
                            for (int i = 0; i < 4; ++i) d[i] = edge_pts(p[i], p[i + 1]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) d[i] = __ldg(mat + (size_t)id[i] * (n + 1) + id[i + 1]);
                        }
                    }, ed, red_f, t);
                }
            } else if (kind == KNAP_GREEDY) {
                res[0] = knap_greedy<BLOCK>(perm, n, sd.wv, sd.capi, red_ll, misc, reinterpret_cast<int2*>(sc));
            } else if (kind == TSPJ) {
                res[0] = tspj_makespan<BLOCK>(perm, n / 2, sd.mat, sd.mat2, red_f);
            }
            if (L.perm_out) {
                int32_t* po = L.perm_out + (size_t)r * n;
                for (int i = t; i < n; i += BLOCK) po[i] = perm[i];
            }
        }
        if (t == 0) dfit[(size_t)r * m] = res[0];
        if (t == 1 && m > 1) dfit[(size_t)r * m + 1] = res[1];
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// elite partition by exact rank counting: the composite key (fitness key << 32 | row) is
// unique, so rank(i) = #{j : key_j < key_i} is a permutation and sorted[rank(i)] = i is
// the stable order.  P^2 compares spread over ceil(P / RK_CH) CTAs per population, TPE
// threads per element (each counts a slice of j), no sort network and no atomics on the
// ranks.  In engine mode the last CTA of a population (completion counter) swaps the
// buffer index and advances the generation; every CTA also draws the parent ranks of its
// slice of the next generation's child rows (they depend only on seed, row, generation).
// ---------------------------------------------------------------------------------------
constexpr int RK_THREADS = 256, RK_TPE = 32, RK_CH = RK_THREADS / RK_TPE;

struct RankArgs {
    PopDesc* descs;       // engine mode (nullptr: raw mode)
    const float* fit;     // raw mode: segments of P fitness values
    int32_t* sorted;
    int P, maximize, flip;
    int only_ls;          // engine mode: only populations whose local search was due
};

__host__ __device__ inline int next_pow2(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

__global__ void __launch_bounds__(RK_THREADS) rank_kernel(RankArgs a) {
    extern __shared__ unsigned long long rk_keys[];
    const int t = threadIdx.x, pop = blockIdx.y;
    dep_wait();
    PopDesc* d = a.descs ? a.descs + pop : nullptr;
    int P, mx, m, buf = 0;
    const float* f;
    int32_t* sorted;
    uint32_t gen_new = 0;
    if (d) {
        // every descriptor field is read before the first branch, so the reads go out
        // together: one round trip before the fitness loads instead of two
        const uint32_t gen = d->gen, gen_limit = d->gen_limit;
        const int ls_interval = d->ls_interval, cur = d->cur;
        const float* f0 = d->fit[0];
        const float* f1 = d->fit[1];
        P = d->P;
        mx = d->maximize;
        m = d->m;
        sorted = d->sorted;
        const bool lim = gen_limit != 0u && gen >= gen_limit;
        if (a.flip && lim) return;
        if (a.only_ls) {
            const bool due = ls_interval > 0 && gen >= 2u && ((gen - 1u) % (uint32_t)ls_interval) == 0u;
            if (!due || lim) return;
        }
        buf = a.flip ? (cur ^ 1) : cur;
        f = buf ? f1 : f0;
        gen_new = a.flip ? gen + 1 : gen;
    } else {
        P = a.P;
        mx = a.maximize;
        m = 1;
        f = a.fit + (size_t)pop * P;
        sorted = a.sorted + (size_t)pop * P;
    }
    const int base = blockIdx.x * RK_CH;
    if (base >= P) return;
    const int e = t / RK_TPE, part = t % RK_TPE;
    const int i = base + e;
    // a batch of this thread's global loads is issued before the first use (one round trip)
    constexpr int RK_BATCH = 8;
    float v[RK_BATCH];
    auto load = [&](int i0) {
#pragma unroll
        for (int u = 0; u < RK_BATCH; ++u) {
            const int j = i0 + u * RK_THREADS;
            v[u] = (j < P) ? __ldg(f + (size_t)j * m) : 0.0f;
        }
    };
    auto store = [&](int i0) {
#pragma unroll
        for (int u = 0; u < RK_BATCH; ++u) {
            const int j = i0 + u * RK_THREADS;
            if (j < P) rk_keys[j] = ((unsigned long long)fitkey(v[u], mx) << 32) | (uint32_t)j;
        }
    };
    load(t);
    if (d && part == 1 && d->parents && i >= d->E && i < P - d->M) {
        // parent ranks of child row i of generation gen_new + 1 (core/solver.hpp:1117-1118);
        // they do not depend on the fitness, so they are drawn while its loads are in flight
        const uint4 pr = draw4(d->seed, 0u, (uint32_t)i, gen_new + 1, (d->island << 8) | TAG_PARENT);
        d->parents[i] = make_int2((int)pick(pr.x, (uint32_t)d->E), d->E + (int)pick(pr.y, (uint32_t)(P - d->E)));
    }
    store(t);
    for (int i0 = t + RK_THREADS * RK_BATCH; i0 < P; i0 += RK_THREADS * RK_BATCH) {
        load(i0);
        store(i0);
    }
    __syncthreads();
    const unsigned long long me = (i < P) ? rk_keys[i] : 0ull;
    // part p counts j = p, p + TPE, ...: the TPE parts of a warp read consecutive keys
    int cnt = 0;
#pragma unroll 8
    for (int j = part; j < P; j += RK_TPE) cnt += (rk_keys[j] < me) ? 1 : 0;
#pragma unroll
    for (int o = RK_TPE / 2; o >= 1; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o, RK_TPE);
    if (part == 0 && i < P) {
        sorted[cnt] = i;
        if (cnt == 0 && d && d->history && (int)gen_new < d->hist_cap) d->history[gen_new] = f[(size_t)i * m];
    }
    if (d) {
        if (a.flip) {
            __syncthreads();
            if (t == 0) {
                __threadfence();
                const int nblocks = (P + RK_CH - 1) / RK_CH;
                if (atomicAdd(d->done, 1) == nblocks - 1) {
                    d->cur = buf;
                    d->gen = gen_new;
                    *d->done = 0;
                    __threadfence();
                }
            }
        }
    }
}

// ring migration (core/solver.hpp:517-558), migrating the true best rows: island i's
// top `mig` rows by rank overwrite island (i+1)%k's worst `mig` rows; one CTA per instance
__global__ void migrate_kernel(PopDesc* descs, int k, int mig) {
    const int inst = blockIdx.x;
    for (int i = 0; i < k; ++i) {
        const PopDesc& a = descs[inst * k + i];
        const PopDesc& b = descs[inst * k + (i + 1) % k];
        const int ld = a.ld, m = a.m;
        for (int q = 0; q < mig; ++q) {
            const int sr = a.sorted[q];
            const int dr = b.sorted[b.P - mig + q];
            const float4* src = reinterpret_cast<const float4*>(a.keys[a.cur] + (size_t)sr * ld);
            float4* dst = reinterpret_cast<float4*>(b.keys[b.cur] + (size_t)dr * ld);
            for (int j = threadIdx.x; j < ld / 4; j += blockDim.x) dst[j] = src[j];
            if (threadIdx.x < m) b.fit[b.cur][(size_t)dr * m + threadIdx.x] = a.fit[a.cur][(size_t)sr * m + threadIdx.x];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
int device_sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// Two CTAs an SM, although one runs at a time: the other starts as soon as any SM is free, while a
// CTA an SM, striding over the rows, gave 985 .. 990 us instead of 978 .. 982 (n = 65 536, P = 512)
// and 122 instead of 119 (n = 20 000, P = 150).  The price is scratch for both.
int row_global_grid(int rows, int max_n) {
    const size_t budget = (size_t)2 << 30;  // scratch for at most 2 GiB of CTAs
    int g = 2 * device_sm_count();
    const size_t by_mem = budget / row_global_stride(max_n);
    if ((size_t)g > by_mem) g = (int)by_mem;
    if (g > rows) g = rows;
    return g < 1 ? 1 : g;
}

// the dynamic shared-memory limit of a kernel is only ever raised, so a later launch
// that needs less never takes it away from a live engine that needs more
static std::mutex g_attr_mu;
static std::map<std::pair<int, const void*>, size_t> g_attr;

cudaError_t raise_smem_limit(const void* fn, size_t smem) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_attr_mu);
    size_t& cur = g_attr[{dev, fn}];
    if (smem <= cur) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) cur = smem;
    return e;
}

// rows beyond shared memory
cudaError_t launch_rows_global(const RowLaunch& L, int kind, int grid, cudaStream_t s) {
    if (!L.gscratch || L.gstride < row_global_stride(L.max_n)) return cudaErrorInvalidValue;
    if (kind == MOVRP) return cudaErrorInvalidValue;  // MO-VRP rows fit in shared memory only
    if (L.ntasks <= 0 || grid <= 0) return cudaSuccess;
    if (grid > L.ntasks) grid = L.ntasks;
    const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(row_kernel_big), big_smem_bytes());
    if (e != cudaSuccess) return e;
    // (n = 1000, P = 2048, a generation with the caller's fitness: 56 us with a sort's block and
    // shared memory)
    const bool built_only = kind == EXTERNAL;
    const int block = built_only ? std::min(kBigBlock, round_up((L.max_n + 3) / 4, 32)) : kBigBlock;
    row_kernel_big<<<grid, block, built_only ? 0 : big_smem_bytes(), s>>>(L);
    return cudaGetLastError();
}

cudaError_t prepare_sort(int maxP) {
    return raise_smem_limit(reinterpret_cast<const void*>(rank_kernel), (size_t)(maxP > 0 ? maxP : 1) * 8);
}

cudaError_t launch_sort_raw(const float* fit, int P, int segments, int maximize, int32_t* sorted,
                            cudaStream_t s) {
    if (P <= 0 || segments <= 0) return cudaSuccess;
    RankArgs a{nullptr, fit, sorted, P, maximize, 0, 0};
    dim3 grid((P + RK_CH - 1) / RK_CH, segments);
    return launch_dep(rank_kernel, grid, dim3(RK_THREADS), (size_t)P * 8, s, a);
}

cudaError_t launch_sort_pops(PopDesc* descs, int npops, int maxP, int flip, cudaStream_t s) {
    if (npops <= 0) return cudaSuccess;
    RankArgs a{descs, nullptr, nullptr, 0, 0, flip, 0};
    dim3 grid((maxP + RK_CH - 1) / RK_CH, npops);
    return launch_dep(rank_kernel, grid, dim3(RK_THREADS), (size_t)maxP * 8, s, a);
}

cudaError_t launch_sort_pops_after_ls(PopDesc* descs, int npops, int maxP, cudaStream_t s) {
    if (npops <= 0) return cudaSuccess;
    RankArgs a{descs, nullptr, nullptr, 0, 0, 0, 1};
    dim3 grid((maxP + RK_CH - 1) / RK_CH, npops);
    return launch_dep(rank_kernel, grid, dim3(RK_THREADS), (size_t)maxP * 8, s, a);
}

cudaError_t launch_migrate(PopDesc* descs, int ninst, int k, int migrants, int max_n, cudaStream_t s) {
    (void)max_n;
    if (ninst <= 0 || k < 2 || migrants <= 0) return cudaSuccess;
    migrate_kernel<<<ninst, 256, 0, s>>>(descs, k, migrants);
    return cudaGetLastError();
}

}  // namespace bk
