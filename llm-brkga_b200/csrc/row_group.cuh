// row_group.cuh -- the work of one chromosome row by a group of T threads (one warp, part of
// a CTA, or a whole CTA): the stable argsort of its keys in shared memory and the fitness of
// every problem kind.  Rows of one CTA run independently: a group waits only for itself.
#pragma once

#include <climits>

#include "kernels.h"

namespace bk {

// ---------------------------------------------------------------------------------------
// the group and its slice of shared memory
// ---------------------------------------------------------------------------------------
template <int T>
struct RowGroup {
    int tid;  // thread of the group
    int rg;   // group of the CTA
    __device__ RowGroup() : tid(T < 1024 ? threadIdx.x % T : threadIdx.x), rg(T < 1024 ? threadIdx.x / T : 0) {}
    // barriers 1 .. 15 (0 is __syncthreads)
    __device__ __forceinline__ void sync() const {
        if constexpr (T == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(rg + 1), "n"(T) : "memory");
    }
};

struct RowBuf {
    uint32_t* cnt;       // bucket counters, then offsets: nb words
    uint16_t* perm;      // the decoded permutation, over the counters once they are dead
    uint16_t* si;        // scattered gene indices (8 entries of padding before, 16 after)
    int32_t* sk;         // scattered sort keys (the same padding); edges, terms and keys later
    float* kin;          // the row's keys in index order, where the launch keeps them
    unsigned char* red;  // reductions
    int nb;              // buckets
};

constexpr int kPadL = 8, kPadR = 16;  // window padding of sk and si

__host__ __device__ inline uint32_t row_align(uint32_t x) { return (x + 15u) & ~15u; }
// positions of the scattered arrays: TSPJ keeps a gap of 16 .. 19 between its two segments
__host__ __device__ inline int row_positions(int n) { return round_up(n, 4) + 20; }
// two 64-bit values a warp, and three more
__host__ __device__ inline uint32_t row_red_bytes(int block) { return block <= 128 ? 128 : block / 2 + 32; }
// buckets of a row: at least one per key, 4 x an odd number per thread: a thread's counters
// are consecutive for the scan, and an odd count of 16-byte words keeps the 128-bit loads of
// neighbouring threads in different banks
__host__ __device__ inline int row_buckets(int block, int n) { return 4 * block * (((n + 4 * block - 1) / (4 * block)) | 1); }
// one row's bytes: a counter per bucket, 6 bytes a key, 4 more where the keys are kept
__host__ __device__ inline uint32_t row_slice_bytes(int block, int max_n, bool keep) {
    const uint32_t np = row_positions(max_n) + kPadL + kPadR;
    return 4u * row_buckets(block, max_n) + row_align(2 * np) + row_align(4 * np) +
           (keep ? row_align(4u * round_up(max_n, 4)) : 0u) + row_red_bytes(block);
}

__device__ __forceinline__ RowBuf row_carve(unsigned char* p, int block, int max_n, bool keep) {
    const uint32_t np = row_positions(max_n) + kPadL + kPadR;
    RowBuf s;
    s.cnt = reinterpret_cast<uint32_t*>(p);
    s.perm = reinterpret_cast<uint16_t*>(p);
    s.nb = row_buckets(block, max_n);
    p += 4u * s.nb;
    s.si = reinterpret_cast<uint16_t*>(p) + kPadL;
    p += row_align(2 * np);
    s.sk = reinterpret_cast<int32_t*>(p) + kPadL;
    p += row_align(4 * np);
    s.kin = reinterpret_cast<float*>(p);
    if (keep) p += row_align(4u * round_up(max_n, 4));
    s.red = p;
    return s;
}

// the scratch behind the permutation: the rest of the counters, si and sk (at least 8 n + 64 bytes)
__device__ __forceinline__ unsigned char* row_scratch(const RowBuf& s, int n) {
    return reinterpret_cast<unsigned char*>(s.perm) + row_align(2u * round_up(n, 4));
}

// ---------------------------------------------------------------------------------------
// stable argsort
// ---------------------------------------------------------------------------------------
// order of the signed integers = order of the keys: -0 = +0, NaN (made canonical by the
// addition: 0x7FFFFFFF) last
__device__ __forceinline__ int32_t sort_key(float f) {
    const int32_t b = __float_as_int(__fadd_rn(f, 0.0f));
    return b ^ ((b >> 31) & 0x7FFFFFFF);
}

// monotone bucket of a key: floor(key * nb) for keys in [0, 1); below -> 0, above and NaN -> nb - 1
__device__ __forceinline__ int key_bucket(float key, float nbf, int nb) {
    const float t = fminf(__fmul_rn(key, nbf), nbf - 1.0f);  // NaN takes the bound
    return max((int)t, 0);
}

// A bucket's keys are ranked against their neighbours, so equal keys, keys outside [0, 1)
// and NaNs (few buckets) cost the square of the bucket.  Up to kWindow + 1 keys a
// bucket take the window below (nearly every row of random keys in [0, 1)), up to kHeavyKeys a
// loop over each key's bucket, and rows beyond that an ascending bitonic network:
// O(n log^2 n) on any input, and the same (key, index) order.
constexpr int kWindow = 8, kHeavyKeys = 32;

// what orders equal keys: the index itself, or the gene an index stands for (indices past the
// last gene are padding)
__device__ __forceinline__ uint32_t gene_of(const uint2* gene, int genes, uint16_t x) {
    if (!gene) return x;
    return (int)x < genes ? gene[x].y : 0xFFFFFFFFu;
}

template <int T>
__device__ __noinline__ void sort_heavy_segment(int32_t* k, uint16_t* x, int n, int tid, int rg, const uint2* gene,
                                                int genes) {
    RowGroup<T> g;
    g.tid = tid;
    g.rg = rg;
    auto order = [&](int i, int j) {
        const int32_t a = k[i], b = k[j];
        const uint16_t u = x[i], v = x[j];
        if (b < a || (b == a && gene_of(gene, genes, v) < gene_of(gene, genes, u))) {
            k[i] = b, k[j] = a;
            x[i] = v, x[j] = u;
        }
    };
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    const int half = n2 >> 1;
    for (int m = 2; m <= n2; m <<= 1) {
        const int hm = m >> 1;
        for (int p = tid; p < half; p += T) {
            const int base = (p / hm) * m, o = p % hm;
            if (base + m - 1 - o < n) order(base + o, base + m - 1 - o);
        }
        g.sync();
        for (int st = m >> 2; st > 0; st >>= 1) {
            for (int p = tid; p < half; p += T) {
                const int i = ((p & ~(st - 1)) << 1) | (p & (st - 1));
                if (i + st < n) order(i, i + st);
            }
            g.sync();
        }
    }
}

// Ranks by a loop over each key's own bucket: rows with a bucket of kWindow + 2 .. kHeavyKeys
// keys.  Populations that have converged are full of them (keys that were selected lie close
// together), so a row must not pay for its largest bucket at every key: over as many
// neighbours as that bucket holds, a generation of a converged population (n = 1000, P = 2048)
// took 48.8 us, now 27.5 (rows that fit the window: 17.7).  cnt holds the buckets' ends and is
// overwritten by the permutation, so the ranks wait in local memory.
template <int T, bool SPLIT, typename BucketF>
__device__ __noinline__ void rank_buckets(const int32_t* sk, const uint16_t* si, const uint32_t* cnt, uint16_t* perm, int n,
                                          int split, int shift, int nb, BucketF bucket, int tid, int rg,
                                          const uint2* gene, int genes) {
    RowGroup<T> g;
    g.tid = tid;
    g.rg = rg;
    const int nbs = SPLIT ? nb / 2 : nb;
    uint16_t rank[4 * kMaxTileGroups];  // tile_covers: n <= T * 4 * kMaxTileGroups
#pragma unroll 1
    for (int q = tid, j = 0; q < n; q += T, ++j) {
        const bool second = SPLIT && q >= split;
        const int sh = second ? shift : 0;
        const int32_t a = sk[q + sh];
        const uint32_t me = gene_of(gene, genes, si[q + sh]);
        const float v = __int_as_float(a ^ ((a >> 31) & 0x7FFFFFFF));
        const int b = bucket(v, nbs) + (second ? nbs : 0);
        const int hi = (int)cnt[b], lo = b > 0 ? (int)cnt[b - 1] : 0;
        int r = lo;
        for (int k = lo; k < hi; ++k) {
            const int32_t x = sk[k + sh];
            r += (x < a || (x == a && gene_of(gene, genes, si[k + sh]) < me)) ? 1 : 0;
        }
        rank[j] = (uint16_t)r;
    }
    g.sync();
#pragma unroll 1
    for (int q = tid, j = 0; q < n; q += T, ++j) perm[rank[j]] = si[q + (SPLIT && q >= split ? shift : 0)];
}

// equal keys in a thread's window: the window took them in position order; by index instead
static __device__ __noinline__ int tie_fix(const int32_t* sk, const uint16_t* si, int p, const uint2* gene, int genes) {
    const int32_t a = sk[p];
    const uint32_t me = gene_of(gene, genes, si[p]);
    int r = 0;
    for (int d = 1; d <= kWindow; ++d) {
        if (sk[p - d] == a && gene_of(gene, genes, si[p - d]) > me) --r;
        if (sk[p + d] == a && gene_of(gene, genes, si[p + d]) < me) ++r;
    }
    return r;
}

// Stable argsort of the row's n keys (n a multiple of 4: the caller pads with NaN, which
// sorts last) into s.perm, in two parts: count_keys for each four keys as they are built,
// then sort_row.  With SPLIT, keys [split, n) form a second segment sorted on its own
// (TSPJ's job keys): it takes the upper half of the buckets.  The counters must be zero at
// the start; the permutation replaces them (zero_counters before the next row).
//
// 1. histogram (shared atomics), scan, scatter of (key, index) into bucket order;
// 2. rank: every key is within its bucket's size of its place, so position p's rank is p
//    plus the smaller keys among the next w positions minus the larger among the last w,
//    w = the largest bucket - 1 (one value for the row).  A thread takes four consecutive
//    positions: 128-bit loads free of bank conflicts, compares in registers, no divergence
//    and no second look at the bucket bounds.  Ranking each key over its own bucket from
//    its index order instead cost a divergent loop of conflicting 64-bit loads (85 of the
//    kernel's 300 instructions a key, and 45 % of its shared-memory wavefronts conflicts).
template <bool SPLIT, typename BucketF>
__device__ __forceinline__ int bucket_at(float v, int i, int split, int nb, BucketF bucket) {
    const int nbs = SPLIT ? nb / 2 : nb;
    int b = bucket(v, nbs);
    if (SPLIT && i >= split) b += nbs;
    return b;
}

template <bool SPLIT, typename BucketF>
__device__ __forceinline__ void count_keys(const float4& k, int q, int split, const RowBuf& s, BucketF bucket) {
    atomicAdd(&s.cnt[bucket_at<SPLIT>(k.x, 4 * q, split, s.nb, bucket)], 1u);
    atomicAdd(&s.cnt[bucket_at<SPLIT>(k.y, 4 * q + 1, split, s.nb, bucket)], 1u);
    atomicAdd(&s.cnt[bucket_at<SPLIT>(k.z, 4 * q + 2, split, s.nb, bucket)], 1u);
    atomicAdd(&s.cnt[bucket_at<SPLIT>(k.w, 4 * q + 3, split, s.nb, bucket)], 1u);
}

// keys(q) returns keys 4 q .. 4 q + 3 as count_keys saw them; gene: what the indices stand for,
// where equal keys go by that instead of the index
template <int T, bool SPLIT, typename BucketF, typename KeysF>
__device__ __forceinline__ void sort_row(int n, int split, const RowBuf& s, const RowGroup<T>& g, BucketF bucket,
                                         KeysF keys, const uint2* gene = nullptr, int genes = 0) {
    constexpr int NW = T / 32;
    const int t = g.tid, lane = t & 31, warp = t >> 5;
    g.sync();
    // exclusive scan of the counters, a thread holding G = nb / 4 T consecutive 128-bit words
    uint32_t big = 0;
    {
        const int G = s.nb / (4 * T);
        uint4* c4 = reinterpret_cast<uint4*>(s.cnt) + t * G;
        uint32_t sum = 0;
#pragma unroll 2
        for (int j = 0; j < G; ++j) {
            const uint4 c = c4[j];
            sum += c.x + c.y + c.z + c.w;
            big = max(big, max(max(c.x, c.y), max(c.z, c.w)));
        }
        big = __reduce_max_sync(0xffffffffu, big);
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        uint32_t run = x - sum;
        if constexpr (NW > 1) {
            uint32_t* wt = reinterpret_cast<uint32_t*>(s.red);
            if (lane == 31) {
                wt[warp] = x;
                wt[NW + warp] = big;
            }
            g.sync();
            // every warp adds up the totals before its own
            const uint32_t v = (lane < NW) ? wt[lane] : 0u;
            run += __reduce_add_sync(0xffffffffu, (lane < warp) ? v : 0u);
            big = __reduce_max_sync(0xffffffffu, (lane < NW) ? wt[NW + lane] : 0u);
        }
#pragma unroll 2
        for (int j = 0; j < G; ++j) {
            const uint4 c = c4[j];
            uint4 o;
            o.x = run;
            o.y = o.x + c.x;
            o.z = o.y + c.y;
            o.w = o.z + c.z;
            run = o.w + c.w;
            c4[j] = o;
        }
    }
    g.sync();
    const int gap0 = SPLIT ? split : n;                          // first position after segment 0
    const int seg1 = SPLIT ? round_up(split + 16, 4) : 0;        // first position of segment 1
    const int shift = SPLIT ? seg1 - split : 0;
    const int npos = n + shift;
    auto put = [&](float v, int i) {
        int p = (int)atomicAdd(&s.cnt[bucket_at<SPLIT>(v, i, split, s.nb, bucket)], 1u);
        if (SPLIT && i >= split) p += shift;
        s.sk[p] = sort_key(v);
        s.si[p] = (uint16_t)i;
    };
#pragma unroll 2
    for (int q = t; 4 * q < n; q += T) {
        const float4 k = keys(q);
        put(k.x, 4 * q);
        put(k.y, 4 * q + 1);
        put(k.z, 4 * q + 2);
        put(k.w, 4 * q + 3);
    }
    // what the windows at both ends (and beside the gap) read: below and above every key
    if (T >= 16 && t < kPadR - 4) {
        s.sk[npos + t] = INT_MAX;
        s.si[npos + t] = 0xFFFFu;
        if (t < kPadL) s.sk[t - kPadL] = INT_MIN;
    }
    if (SPLIT && t < shift) {
        s.sk[gap0 + t] = (t < kWindow) ? INT_MAX : INT_MIN;
        s.si[gap0 + t] = 0xFFFFu;
    }
    g.sync();
    const int w = (int)big - 1;
    if (w > kWindow) {
        if (big > (uint32_t)kHeavyKeys) {
            sort_heavy_segment<T>(s.sk, s.si, gap0, t, g.rg, gene, genes);
            if (SPLIT) sort_heavy_segment<T>(s.sk + seg1, s.si + seg1, n - split, t, g.rg, gene, genes);
            for (int p = t; p < n; p += T) s.perm[p] = s.si[p < gap0 ? p : p + shift];
        } else {
            rank_buckets<T, SPLIT>(s.sk, s.si, s.cnt, s.perm, n, split, shift, s.nb, bucket, t, g.rg, gene, genes);
        }
        g.sync();
        return;
    }
    const int4* k4 = reinterpret_cast<const int4*>(s.sk);
#pragma unroll 1
    for (int c = t; 4 * c < npos; c += T) {
        int a[20];
        auto get = [&](int at, int4 y) { a[at] = y.x, a[at + 1] = y.y, a[at + 2] = y.z, a[at + 3] = y.w; };
        get(4, k4[c - 1]);
        get(8, k4[c]);
        get(12, k4[c + 1]);
        const uint2 x2 = *reinterpret_cast<const uint2*>(s.si + 4 * c);
        int r[4] = {4 * c, 4 * c + 1, 4 * c + 2, 4 * c + 3};
        bool tie = false;
        auto step = [&](int d) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int me = a[8 + i], rt = a[8 + i + d], lf = a[8 + i - d];
                if (me > rt) ++r[i];
                if (lf > me) --r[i];
                tie = tie | (me == rt) | (lf == me);
            }
        };
        step(1);
        step(2);
        step(3);
        if (w > 3) {
            step(4);
            if (w > 4) {
                get(0, k4[c - 2]);
                get(16, k4[c + 2]);
                step(5);
                if (w > 5) {
                    step(6);
                    if (w > 6) {
                        step(7);
                        step(8);
                    }
                }
            }
        }
        if (tie) {
#pragma unroll
            for (int i = 0; i < 4; ++i) r[i] += tie_fix(s.sk, s.si, 4 * c + i, gene, genes);
        }
        const uint32_t x[4] = {x2.x & 0xFFFFu, x2.x >> 16, x2.y & 0xFFFFu, x2.y >> 16};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!SPLIT) {
                s.perm[r[i]] = (uint16_t)x[i];
            } else {
                const int p = 4 * c + i;
                if (p < gap0) s.perm[r[i]] = (uint16_t)x[i];
                else if (p >= seg1 && p < npos) s.perm[r[i] - shift] = (uint16_t)x[i];
            }
        }
    }
    g.sync();
}

template <int T>
__device__ __forceinline__ void zero_counters(const RowBuf& s, int tid) {
    uint4* c = reinterpret_cast<uint4*>(s.cnt);
#pragma unroll 2
    for (int j = tid; 4 * j < s.nb; j += T) c[j] = make_uint4(0u, 0u, 0u, 0u);
}

// ---------------------------------------------------------------------------------------
// fitness
// ---------------------------------------------------------------------------------------
// Euclidean edge exactly as the reference builds its matrix (configs/tsp_config.hpp:366-368):
// float dx, dy; sqrt(dx*dx + dy*dy), no contraction, correctly rounded sqrt
__device__ __forceinline__ float edge_pts(float2 pa, float2 pb) {
    const float dx = __fsub_rn(pa.x, pb.x);
    const float dy = __fsub_rn(pa.y, pb.y);
    return __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
}

// canonical FP32 sum of m edge terms held in shared memory: 256 virtual lanes (term e in
// lane e % 256, in order), xor butterflies inside each group of 32 lanes, a fixed tree over
// the eight group totals.  A thread holds the lanes t, t + T, ... of LPT groups, and its
// warp folds their butterflies into one: after the step over lane bit 16 a thread keeps half
// of the groups, after bit 8 a quarter, and so on (addition commutes, so every sum is the one
// the plain butterflies give): 12 shuffles instead of 40 for a row of one warp.
template <int T>
__device__ __forceinline__ float canon_terms(const float* ed, int m, const RowBuf& s, const RowGroup<T>& g) {
    constexpr int LPT = T >= 256 ? 1 : 256 / T;
    const int t = g.tid, lane = t & 31;
    float acc[LPT];
#pragma unroll
    for (int j = 0; j < LPT; ++j) acc[j] = 0.0f;
    if (T <= 256 || t < 256)
        for (int e0 = t; e0 < m; e0 += 256)
#pragma unroll
            for (int j = 0; j < LPT; ++j)
                if (j == 0 || e0 + j * T < m) acc[j] = __fadd_rn(acc[j], ed[e0 + j * T]);
    int mine = 0;  // the group of acc[0] among the thread's LPT
#pragma unroll
    for (int h = LPT / 2, bit = 16; bit >= 1; h /= 2, bit /= 2) {
        if (h >= 1) {
            const bool up = (lane & bit) != 0;
            if (up) mine += h;
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float keep = up ? acc[j + h] : acc[j], send = up ? acc[j] : acc[j + h];
                acc[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, bit));
            }
        } else {
            acc[0] = __fadd_rn(acc[0], __shfl_xor_sync(0xffffffffu, acc[0], bit));
        }
    }
    if constexpr (T == 32) {
        // the tree over the groups, which the lanes hold in order 0 4 2 6 1 5 3 7 of bits 4, 8, 16
        float x = acc[0];
        x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, 4));
        x = __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, 8));
        return __fadd_rn(x, __shfl_xor_sync(0xffffffffu, x, 16));
    } else {
        float* red = reinterpret_cast<float*>(s.red);
        if ((lane & (32 / LPT - 1)) == 0 && (T <= 256 || t < 256)) red[(t >> 5) + mine * (T / 32)] = acc[0];
        g.sync();
        return __fadd_rn(__fadd_rn(__fadd_rn(red[0], red[1]), __fadd_rn(red[2], red[3])),
                         __fadd_rn(__fadd_rn(red[4], red[5]), __fadd_rn(red[6], red[7])));
    }
}

// the edge terms of a tour over m stops in s.perm into ed, a thread taking four consecutive
// edges (five points for four edges).  CLOSED: edge e joins stops e and e + 1, the last one
// the first; else the tour starts and ends at node 0, stop j is city perm[j] + 1 and edge e
// joins stops e - 1 and e (m + 1 edges).
template <int T, bool CLOSED, typename EdgeF>
__device__ __forceinline__ void tour_edges(int m, float* ed, const uint16_t* perm, EdgeF edge, const RowGroup<T>& g) {
    const int edges = CLOSED ? m : m + 1;
#pragma unroll 1
    for (int c = g.tid; 4 * c < edges; c += T) {
        // stops 4 c - 1 .. 4 c + 4
        const uint2 x = *reinterpret_cast<const uint2*>(perm + 4 * c);
        int id[5];
        if (CLOSED) {
            id[0] = x.x & 0xFFFFu, id[1] = x.x >> 16, id[2] = x.y & 0xFFFFu, id[3] = x.y >> 16;
            if (4 * c + 4 < m) {
                id[4] = perm[4 * c + 4];
            } else {
                const int first = perm[0];
#pragma unroll
                for (int i = 1; i < 5; ++i)
                    if (4 * c + i >= m) id[i] = first;
            }
        } else {
            id[0] = (c == 0) ? 0 : perm[4 * c - 1] + 1;
            id[1] = (x.x & 0xFFFFu) + 1, id[2] = (x.x >> 16) + 1, id[3] = (x.y & 0xFFFFu) + 1, id[4] = (x.y >> 16) + 1;
            if (4 * c + 4 > m) {
#pragma unroll
                for (int i = 1; i < 5; ++i)
                    if (4 * c + i > m) id[i] = 0;
            }
        }
        float4 d;
        edge(id, &d.x);
        reinterpret_cast<float4*>(ed)[c] = d;  // past the last edge: within the padding of the row's slice
    }
}

// sums of a group (T == 32: within the warp)
template <int T>
__device__ __forceinline__ long long group_sum_ll(long long v, const RowBuf& s, const RowGroup<T>& g) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if constexpr (T > 32) {
        long long* red = reinterpret_cast<long long*>(s.red);
        if ((g.tid & 31) == 0) red[g.tid >> 5] = v;
        g.sync();
        v = 0;
#pragma unroll
        for (int i = 0; i < T / 32; ++i) v += red[i];
        g.sync();
    }
    return v;
}

// exclusive scan of two 64-bit values over the group, and their totals
template <int T>
__device__ __forceinline__ void group_scan_ll2(long long a, long long b, const RowBuf& s, const RowGroup<T>& g,
                                               long long* ea, long long* eb, long long* ta) {
    constexpr int NW = T / 32;
    const int lane = g.tid & 31, w = g.tid >> 5;
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
    long long bx = 0, by = 0, tx;
    if constexpr (NW == 1) {
        tx = __shfl_sync(0xffffffffu, x, 31);
    } else {
        long long* red = reinterpret_cast<long long*>(s.red);
        if (lane == 31) {
            red[w] = x;
            red[NW + w] = y;
        }
        g.sync();
        // every warp scans the warp totals for itself
        long long p = (lane < NW) ? red[lane] : 0ll, q = (lane < NW) ? red[NW + lane] : 0ll;
        const long long p0 = p, q0 = q;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long pu = __shfl_up_sync(0xffffffffu, p, o);
            const long long qu = __shfl_up_sync(0xffffffffu, q, o);
            if (lane >= o) {
                p += pu;
                q += qu;
            }
        }
        tx = __shfl_sync(0xffffffffu, p, 31);
        bx = __shfl_sync(0xffffffffu, p - p0, w);
        by = __shfl_sync(0xffffffffu, q - q0, w);
        g.sync();
    }
    *ea = bx + x - a;
    *eb = by + y - b;
    *ta = tx;
}

// knapsack greedy in key order: the longest prefix of the sorted items that fits, then a
// first-fit walk over the rest by one warp (weights >= 0).  The items' (weight, value)
// pairs come in key order into the scratch behind the permutation, one 8-byte load each.
template <int T>
__device__ __forceinline__ float knap_greedy(int n, const int2* __restrict__ items, long long C, const RowBuf& s,
                                             const RowGroup<T>& g) {
    const int t = g.tid;
    int2* wv = reinterpret_cast<int2*>(row_scratch(s, n));
    for (int p = t; p < n; p += T) wv[p] = __ldg(items + s.perm[p]);
    g.sync();
    // an odd number of items per thread: neighbouring threads start in different banks
    const int ch = ((n + T - 1) / T) | 1;
    const int p0 = min(n, t * ch), p1 = min(n, p0 + ch);
    long long ws = 0, vs = 0;
    for (int p = p0; p < p1; ++p) {
        const int2 x = wv[p];
        ws += x.x;
        vs += x.y;
    }
    long long S, V, totw;
    group_scan_ll2<T>(ws, vs, s, g, &S, &V, &totw);
    // the prefix weight only grows, so exactly one position breaks it (none when all fits):
    // the thread that holds it records the prefix's weight, length and value
    long long* misc = reinterpret_cast<long long*>(s.red) + 2 * (T / 32);
    if (t == T - 1 && totw <= C) {
        misc[0] = totw;
        misc[1] = n;
        misc[2] = V + vs;
    }
    if (S <= C && S + ws > C) {
        for (int p = p0; p < p1; ++p) {
            const int2 x = wv[p];
            if (S <= C && S + x.x > C) {
                misc[0] = S;
                misc[1] = p;
                misc[2] = V;
            }
            S += x.x;
            V += x.y;
        }
    }
    g.sync();
    const long long f = misc[1], v0 = misc[2];
    long long vt = 0;
    if (t < 32 && f < n) {
        // the spare capacity is below the weight of the item that broke the prefix: 32 bits
        int r = (int)(C - misc[0]);
        for (int b0 = (int)f + 1; b0 < n; b0 += 256) {
            int2 x[8];
            int mn = INT_MAX;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int pos = b0 + 32 * c + t;
                x[c] = (pos < n) ? wv[pos] : make_int2(INT_MAX, 0);
                mn = min(mn, x[c].x);
            }
            // one vote per 256 items: once little is spare most hold no item that fits
            if (!__any_sync(0xffffffffu, mn <= r)) continue;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
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
    return (float)(v0 + vt);  // thread 0's value is the row's
}

// TSPJ makespan (configs/tspj_config.hpp:555-585): the city tour from the depot (node 0)
// and back; at each position the arrival time plus the duration of the job type assigned
// there; the larger of the tour length and the latest completion.  perm[0, c) is the city
// order (cities perm + 1), perm[c, 2c) the job order (types perm - c + 1).  The legs and
// durations are gathered in parallel; the additions follow the reference's own order, so
// the value equals the reference's bit for bit.
template <int T>
__device__ __forceinline__ float tspj_makespan(int nc, const float* __restrict__ travel,
                                               const float* __restrict__ jobs, const RowBuf& s, const RowGroup<T>& g) {
    const size_t D = (size_t)nc + 1;
    float* le = reinterpret_cast<float*>(s.sk);
    float* jd = le + round_up(nc, 4);
    for (int i = g.tid; i < nc; i += T) {
        const int city = s.perm[i] + 1, prev = (i == 0) ? 0 : s.perm[i - 1] + 1, job = s.perm[nc + i] - nc + 1;
        le[i] = __ldg(travel + (size_t)prev * D + city);
        jd[i] = __ldg(jobs + (size_t)city * D + job);
    }
    const float back = __ldg(travel + (size_t)(s.perm[nc - 1] + 1) * D);
    g.sync();
    float run = 0.0f, mjc = 0.0f;
    if (g.tid < 32) {
        int i = 0;
        for (; i + 4 <= nc; i += 4) {
            const float4 e = *reinterpret_cast<const float4*>(le + i), j = *reinterpret_cast<const float4*>(jd + i);
            float jc;
            run = __fadd_rn(run, e.x), jc = __fadd_rn(run, j.x), mjc = (mjc < jc) ? jc : mjc;
            run = __fadd_rn(run, e.y), jc = __fadd_rn(run, j.y), mjc = (mjc < jc) ? jc : mjc;
            run = __fadd_rn(run, e.z), jc = __fadd_rn(run, j.z), mjc = (mjc < jc) ? jc : mjc;
            run = __fadd_rn(run, e.w), jc = __fadd_rn(run, j.w), mjc = (mjc < jc) ? jc : mjc;
        }
        for (; i < nc; ++i) {
            run = __fadd_rn(run, le[i]);
            const float jc = __fadd_rn(run, jd[i]);
            mjc = (mjc < jc) ? jc : mjc;
        }
    }
    const float tt = __fadd_rn(run, back);
    return (tt < mjc) ? mjc : tt;  // thread 0's value is the row's
}

// ContinuousOptGPUConfig (configs/continuous_opt_gpu_config.hpp:114-173): x = key * (upper -
// lower) + lower; sphere sum x^2; Rastrigin 10 n + sum (x^2 - 10 cos(2 pi x)); Rosenbrock
// sum 100 (x_{i+1} - x_i^2)^2 + (1 - x_i)^2.  The terms are computed in parallel (keys in
// s.sk, terms over the unused counters); the sum follows the reference's sequential order,
// four cycles a term: the chain reads four terms per 128-bit load and nothing but the
// addition depends on the last one.  Adding lane by lane with a shuffle per term took about
// 30 cycles (n = 1000, P = 2048: 52 us).
template <int T>
__device__ __forceinline__ float continuous_fitness(int n, int fn, float lo, float hi, const RowBuf& s,
                                                    const RowGroup<T>& g) {
    const float* keys = reinterpret_cast<const float*>(s.sk);
    float* term = reinterpret_cast<float*>(s.cnt);
    const float range = __fsub_rn(hi, lo), two_pi = __fmul_rn(2.0f, 3.14159265358979323846f);
    const int terms = (fn == FN_ROSENBROCK) ? n - 1 : n;
    for (int i = g.tid; i < terms; i += T) {
        const float x = __fadd_rn(__fmul_rn(keys[i], range), lo);
        if (fn == FN_SPHERE) {
            term[i] = __fmul_rn(x, x);
        } else if (fn == FN_RASTRIGIN) {
            term[i] = __fsub_rn(__fmul_rn(x, x), __fmul_rn(10.0f, cosf(__fmul_rn(two_pi, x))));
        } else {
            const float xn = __fadd_rn(__fmul_rn(keys[i + 1], range), lo);
            const float t1 = __fsub_rn(xn, __fmul_rn(x, x));
            const float t2 = __fsub_rn(1.0f, x);
            term[i] = __fadd_rn(__fmul_rn(__fmul_rn(100.0f, t1), t1), __fmul_rn(t2, t2));
        }
    }
    g.sync();
    float sum = (fn == FN_RASTRIGIN) ? __fmul_rn(10.0f, (float)n) : 0.0f;
    if (g.tid < 32) {
        int i = 0;
#pragma unroll 1
        for (; i + 16 <= terms; i += 16) {
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = *reinterpret_cast<const float4*>(term + i + 4 * u);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, q[u].x), q[u].y), q[u].z), q[u].w);
        }
        for (; i < terms; ++i) sum = __fadd_rn(sum, term[i]);
    }
    return sum;  // thread 0's value is the row's
}

// JobSchedulingGPUConfig (configs/job_scheduling_gpu_config.hpp:132-148): job i goes to
// machine (int)(key_i * machines), capped at machines - 1; each machine's load adds its jobs
// in index order; the makespan is the largest load.  The machines of all jobs are staged as
// integers over s.sk; a thread keeps up to NM machines and passes all jobs in order, four
// per 128-bit load (every lane of a warp reads the same four): a compare, a select and an
// addition per machine and job, so each load equals the reference's sequential sum bit for
// bit.  Handing the jobs round by two shuffles each took 60 us at n = 1000, 32 machines,
// P = 2048.
template <int T, int NM>
__device__ __forceinline__ float jobsched_pass(const int32_t* mid, int n, const float* jt, int M, int m0) {
    float load[NM];
#pragma unroll
    for (int u = 0; u < NM; ++u) load[u] = 0.0f;
    // a job of another machine adds zero: a load is never -0, so that changes nothing, and only
    // the addition itself is on the chain (branches took 56 cycles a job)
    int i = 0;
#pragma unroll 1
    for (; i + 16 <= n; i += 16) {
        int4 q[4];
        float4 v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            q[c] = *reinterpret_cast<const int4*>(mid + i + 4 * c);
            v[c] = *reinterpret_cast<const float4*>(jt + i + 4 * c);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                const int me = m0 + u * T;
                load[u] = __fadd_rn(load[u], q[c].x == me ? v[c].x : 0.0f);
                load[u] = __fadd_rn(load[u], q[c].y == me ? v[c].y : 0.0f);
                load[u] = __fadd_rn(load[u], q[c].z == me ? v[c].z : 0.0f);
                load[u] = __fadd_rn(load[u], q[c].w == me ? v[c].w : 0.0f);
            }
    }
    for (; i < n; ++i)
#pragma unroll
        for (int u = 0; u < NM; ++u)
            if (mid[i] == m0 + u * T) load[u] = __fadd_rn(load[u], jt[i]);
    float best = -INFINITY;
#pragma unroll
    for (int u = 0; u < NM; ++u)
        if (m0 + u * T < M) best = (best < load[u]) ? load[u] : best;
    return best;
}

template <int T>
__device__ __forceinline__ float jobsched_makespan(int n, const float* jt, int M, const RowBuf& s,
                                                   const RowGroup<T>& g) {
    float best = -INFINITY;
    for (int m0 = 0; m0 < M; m0 += 4 * T) {
        if (m0 + (g.tid & ~31) >= M) break;  // no machine for this warp
        const int left = M - m0;
        float b;
        if (left <= T) b = jobsched_pass<T, 1>(s.sk, n, jt, M, m0 + g.tid);
        else if (left <= 2 * T) b = jobsched_pass<T, 2>(s.sk, n, jt, M, m0 + g.tid);
        else b = jobsched_pass<T, 4>(s.sk, n, jt, M, m0 + g.tid);
        best = (best < b) ? b : best;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, best, o);
        best = (best < other) ? other : best;
    }
    if constexpr (T > 32) {
        float* red = reinterpret_cast<float*>(s.red);
        if ((g.tid & 31) == 0) red[g.tid >> 5] = best;
        g.sync();
        best = red[0];
        for (int w = 1; w < T / 32; ++w) best = (best < red[w]) ? red[w] : best;
    }
    return best;
}

// MO-VRP routes and objectives of the sorted customers perm[j] + 1
// (configs/multi_objective_vrp_config.hpp:233-313): customers in order; one that would take
// a non-empty route over capacity closes it.  The legs and the running demand come in
// parallel; a route's end is the first customer whose running demand passes the start's by
// more than the capacity (32 candidates per vote; the subtraction is exact modulo 2^32,
// since the demand up to the first that passes stays below 2^31); a lane then adds one
// route's legs in visiting order, and the routes' totals are added in route order: every
// float addition of the reference, in its order.  Walking customer by customer was one
// chain of n dependent decisions (about 50 cycles each).
template <int T>
__device__ __forceinline__ void movrp_objectives(int n, const float* xy, const int32_t* __restrict__ dem, int cap,
                                                 int vehicles, const RowBuf& s, const RowGroup<T>& g, float* out) {
    const float2* pt = reinterpret_cast<const float2*>(xy);
    const float2 depot = pt[0];
    float* leg = reinterpret_cast<float*>(row_scratch(s, n));  // leg into customer j from customer j - 1
    uint32_t* cum = reinterpret_cast<uint32_t*>(leg + round_up(n, 4));  // demand of customers [0, j)
    for (int j = g.tid; j < n; j += T) {
        const int cust = s.perm[j] + 1;
        leg[j] = (j == 0) ? 0.0f : edge_pts(pt[s.perm[j - 1] + 1], pt[cust]);
        cum[j + 1] = (uint32_t)__ldg(dem + cust);
    }
    g.sync();
    if (g.tid >= 32) return;
    const int lane = g.tid;
    uint32_t run = 0;
    if (lane == 0) cum[0] = 0u;
    for (int j0 = 0; j0 < n; j0 += 32) {
        uint32_t x = (j0 + lane < n) ? cum[j0 + lane + 1] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        x += run;
        if (j0 + lane < n) cum[j0 + lane + 1] = x;
        run = __shfl_sync(0xffffffffu, x, 31);
    }
    __syncwarp();
    float total = 0.0f, longest = 0.0f, pen = 0.0f;
    int routes = 0, start = 0;
    while (start < n) {
        // up to 32 routes, lane r holding route r's customers [a, b)
        int a = 0, b = 0, got = 0;
        while (start < n && got < 32) {
            const uint32_t base = cum[start];
            int end = n;
            for (int j0 = start + 1; j0 < n; j0 += 32) {
                const int j = j0 + lane;
                const unsigned over = __ballot_sync(0xffffffffu, j < n && cum[min(j, n - 1) + 1] - base > (uint32_t)cap);
                if (over) {
                    end = j0 + __ffs(over) - 1;
                    break;
                }
            }
            if (lane == got) a = start, b = end;
            start = end;
            ++got;
        }
        float dist = 0.0f;
        int load = 0;
        if (lane < got) {
            const float first = edge_pts(pt[s.perm[a] + 1], depot), last = edge_pts(pt[s.perm[b - 1] + 1], depot);
            dist = first;
            for (int j = a + 1; j < b; ++j) dist = __fadd_rn(dist, leg[j]);
            dist = __fadd_rn(dist, last);
            load = (int)(cum[b] - cum[a]);
        }
        for (int r = 0; r < got; ++r) {
            const float d = __shfl_sync(0xffffffffu, dist, r);
            const int ld = __shfl_sync(0xffffffffu, load, r);
            total = __fadd_rn(total, d);
            longest = (d > longest) ? d : longest;
            if (ld > cap) pen = __fadd_rn(pen, __fmul_rn((float)(ld - cap), 100.0f));
        }
        routes += got;
    }
    out[0] = __fadd_rn(total, pen);
    out[1] = longest;
    if (routes > vehicles) {
        const float vp = __fmul_rn((float)(routes - vehicles), 500.0f);
        out[0] = __fadd_rn(out[0], vp);
        out[1] = __fadd_rn(out[1], vp);
    }
}

}  // namespace bk
