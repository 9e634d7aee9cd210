// nsga2.cu -- NSGA-II selection on the device.
//
// Reference: Solver::evolve_generation_nsga2 (core/solver.hpp:751-817) and
// Population::fast_non_dominated_sort / calculate_crowding_distance /
// select_next_generation_nsga2 / ensure_minimum_diversity (core/population.hpp:130-517).
//
// The reference pushes every first-front point into fronts[0] twice (once in
// fast_non_dominated_sort, core/population.hpp:431-434, again in
// build_fronts_from_domination, :335-340).  Its ranks therefore come from a peeling in
// which the first front decrements twice, its crowding pass sees every first-front point
// as two adjacent entries, and its survivor list takes first-front points twice.  All
// three are reproduced here (ties fixed by index), bit for bit against the oracle.
//
// Ranks: bit-packed dominator rows, peeled front by front on a thread-block cluster.
// Crowding: each point's place, neighbours and extremes in its front in both objective
// orders, by counting; each entry adds (next - prev) / range in list order.
// Survivors: the entries (first-front points twice) by (rank, last objective or -crowding
// for the front that is cut, index, copy); the first P of them.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "engine.h"
#include "nsga2.h"

namespace bk {

constexpr int kNsgaBlock = 1024;
constexpr int kMaxPool = 4096;  // largest pool (2P) of the in-shared-memory select kernel

__host__ __device__ inline int npow2(int x) {
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Ascending bitonic sort of s[0, N2) (N2 a power of two) by the whole block.  Strides of 64
// and more go through shared memory with a barrier each; strides 32 .. 1 run in registers:
// warp w owns the 64-element blocks w, w + warps, ..., lane l holding elements l and l + 32
// of a block (stride 32 inside the lane, strides 16 .. 1 by shuffles), so each k costs one
// barrier for all of its small strides instead of six.
__device__ __forceinline__ unsigned long long cx_keep(unsigned long long x, unsigned long long y, int g, int j,
                                                      int k) {
    // element g of the pair (g, g ^ j): the lower index keeps the minimum in an ascending
    // run ((g & k) == 0), the maximum in a descending one
    const bool keep_min = ((g & j) == 0) == ((g & k) == 0);
    return keep_min ? (x < y ? x : y) : (x < y ? y : x);
}

template <int BLOCK>
__device__ void bitonic_u64(unsigned long long* s, int N2) {
    const int t = threadIdx.x;
    if (N2 < 64) {
        for (int k = 2; k <= N2; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int p = t; p < (N2 >> 1); p += BLOCK) {
                    const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));
                    const int ixj = i + j;
                    const bool up = (i & k) == 0;
                    const unsigned long long a = s[i], b = s[ixj];
                    if ((a > b) == up) {
                        s[i] = b;
                        s[ixj] = a;
                    }
                }
                __syncthreads();
            }
        return;
    }
    constexpr int NW = BLOCK / 32;
    const int lane = t & 31, warp = t >> 5;
    // strides min(32, k / 2) .. 1 of step k on every 64-element block, in registers
    auto small_strides = [&](int k, int jmax) {
        for (int base = warp * 64; base < N2; base += NW * 64) {
            const int g0 = base + lane, g1 = g0 + 32;
            unsigned long long x0 = s[g0], x1 = s[g1];
            if (jmax >= 32) {
                const unsigned long long lo = x0 < x1 ? x0 : x1, hi = x0 < x1 ? x1 : x0;
                const bool up = (g0 & k) == 0;
                x0 = up ? lo : hi;
                x1 = up ? hi : lo;
            }
            for (int j = (jmax >= 32 ? 16 : jmax); j > 0; j >>= 1) {
                const unsigned long long y0 = __shfl_xor_sync(0xffffffffu, x0, j);
                const unsigned long long y1 = __shfl_xor_sync(0xffffffffu, x1, j);
                x0 = cx_keep(x0, y0, g0, j, k);
                x1 = cx_keep(x1, y1, g1, j, k);
            }
            s[g0] = x0;
            s[g1] = x1;
        }
        __syncthreads();
    };
    for (int k = 2; k <= 64; k <<= 1) small_strides(k, k >> 1);
    for (int k = 128; k <= N2; k <<= 1) {
        for (int j = k >> 1; j >= 64; j >>= 1) {
            for (int p = t; p < (N2 >> 1); p += BLOCK) {
                const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));
                const int ixj = i + j;
                const bool up = (i & k) == 0;
                const unsigned long long a = s[i], b = s[ixj];
                if ((a > b) == up) {
                    s[i] = b;
                    s[ixj] = a;
                }
            }
            __syncthreads();
        }
        small_strides(k, 32);
    }
}

constexpr int kCB = 16;  // count planes (two's complement)
constexpr int kDB = 15;  // decrement planes

__device__ __forceinline__ bool dominates_m(const float* a, const float* b, int m) {
    bool better = false;
    for (int o = 0; o < m; ++o) {
        if (a[o] > b[o]) return false;
        if (a[o] < b[o]) better = true;
    }
    return better;
}

struct DomArgs {
    PopDesc* dd;          // engine mode: the P population blockIdx.y (objectives fit[cur], buffers);
                          // a generation's 2P pool goes through dom2_pool_kernel
    int only_rebuilt;     // engine mode: skip populations whose diversity pass kept them (*nu >= P)
    const float* obj;     // raw mode
    int rawN, m;
    uint32_t* S;          // raw mode: [N][Wmax]
    int32_t* cnt;         // raw mode: [N] dominator counts (null: not wanted)
    int Wmax;
    int dominators;       // rows hold the points that dominate i (the row peel), not those i dominates
};

__global__ void dom_build_kernel(DomArgs a) {
    const float* obj = a.obj;
    const int N = a.rawN, m = a.m, Wmax = a.Wmax;
    uint32_t* S = a.S;
    int32_t* cnt = a.cnt;
    const int W = (N + 31) / 32;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < N; i += nwarps) {
        float oi[4];
        for (int o = 0; o < m && o < 4; ++o) oi[o] = __ldg(obj + (size_t)i * m + o);
        int c = 0;
        for (int w = 0; w < W; ++w) {
            const int j = 32 * w + lane;
            bool dij = false, dji = false;
            if (j < N && j != i) {
                float oj[4];
                for (int o = 0; o < m && o < 4; ++o) oj[o] = __ldg(obj + (size_t)j * m + o);
                dij = dominates_m(oi, oj, m);
                dji = dominates_m(oj, oi, m);
            }
            const uint32_t si = __ballot_sync(0xffffffffu, dij);
            const uint32_t di = __ballot_sync(0xffffffffu, dji);
            if (lane == 0) S[(size_t)i * Wmax + w] = a.dominators ? di : si;
            c += __popc(di);
        }
        if (lane == 0 && cnt) cnt[i] = c;
    }
}

// Two objectives (every NSGA-II problem of the engine): the objectives are staged in
// shared memory and each warp tests four rows against 32 columns per step.  The four
// comparisons of a pair give both directions: i dominates j iff !(a0 > b0) && !(a1 > b1)
// && (a0 < b0 || a1 < b1), the reference's Individual::dominates (core/individual.hpp:99-114)
// with its NaN behaviour; padding columns are NaN, which dominates nothing either way.
// Element i of [0, count) for i = threadIdx.x + k * T: a thread issues the loads of K of
// its elements before the first store, so staging takes one memory round trip per K
// elements instead of one per element.
template <int T, int K, typename Ld, typename St>
__device__ __forceinline__ void staged(int count, Ld ld, St st) {
    for (int i0 = (int)threadIdx.x; i0 < count; i0 += T * K) {
        decltype(ld(0)) v[K];
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (i0 + u * T < count) v[u] = ld(i0 + u * T);
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (i0 + u * T < count) st(i0 + u * T, v[u]);
    }
}

// 32 x 32 bit transpose across a warp: lane l holds row l on entry (bit c = element (l, c))
// and column l on exit (bit r = element (r, l)); five exchange steps of halving blocks.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t w, int lane) {
    const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int s = 16 >> k;
        const uint32_t m = masks[k];
        const uint32_t y = __shfl_xor_sync(0xffffffffu, w, s);
        w = (lane & s) ? ((w & ~m) | ((y & ~m) >> s)) : ((w & m) | ((y & m) << s));
    }
    return w;
}

// The pool's dominator rows (row i, bit j: j dominates i), each unordered pair of 32-point
// blocks (I <= J) visited once by one warp: for row r of block I against lane j of block J
// the four compares give both directions.  Block I's rows at word J come from one
// direction's ballots directly; block J's rows at word I from the other's by a bit
// transpose.  The same compares as dom2_build_kernel, half the pair tests.
constexpr int kSymWarps = 16;

__global__ void __launch_bounds__(kSymWarps * 32) dom2_pool_kernel(PopDesc* dd) {
    dep_wait();
    __shared__ float2 srow[kSymWarps][32];
    PopDesc& d = dd[blockIdx.y];
    if (at_limit(d)) return;
    const int N = 2 * d.P, W = (N + 31) / 32, Wmax = d.domW;
    const int T = W * (W + 1) / 2;
    const float2* __restrict__ o2 = reinterpret_cast<const float2*>(d.fit[d.cur]);
    uint32_t* const S = d.domS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2* const rows = srow[warp];
    // consecutive tiles go to different CTAs, so that every CTA (and SM) gets the same
    // share; each warp loads the next tile's objectives before it works on the current one
    const int nw = gridDim.x * kSymWarps;
    auto block_pair = [](int tile, int& I, int& J) {  // tile = J (J + 1) / 2 + I with I <= J
        J = (int)((sqrtf(8.0f * (float)tile + 1.0f) - 1.0f) * 0.5f);
        while (J * (J + 1) / 2 > tile) --J;
        while ((J + 1) * (J + 2) / 2 <= tile) ++J;
        I = tile - J * (J + 1) / 2;
    };
    auto objectives = [&](int I, int J, float2& oi, float2& oj) {
        const int i = 32 * I + lane, j = 32 * J + lane;
        oi = (i < N) ? __ldg(o2 + i) : make_float2(NAN, NAN);
        oj = (j < N) ? __ldg(o2 + j) : make_float2(NAN, NAN);
    };
    int tile = warp * gridDim.x + blockIdx.x, I = 0, J = 0;
    float2 oi = make_float2(NAN, NAN), oj = make_float2(NAN, NAN);
    if (tile < T) {
        block_pair(tile, I, J);
        objectives(I, J, oi, oj);
    }
    for (; tile < T; tile += nw) {
        int nI = 0, nJ = 0;
        float2 noi = make_float2(NAN, NAN), noj = make_float2(NAN, NAN);
        if (tile + nw < T) {
            block_pair(tile + nw, nI, nJ);
            objectives(nI, nJ, noi, noj);
        }
        const int i = 32 * I + lane, j = 32 * J + lane;
        __syncwarp();
        rows[lane] = oi;
        __syncwarp();
        uint32_t rw = 0u, cw = 0u;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
            const float2 a = rows[r];
            const bool gt0 = a.x > oj.x, gt1 = a.y > oj.y;
            const bool lt0 = a.x < oj.x, lt1 = a.y < oj.y;
            const uint32_t s1 = __ballot_sync(0xffffffffu, !gt0 && !gt1 && (lt0 || lt1));  // row r dominates lane
            const uint32_t s2 = __ballot_sync(0xffffffffu, !lt0 && !lt1 && (gt0 || gt1));  // lane dominates row r
            if (lane == r) {
                rw = s1;
                cw = s2;
            }
        }
        if (i < N) S[(size_t)i * Wmax + J] = cw;
        if (I != J) {
            const uint32_t tw = warp_transpose32(rw, lane);  // row j, word I
            if (j < N) S[(size_t)j * Wmax + I] = tw;
        }
        I = nI;
        J = nJ;
        oi = noi;
        oj = noj;
    }
}

constexpr int kDom2Rows = 4;       // rows per warp
constexpr int kDom2RowWarps = 4;   // row groups per CTA
constexpr int kDom2ColGroups = 4;  // column groups: warp g of a row group takes the 32-word blocks b % 4 == g
constexpr int kDom2Warps = kDom2RowWarps * kDom2ColGroups;

__global__ void __launch_bounds__(kDom2Warps * 32) dom2_build_kernel(DomArgs a) {
    dep_wait();
    extern __shared__ float2 so[];  // [32 * ceil(N / 32)] objectives
    __shared__ int cpart[kDom2ColGroups][kDom2RowWarps * kDom2Rows];
    const float* obj;
    int N, Wmax;
    uint32_t* S;
    int32_t* cnt;
    if (a.dd) {
        const PopDesc& d = a.dd[blockIdx.y];
        if (a.only_rebuilt && (!d.advanced || __ldg(d.nu) >= d.P)) return;
        N = d.P;
        obj = d.fit[d.cur];
        S = d.domS;
        cnt = nullptr;
        Wmax = d.domW;
    } else {
        N = a.rawN;
        obj = a.obj;
        S = a.S;
        cnt = a.cnt;
        Wmax = a.Wmax;
    }
    constexpr int RPC = kDom2Rows * kDom2RowWarps;  // rows per CTA
    const int row0 = blockIdx.x * RPC;
    if (row0 >= N) return;
    const int W = (N + 31) / 32;
    const float2* o2 = reinterpret_cast<const float2*>(obj);
    staged<kDom2Warps * 32, 8>(
        32 * W, [&](int j) { return (j < N) ? __ldg(o2 + j) : make_float2(NAN, NAN); },
        [&](int j, float2 v) { so[j] = v; });
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rg = warp % kDom2RowWarps, cg = warp / kDom2RowWarps;
    const int i0 = row0 + rg * kDom2Rows;
    float2 oi[kDom2Rows];
    int c[kDom2Rows];
#pragma unroll
    for (int r = 0; r < kDom2Rows; ++r) {
        oi[r] = so[min(i0 + r, N - 1)];
        c[r] = 0;
    }
    const int nblk = (W + 31) / 32;
    for (int b = cg; b < nblk; b += kDom2ColGroups) {
        uint32_t buf[kDom2Rows];
#pragma unroll
        for (int r = 0; r < kDom2Rows; ++r) buf[r] = 0u;
        const int wend = min(W, 32 * b + 32);
        for (int w = 32 * b; w < wend; ++w) {
            const float2 oj = so[32 * w + lane];
#pragma unroll
            for (int r = 0; r < kDom2Rows; ++r) {
                const bool gt0 = oi[r].x > oj.x, gt1 = oi[r].y > oj.y;
                const bool lt0 = oi[r].x < oj.x, lt1 = oi[r].y < oj.y;
                const uint32_t si = __ballot_sync(0xffffffffu, !gt0 && !gt1 && (lt0 || lt1));
                const uint32_t di = __ballot_sync(0xffffffffu, !lt0 && !lt1 && (gt0 || gt1));
                c[r] += __popc(di);
                if (lane == (w & 31)) buf[r] = a.dominators ? di : si;
            }
        }
        // lane l holds word 32 b + l of each row: one coalesced store per row
        const int wl = 32 * b + lane;
#pragma unroll
        for (int r = 0; r < kDom2Rows; ++r)
            if (i0 + r < N && wl < wend) S[(size_t)(i0 + r) * Wmax + wl] = buf[r];
    }
    // dominator counts: the column groups' partial counts, added in a fixed order
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < kDom2Rows; ++r) cpart[cg][rg * kDom2Rows + r] = c[r];
    }
    __syncthreads();
    if (cnt && threadIdx.x < RPC && row0 + (int)threadIdx.x < N) {
        int sum = 0;
#pragma unroll
        for (int g = 0; g < kDom2ColGroups; ++g) sum += cpart[g][threadIdx.x];
        cnt[row0 + threadIdx.x] = sum;
    }
}

struct PeelSmem {
    uint32_t* C;      // [kCB][W] count planes
    uint32_t* A;      // [W] ranked
    uint32_t* F;      // [W] current front
    uint32_t* V;      // [W] valid points
    uint16_t* list;   // [N] front members
};

__host__ __device__ inline size_t peel_smem_bytes(int N) {
    const int W = (N + 31) / 32;
    return (size_t)(kCB + 4) * W * 4 + (((size_t)N * 2 + 15) / 16) * 16;
}

__device__ inline PeelSmem peel_carve(unsigned char* base, int N) {
    const int W = (N + 31) / 32;
    PeelSmem p;
    p.C = (uint32_t*)base;
    p.A = p.C + (size_t)kCB * W;
    p.F = p.A + W;
    p.V = p.F + W;
    p.list = (uint16_t*)(p.V + 2 * W);  // V[W..2W) stages the next front
    return p;
}

// ranks of N points into rank[] (shared memory); S rows of stride Wmax, counts cnt[]
template <int T>
__device__ int peel_ranks(int N, const uint32_t* __restrict__ S, int Wmax, const int32_t* __restrict__ cnt,
                          uint16_t* rank, const PeelSmem& ps, uint32_t* wt32) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int W = (N + 31) / 32;
    // counts -> planes, valid mask
    for (int w = warp; w < W; w += T / 32) {
        const int i = 32 * w + lane;
        const int c = (i < N) ? __ldg(cnt + i) : 0;
#pragma unroll
        for (int b = 0; b < kCB; ++b) {
            const uint32_t pl = __ballot_sync(0xffffffffu, (c >> b) & 1);
            if (lane == 0) ps.C[(size_t)b * W + w] = pl;
        }
        const uint32_t v = __ballot_sync(0xffffffffu, i < N);
        if (lane == 0) ps.V[w] = v;
    }
    __syncthreads();
    // first front: zero counts
    for (int w = t; w < W; w += T) {
        uint32_t z = ps.V[w];
#pragma unroll
        for (int b = 0; b < kCB; ++b) z &= ~ps.C[(size_t)b * W + w];
        ps.F[w] = z;
        ps.A[w] = z;
        for (uint32_t x = z; x; x &= x - 1) rank[32 * w + __ffs(x) - 1] = 0;
    }
    __syncthreads();
    // lanes per word for the column sums: a power of two, at most 32, SP * W <= T
    int SP = 32;
    while (SP > 1 && SP * W > T) SP >>= 1;
    int k = 0;
    for (; k < N; ++k) {
        // front member list
        const uint32_t pc = (t < W) ? __popc(ps.F[t]) : 0u;
        uint32_t nf = 0;
        uint32_t base = block_exclusive_scan<T>(pc, wt32, &nf);
        if (t < W)
            for (uint32_t x = ps.F[t]; x; x &= x - 1) ps.list[base++] = (uint16_t)(32 * t + __ffs(x) - 1);
        __syncthreads();
        if (nf == 0) break;
        const int w = t / SP, sl = t % SP;
        uint32_t acc[kDB];
#pragma unroll
        for (int b = 0; b < kDB; ++b) acc[b] = 0u;
        if (w < W) {
            // bit-sliced column sums: the member rows' words are loaded eight at a time
            // (eight L2 requests in flight per lane), counted in a 4-plane counter and
            // added into the kDB-plane accumulator once per batch
            constexpr int kBatch = 8;
            for (int j0 = sl; j0 < (int)nf; j0 += kBatch * SP) {
                uint32_t xs[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int j = j0 + u * SP;
                    xs[u] = (j < (int)nf) ? __ldg(S + (size_t)ps.list[j] * Wmax + w) : 0u;
                }
                uint32_t s0 = 0u, s1 = 0u, s2 = 0u, s3 = 0u;
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const uint32_t c0 = s0 & xs[u];
                    s0 ^= xs[u];
                    const uint32_t c1 = s1 & c0;
                    s1 ^= c0;
                    const uint32_t c2 = s2 & c1;
                    s2 ^= c1;
                    s3 ^= c2;
                }
                uint32_t cy = 0u;
                const uint32_t sv[4] = {s0, s1, s2, s3};
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t x = acc[b], y = sv[b];
                    acc[b] = x ^ y ^ cy;
                    cy = (x & y) | (cy & (x ^ y));
                }
#pragma unroll
                for (int b = 4; b < kDB; ++b) {
                    const uint32_t x = acc[b];
                    acc[b] = x ^ cy;
                    cy = x & cy;
                }
            }
        }
        // combine the SP partial sums of a word (consecutive lanes) with full adders
        for (int off = 1; off < SP; off <<= 1) {
            uint32_t c = 0u;
#pragma unroll
            for (int b = 0; b < kDB; ++b) {
                const uint32_t o = __shfl_xor_sync(0xffffffffu, acc[b], off);
                const uint32_t s2 = acc[b] ^ o ^ c;
                c = (acc[b] & o) | (c & (acc[b] ^ o));
                acc[b] = s2;
            }
        }
        if (w < W && sl == 0) {
            // decrement: doubled for the first front
            uint32_t dec[kCB];
#pragma unroll
            for (int b = 0; b < kCB; ++b) dec[b] = 0u;
            if (k == 0) {
#pragma unroll
                for (int b = 1; b < kCB; ++b) dec[b] = (b - 1 < kDB) ? acc[b - 1] : 0u;
            } else {
#pragma unroll
                for (int b = 0; b < kDB; ++b) dec[b] = acc[b];
            }
            uint32_t bor = 0u, any = 0u;
#pragma unroll
            for (int b = 0; b < kCB; ++b) {
                const uint32_t x = ps.C[(size_t)b * W + w];
                const uint32_t d = x ^ dec[b] ^ bor;
                bor = (~x & dec[b]) | (~(x ^ dec[b]) & bor);
                ps.C[(size_t)b * W + w] = d;
                any |= d;
            }
            const uint32_t sign = ps.C[(size_t)(kCB - 1) * W + w];
            const uint32_t nz = (sign | ~any) & ~ps.A[w] & ps.V[w];
            ps.A[w] |= nz;
            for (uint32_t x = nz; x; x &= x - 1) rank[32 * w + __ffs(x) - 1] = (uint16_t)(k + 1);
            ps.V[W + w] = nz;  // next front, staged after the valid mask
        }
        __syncthreads();
        if (t < W) ps.F[t] = ps.V[W + t];
        __syncthreads();
    }
    return k;
}


// ---------------------------------------------------------------------------------------
// crowding and survivors (two objectives), one CTA per population
// ---------------------------------------------------------------------------------------
struct SelSmem {
    float* obj;                 // [N][2]
    uint16_t* rank;             // [N]
    float* cd;                  // [N]
    unsigned long long* key;    // [K2]: next_pow2(2N) sort entries
    uint16_t* fs;               // [N] first sorted position of each rank
    uint16_t* fe;               // [N] last sorted position of each rank
    uint32_t* rb;               // [N + 1] survivor entries before each rank
    unsigned char* peel;        // peel_smem_bytes(N)
};

__host__ __device__ inline size_t sel_smem_bytes(int N) {
    const int K2 = npow2(2 * N);
    size_t b = (size_t)N * 8;
    b += ((size_t)N * 2 + 15) / 16 * 16;
    b += ((size_t)N * 4 + 15) / 16 * 16;
    b += (size_t)K2 * 8;
    b += ((size_t)N * 2 + 15) / 16 * 16 * 2;
    b += ((size_t)(N + 1) * 4 + 15) / 16 * 16;
    b += peel_smem_bytes(N);
    return (b + 15) / 16 * 16;
}

__device__ inline SelSmem sel_carve(unsigned char* base, int N) {
    const int K2 = npow2(2 * N);
    SelSmem s;
    size_t off = 0;
    s.obj = (float*)(base + off);
    off += (size_t)N * 8;
    s.rank = (uint16_t*)(base + off);
    off += ((size_t)N * 2 + 15) / 16 * 16;
    s.cd = (float*)(base + off);
    off += ((size_t)N * 4 + 15) / 16 * 16;
    s.key = (unsigned long long*)(base + off);
    off += (size_t)K2 * 8;
    s.fs = (uint16_t*)(base + off);
    off += ((size_t)N * 2 + 15) / 16 * 16;
    s.fe = (uint16_t*)(base + off);
    off += ((size_t)N * 2 + 15) / 16 * 16;
    s.rb = (uint32_t*)(base + off);
    off += ((size_t)(N + 1) * 4 + 15) / 16 * 16;
    s.peel = base + off;
    return s;
}

__device__ __forceinline__ uint32_t cd_key(float c) {
    const uint32_t k = okey(c);
    return (k == 0xFFFFFFFFu) ? 0xFFFFFFFFu : ~k;
}

// front bounds of the (rank, objective, index) order held in s.key[0, N)
template <int T>
__device__ void front_bounds(int N, const SelSmem& s) {
    for (int p = threadIdx.x; p < N; p += T) {
        const int r = (int)(s.key[p] >> 48);
        if (p == 0 || (int)(s.key[p - 1] >> 48) != r) s.fs[r] = (uint16_t)p;
        if (p == N - 1 || (int)(s.key[p + 1] >> 48) != r) s.fe[r] = (uint16_t)p;
    }
}

// one objective's contribution to the crowding distance (core/population.hpp:453-489) over
// the reference's front lists, s.key[0, N) in (rank, objective o, index) order: rank-0
// points are two adjacent entries (index, copy 0/1), other points one
template <int T>
__device__ void crowding_pass(int N, int o, const SelSmem& s) {
#define VAL(pos) s.obj[2 * (int)(s.key[pos] & 0xFFFFu) + o]
    for (int p = threadIdx.x; p < N; p += T) {
        const int i = (int)(s.key[p] & 0xFFFFu);
        const int r = (int)(s.key[p] >> 48);
        const int f = s.fs[r], l = s.fe[r];
        const int size = l - f + 1;
        if (r == 0) {
            // entries 2(p-f) and 2(p-f)+1 of the doubled list of 2*size entries
            if (size == 1 || p == f || p == l) {
                s.cd[i] = INFINITY;
            } else {
                const float range = __fsub_rn(VAL(l), VAL(f));
                if (range > 0.0f) {
                    const float v = VAL(p);
                    const float da = __fdiv_rn(__fsub_rn(v, VAL(p - 1)), range);
                    const float db = __fdiv_rn(__fsub_rn(VAL(p + 1), v), range);
                    s.cd[i] = __fadd_rn(__fadd_rn(s.cd[i], da), db);
                }
            }
        } else {
            if (size <= 2 || p == f || p == l) {
                s.cd[i] = INFINITY;
            } else {
                const float range = __fsub_rn(VAL(l), VAL(f));
                if (range > 0.0f)
                    s.cd[i] = __fadd_rn(s.cd[i], __fdiv_rn(__fsub_rn(VAL(p + 1), VAL(p - 1)), range));
            }
        }
    }
#undef VAL
}

__device__ __forceinline__ unsigned long long order_key(int rank, float v, int i) {
    return ((unsigned long long)rank << 48) | ((unsigned long long)okey(v) << 16) | (unsigned long long)i;
}

// crowding from the orders nsga_order_kernel computed (ord[o * ostride + position]); leaves
// s.key holding the objective-1 order and s.fs / s.fe its front bounds
template <int T>
__device__ void crowding_given(int N, const SelSmem& s, const int32_t* __restrict__ ord, int ostride) {
    const int t = threadIdx.x;
    for (int i = t; i < N; i += T) s.cd[i] = 0.0f;
    for (int o = 0; o < 2; ++o) {
        __syncthreads();
        staged<T, 4>(
            N, [&](int p) { return __ldg(ord + (size_t)o * ostride + p); },
            [&](int p, int i) { s.key[p] = order_key(s.rank[i], s.obj[2 * i + o], i); });
        __syncthreads();
        front_bounds<T>(N, s);
        __syncthreads();
        crowding_pass<T>(N, o, s);
    }
    __syncthreads();
}

// survivors (core/population.hpp:491-517): whole fronts while they fit, ordered by
// (last objective, index, copy) -- the objective-1 order in s.key with every rank-0 point
// taken twice -- then the cut front by (-crowding, index, copy), sorted alone
template <int T>
__device__ void select_given(int N, int P, const SelSmem& s, int32_t* g_sel, int32_t* g_rank, float* g_cd,
                             float* fmin_out, uint32_t* wt32) {
    const int t = threadIdx.x;
    __shared__ int s_cut;
    const int R = (int)(s.key[N - 1] >> 48) + 1;  // ranks 0 .. R-1 all occur
    // survivor entries of each rank (rank 0 counts twice), prefix over ranks
    const int ch = (R + T - 1) / T;
    const int r0 = min(R, t * ch), r1 = min(R, r0 + ch);
    uint32_t loc = 0;
    for (int r = r0; r < r1; ++r) loc += (uint32_t)(s.fe[r] - s.fs[r] + 1) * (r == 0 ? 2u : 1u);
    if (t == 0) s_cut = R;
    uint32_t run = block_exclusive_scan<T>(loc, wt32, nullptr);
    for (int r = r0; r < r1; ++r) {
        s.rb[r] = run;
        run += (uint32_t)(s.fe[r] - s.fs[r] + 1) * (r == 0 ? 2u : 1u);
        if (run > (uint32_t)P && s.rb[r] <= (uint32_t)P) s_cut = r;  // exactly one rank crosses P
    }
    __syncthreads();
    const int cut = s_cut;
    float fmin = INFINITY;
    // whole fronts before the cut
    for (int p = t; p < N; p += T) {
        const int r = (int)(s.key[p] >> 48);
        if (r >= cut) continue;
        const int i = (int)(s.key[p] & 0xFFFFu);
        const int k = p - s.fs[r];
        const int q = (int)s.rb[r] + (r == 0 ? 2 * k : k);
        for (int c = 0; c < (r == 0 ? 2 : 1); ++c) {
            g_sel[q + c] = i;
            g_rank[q + c] = r;
            g_cd[q + c] = s.cd[i];
        }
        fmin = fminf(fmin, s.obj[2 * i]);
    }
    const int f = (cut < R) ? s.fs[cut] : 0;
    const int nc = (cut < R) ? s.fe[cut] - f + 1 : 0;
    __syncthreads();
    if (cut < R) {
        // the cut front's points, in order, into s.fs; then its entries sorted by
        // (cd descending, index, copy) in s.key (sized for 2N entries)
        for (int k = t; k < nc; k += T) s.fs[k] = (uint16_t)(s.key[f + k] & 0xFFFFu);
        __syncthreads();
        const int mult = (cut == 0) ? 2 : 1;
        const int E = nc * mult, K2 = npow2(E);
        const int take = P - (int)s.rb[cut];
        for (int e = t; e < K2; e += T) {
            unsigned long long kk = ~0ull;
            if (e < E) {
                const int i = s.fs[e / mult];
                kk = ((unsigned long long)cd_key(s.cd[i]) << 32) | ((unsigned long long)i << 1) |
                     (unsigned long long)(e % mult);
            }
            s.key[e] = kk;
        }
        __syncthreads();
        bitonic_u64<T>(s.key, K2);
        for (int k = t; k < take; k += T) {
            const int i = (int)((s.key[k] >> 1) & 0x7FFFu);
            const int q = (int)s.rb[cut] + k;
            g_sel[q] = i;
            g_rank[q] = cut;
            g_cd[q] = s.cd[i];
            fmin = fminf(fmin, s.obj[2 * i]);
        }
    }
    *fmin_out = fmin;
}

__device__ float block_min_f(float v, float* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) red[w] = v;
    __syncthreads();
    float r = red[0];
    for (int i = 1; i < (int)(blockDim.x / 32); ++i) r = fminf(r, red[i]);
    __syncthreads();
    return r;
}

// Selection launches (core/population.hpp:409-517): mode 0 works on the 2P pool of fit[cur]
// and picks the survivors; mode 1 ranks the P population (initialisation); mode 2 does
// the same only for populations the diversity pass rebuilt (*nu < P).  A population whose peel
// gave up a wait has a front table that is half written: nothing of it is selected any more.
__device__ __forceinline__ bool select_active(const PopDesc& d, int mode) {
    if (d.stuck) return false;
    if (mode == 0) return !at_limit(d);
    if (mode == 2) return d.advanced && __ldg(d.nu) < d.P;
    return true;
}

// Ranks by peeling, on one thread-block cluster per population.  A point's dominator row
// stays in registers for the whole peel: eight lanes hold it, 4 WL bytes each, and a warp
// 16 points.  Mask k holds the points of the fronts 0..k; a point joins front k + 1 when its
// dominators outside the mask are no more than those of the first front (whose points are
// listed twice, so that each takes two off the count).
//
// A front is a chain: counts, the CTA's 256 bits gathered, the exchange, the mask's size.
//  - A CTA sends its words to every CTA with st.async, which completes on the receiver's
//    mbarrier: 650 cycles a front for 16 CTAs, where 16-bit stores by every warp and a cluster
//    barrier took 1900 and one warp's stores and a cluster barrier 1300.  Four masks go round:
//    a CTA sends mask k + 3 only after every other CTA has sent mask k + 2, and none does
//    before it is done reading masks k - 1 and k.
//  - Waits are bounded.  A CTA whose wait runs out gives up, but words may still be on their way
//    to it: it says how many masks it has sent, sends the one that others wait for, and leaves
//    when every mask that was sent has arrived (a second bounded wait).
//  - A step (four points) is counted only if one of its points can come to zero: its count less
//    the points that joined since it was last counted.  About half the steps of a front are.
//  - Counts are bound by logic (two cycles a warp) and population counts (eight): 16 words take
//    6 full adders and 10 counts, about equal shares.
// Measured, NSGA-II generations of 4096-point pools (7 fronts) and 3000-point pools (15 to 19
// fronts): 67.3 -> 64.8 and 56.0 -> 51.6 us a generation; the ranks of 4096 points in all fronts
// and their crowding 94.4 -> 86.8 us.  (Merging the rows of a front's members by column instead,
// bit-sliced, took about 6 us a front at N = 4096.)
//
// The pool of a generation (mode 0) is peeled only up to the front where the survivors
// (rank-0 points counted twice) first exceed P: that front is cut by crowding, and no
// later front is selected.  The points left then get that front's rank + 1 as one last
// front.  Selection, crowding of every selected point and the ranks kept for the next
// generation are the same as with every front peeled.  Ranks -> domcnt[0, N).
constexpr int kPeelThreads = 512;
// points of a CTA whose warps take S steps of four points
constexpr int peel_points(int S) { return kPeelThreads / 32 * 4 * S; }

// set bits of x[0, n) (n = 4, 8 or 16): full adders until the logic (two cycles a warp) takes
// about as long as the counts left (eight cycles a warp)
template <int n>
__device__ __forceinline__ int count_bits(const uint32_t (&x)[n]) {
    int one = 0, two = 0;
    auto add3 = [](uint32_t& s, uint32_t b, uint32_t c) {  // s <- the sum bit; returns the carry
        const uint32_t cy = (s & b) | (c & (s | b));
        s = s ^ b ^ c;
        return cy;
    };
    auto add7 = [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t e, uint32_t f, uint32_t g) {
        two += __popc(add3(a, b, c)) + __popc(add3(d, e, f));
        two += __popc(add3(a, d, g));
        return a;
    };
    if constexpr (n == 4) {
        uint32_t a = x[0];
        two = __popc(add3(a, x[1], x[2]));
        one = __popc(a) + __popc(x[3]);
    } else {
#pragma unroll
        for (int i = 0; i < n; i += 8)
            one += __popc(add7(x[i], x[i + 1], x[i + 2], x[i + 3], x[i + 4], x[i + 5], x[i + 6])) + __popc(x[i + 7]);
    }
    return one + 2 * two;
}

__device__ __forceinline__ uint32_t shared_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// the current phase of the barrier at `at` has the given parity and completes within `polls` polls
__device__ __forceinline__ bool mask_arrived(uint32_t at, uint32_t parity, uint32_t polls) {
    uint32_t done = 0u;
    for (uint32_t n = 0; n < polls && !done; ++n)
        asm volatile(
            "{.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;}"
            : "=r"(done)
            : "r"(at), "r"(parity)
            : "memory");
    return done != 0u;
}

__device__ __forceinline__ uint32_t shared_addr_in(uint32_t addr, int cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}

// A CTA that gave up at mask k waits here for the words on their way to it; every CTA has sent all
// that it is going to.  A CTA that sent mask k + 1 waits for it, so it gave up too, and none got
// further without this CTA's part, which it sends now (its bits do not matter).  CTAs that did
// not give up have all of mask k, the last one sent then.  (Out of line: in the kernel it took
// registers that the rows need, 31.0 -> 32.5 us for 4096 points of 12 fronts.)
template <int QW>
__device__ __noinline__ void peel_drain(uint32_t masks, int mask_words, uint32_t bars, const int* gave_up, int k, int csize,
                                        int crank) {
    const int t = threadIdx.x;
    int last = k;
    for (int c = 0; c < csize; ++c) last = max(last, gave_up[c]);
    if (last > k && t < 4 * csize) {
        const int q = t & 3, b = last & 3;
        if (t == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 8 * b), "r"(16 * QW * csize)
                         : "memory");
        const uint32_t to = shared_addr_in(masks + 4 * (b * mask_words + QW * (q * csize + crank)), t >> 2);
        const uint32_t at = shared_addr_in(bars + 8 * b, t >> 2);
        for (int w = 0; w < QW; ++w)
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(to + 4 * w),
                         "r"(0u), "r"(at)
                         : "memory");
    }
    for (int b = k; b <= last; ++b) mask_arrived(bars + 8 * (b & 3), (uint32_t)(b >> 2) & 1u, 4u * kWaitPolls);
}

// S = 4: the rows fit the registers.  S = 8 (half of them spill): clusters of half the size, for
// devices that cannot place 16 CTAs together (launch_peel).
template <int WL, int S>
__global__ void __launch_bounds__(kPeelThreads, 1) nsga_peel_rows_kernel(PopDesc* dd, int mode) {
    dep_wait();
    namespace cg = cooperative_groups;
    using Part = std::conditional_t<S == 4, uint16_t, uint32_t>;  // a warp's points
    constexpr int NW = 8 * WL;  // words of a mask
    constexpr int QW = S / 2;   // words of a CTA in each quarter of the points
    constexpr uint32_t kAll = (1u << S) - 1u;
    __shared__ __align__(16) uint32_t F[4][NW];  // the points of the fronts 0..k in F[k & 3]
    __shared__ __align__(16) Part out[kPeelThreads / 32];  // the CTA's part of the next mask
    __shared__ __align__(8) uint64_t bar[4];  // of each mask: every CTA's part has arrived
    __shared__ uint32_t s_polls;  // of one wait (no register to spare for it)
    __shared__ int gave_up[16];  // the last mask that each CTA of the cluster sent before it gave up, or -1
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    PopDesc& d = dd[blockIdx.x / csize];
    // (loaded together: one trip to L2, not one for the decision and one for the rest)
    const volatile PopDesc& vd = d;
    const int P = vd.P, Wmax = vd.domW;
    const uint32_t polls = vd.wait_polls;
    if (!select_active(d, mode)) return;  // the same decision in every CTA of the cluster
    const int N = (mode == 0) ? 2 * P : P;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, sub = lane & 7;
    // A CTA has QW words from each of the four quarters of the points: a pool's survivors come in
    // the order of their last fronts, so neighbours are at work together.
    auto word_of = [&](int quarter) { return QW * (quarter * csize + crank); };
    const int word = word_of(warp / 4) + (warp & 3) * 4 * S / 32, bit0 = (warp & 3) * 4 * S % 32;
    const int p0 = 32 * word + bit0;  // the warp's points; step s: p0 + 4 s + lane / 8

    if (t < 4) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_addr(&bar[t])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (t < 16) gave_up[t] = -1;
    if (t == 0) s_polls = 4u * polls;  // a poll of shared memory is shorter than one of L2
    // (Words past N stay zero in the masks: rows may hold anything there.)
    for (int w = t; w < NW; w += kPeelThreads) {
        F[1][w] = (w < N / 32) ? 0xFFFFFFFFu : (w == N / 32 && (N & 31)) ? (1u << (N & 31)) - 1u : 0u;
        F[0][w] = F[2][w] = F[3][w] = 0u;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    uint32_t x[S][WL];
#pragma unroll
    for (int st = 0; st < S; ++st) {
        const int p = p0 + 4 * st + (lane >> 3);
#pragma unroll
        for (int c = 0; c < WL / 4; ++c) {
            const int w = 32 * c + 4 * sub;
            const uint4 v = (p < N && w < Wmax) ? __ldg(reinterpret_cast<const uint4*>(d.domS + (size_t)p * Wmax + w))
                                                : make_uint4(0u, 0u, 0u, 0u);
            x[st][4 * c] = v.x, x[st][4 * c + 1] = v.y, x[st][4 * c + 2] = v.z, x[st][4 * c + 3] = v.w;
        }
    }
    // counts of the points' dominators in a mask, for the steps in `act` (0 for the others)
    auto dominators_in = [&](const uint32_t* f, uint32_t act, int (&cnt)[S]) {
        uint32_t m[WL];
#pragma unroll
        for (int c = 0; c < WL / 4; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(f + 32 * c + 4 * sub);
            m[4 * c] = v.x, m[4 * c + 1] = v.y, m[4 * c + 2] = v.z, m[4 * c + 3] = v.w;
        }
        uint32_t pk[S / 2] = {};  // two steps a word
#pragma unroll
        for (int st = 0; st < S; ++st) {
            if (!((act >> st) & 1u)) continue;
            uint32_t y[WL];
#pragma unroll
            for (int u = 0; u < WL; ++u) y[u] = x[st][u] & m[u];
            pk[st >> 1] |= (uint32_t)count_bits<WL>(y) << (16 * (st & 1));
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1)
#pragma unroll
            for (int h = 0; h < S / 2; ++h) pk[h] += __shfl_xor_sync(0xffffffffu, pk[h], o);
#pragma unroll
        for (int st = 0; st < S; ++st) cnt[st] = (int)((pk[st >> 1] >> (16 * (st & 1))) & 0xFFFFu);
    };
    uint32_t ranked = 0u, mine = 0u;  // the warp's points in the fronts so far, in the next one: bit 4 s + lane / 8
    // the CTA's part of mask b to every CTA, a quarter's words a thread
    auto deliver = [&](int b) {
        if (t < 4 * csize) {
            const int q = t & 3;
            const uint32_t to = shared_addr(&F[b][word_of(q)]), at = shared_addr(&bar[b]);
            if (t == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(at), "r"(16 * QW * csize) : "memory");
            const uint32_t rto = shared_addr_in(to, t >> 2), rat = shared_addr_in(at, t >> 2);
            if constexpr (QW == 2) {
                const uint2 v = reinterpret_cast<const uint2*>(out)[q];
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
                             ::"r"(rto), "r"(v.x), "r"(v.y), "r"(rat)
                             : "memory");
            } else {
                const uint4 v = reinterpret_cast<const uint4*>(out)[q];
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                             ::"r"(rto), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(rat)
                             : "memory");
            }
        }
    };
    // points of the steps `act` at or below zero and not ranked yet join the next front: the
    // CTA's bits of mask b gathered, then sent to every CTA
    auto send_front = [&](int b, uint32_t act, const int (&left)[S]) {
        uint32_t bits = 0u;
        if (act) {
#pragma unroll
            for (int st = 0; st < S; ++st) {
                const uint32_t v =
                    __ballot_sync(0xffffffffu, ((act >> st) & 1u) && left[st] <= 0 && p0 + 4 * st + (lane >> 3) < N);
                bits |= ((v & 1u) | ((v >> 7) & 2u) | ((v >> 14) & 4u) | ((v >> 21) & 8u)) << (4 * st);
            }
        }
        mine = bits & ~ranked;
        ranked |= mine;
        if (lane == 0) out[warp] = (Part)ranked;
        __syncthreads();
        deliver(b);
    };
    // mask k is complete; false (in every thread of the CTA) when the wait ran out
    auto await_front = [&](int k) {
        const uint32_t left = *static_cast<volatile uint32_t*>(&s_polls);
        return __syncthreads_and(mask_arrived(shared_addr(&bar[k & 3]), (uint32_t)(k >> 2) & 1u, left)) != 0;
    };
    __syncthreads();
    int need[S];  // every point: all its dominators, and once those of the first front are known, them once more
    dominators_in(F[1], kAll, need);
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA's masks and barriers are set up
    send_front(0, kAll, need);

    int survivors = 0, rest = 0, start = 0;
    int reach[S] = {};  // listed points at which a step's points may come to zero
    // thread 0 of the cluster's first CTA records the front table (start of each front in
    // rank order, the cut front) for the grid-wide crowding and placement of mode 0
    int32_t* const ft = (crank == 0 && t == 0) ? d.nft : nullptr;
    int k = 0;
    bool stuck = false;
    for (;; ++k) {
        const uint32_t* const f = F[k & 3];
        if (!await_front(k)) {
            stuck = true;
            break;
        }
        int total = 0;  // points of the fronts 0..k
#pragma unroll
        for (int c = 0; c < NW / 32; ++c) total += __popc(f[32 * c + lane]);
        total = __reduce_add_sync(0xffffffffu, total);
        const int nf = total - start;  // every CTA sees the same front
        survivors += (k == 0) ? 2 * nf : nf;
        const bool cut = mode == 0 && nf > 0 && survivors > d.P;
        const uint32_t members = mine;
        if (nf > 0 && !cut) {
            // the steps with a point that may come to zero with this front
            uint32_t act = 0u;
#pragma unroll
            for (int st = 0; st < S; ++st)
                act |= __any_sync(0xffffffffu, reach[st] <= total && !((ranked >> (4 * st + (lane >> 3))) & 1u)) ? 1u << st : 0u;
            int left[S];
#pragma unroll
            for (int st = 0; st < S; ++st) left[st] = 1;
            if (act) {
                int cnt[S];
                dominators_in(f, act, cnt);
#pragma unroll
                for (int st = 0; st < S; ++st) {
                    if (!((act >> st) & 1u)) continue;
                    if (k == 0) need[st] -= cnt[st];
                    left[st] = need[st] - cnt[st];
                    reach[st] = (p0 + 4 * st + (lane >> 3) < N) ? left[st] + total : INT_MAX;
                }
            }
            send_front((k + 1) & 3, act, left);
        }
        // while the next mask is on its way: the ranks of the warp's members of front k, and
        // their places in the list of fronts
        if (ft) ft[2 + k] = start;
        if (members) {
            const uint32_t* const before = F[(k + 3) & 3];  // fronts 0..k - 1
            int pre = 0;
#pragma unroll
            for (int c = 0; c < NW / 32; ++c) {
                const int w = 32 * c + lane;
                const uint32_t v = (k == 0) ? f[w] : f[w] & ~before[w];
                pre += (w < word) ? __popc(v) : (w == word) ? __popc(v & ((1u << bit0) - 1u)) : 0;
            }
            pre = __reduce_add_sync(0xffffffffu, pre);
            if (lane < 4 * S && ((members >> lane) & 1u)) {
                d.domcnt[p0 + lane] = k;
                if (d.nlist) d.nlist[start + pre + __popc(members & ((1u << lane) - 1u))] = p0 + lane;
            }
        }
        start = total;
        if (nf == 0) {
            if (ft) {
                ft[0] = k;
                ft[1] = -1;
            }
            break;
        }
        if (cut) {
            rest = k + 1;
            if (ft) {  // the cut front k, then the points left as one last front
                ft[1] = k;
                ft[3 + k] = start;
                ft[4 + k] = N;
                ft[0] = (start < N) ? k + 2 : k + 1;
            }
            break;
        }
    }
    if (stuck) {
        if (t < csize) *cluster.map_shared_rank(&gave_up[crank], t) = k;
        if (t == 0) set_stuck(d);
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (lane < 4 * S && p0 + lane < N && !((ranked >> lane) & 1u)) d.domcnt[p0 + lane] = rest;
    // no CTA leaves while another may still send to it
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (stuck) peel_drain<QW>(shared_addr(F), NW, shared_addr(bar), gave_up, k, csize, crank);
}

using PeelFn = void (*)(PopDesc*, int);

// CTAs of a peel cluster at most: 16, or the 8 that any device places, where 16 (a non-portable size:
// as many free SMs in one GPC) cannot be: a partition of the GPU, or BRKGA_PEEL_CLUSTER=8
static int peel_cluster_limit(PeelFn fn) {
    const char* v = std::getenv("BRKGA_PEEL_CLUSTER");
    if (v && std::atoi(v) == 8) return 8;
    static std::mutex mu;
    static std::map<int, int> known;  // device -> limit
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find(dev);
    if (it != known.end()) return it->second;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kPeelThreads);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    return known[dev] = (e == cudaSuccess && clusters > 0) ? 16 : 8;
}

// one cluster per population: a CTA for every 256 of its (at most maxN) points, 512 where the
// cluster would be too large for the device
static cudaError_t launch_peel(PopDesc* dd, int npops, int maxN, int mode, cudaStream_t s) {
    if (maxN > kMaxPool) return cudaErrorInvalidValue;
    PeelFn fn = maxN <= 1024   ? nsga_peel_rows_kernel<4, 4>
                : maxN <= 2048 ? nsga_peel_rows_kernel<8, 4>
                               : nsga_peel_rows_kernel<16, 4>;
    int csize = 1;
    while (csize * peel_points(4) < maxN) csize *= 2;
    if (csize > 8 && peel_cluster_limit(fn) < csize) {
        fn = nsga_peel_rows_kernel<16, 8>;
        csize = 8;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(npops * csize);
    cfg.blockDim = dim3(kPeelThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = csize;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, dd, mode);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

// The pool ordered by (rank, objective o, index) for o = blockIdx.y, by exact counting:
// position(i) = #{j : key_j < key_i} over unique composite keys.  N^2 compares per
// objective spread over the grid; one warp per point.
constexpr int kOrdThreads = 1024, kOrdPerCta = kOrdThreads / 32;

__global__ void __launch_bounds__(kOrdThreads) nsga_order_kernel(PopDesc* dd, int mode) {
    dep_wait();
    extern __shared__ unsigned long long okeys[];  // [N]
    const PopDesc& d = dd[blockIdx.z];
    if (!select_active(d, mode)) return;
    const int N = (mode == 0) ? 2 * d.P : d.P;
    const int base = blockIdx.x * kOrdPerCta;
    if (base >= N) return;
    const int o = blockIdx.y, t = threadIdx.x;
    const float* f = d.fit[d.cur];
    staged<kOrdThreads, 4>(
        N, [&](int i) { return make_int2(__ldg(d.domcnt + i), __float_as_int(__ldg(f + 2 * i + o))); },
        [&](int i, int2 v) { okeys[i] = order_key(v.x, __int_as_float(v.y), i); });
    __syncthreads();
    const int lane = t & 31, i = base + (t >> 5);
    const unsigned long long me = (i < N) ? okeys[i] : 0ull;
    int cnt = 0;
#pragma unroll 8
    for (int j = lane; j < N; j += 32) cnt += (okeys[j] < me) ? 1 : 0;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
    if (lane == 0 && i < N) d.nord[(size_t)o * 2 * d.P + cnt] = i;
}

// Mode 0 (the pool of a generation), one warp per pool point, over the members of its own
// front only (the peel's lists): its position in the front in each objective order, its
// neighbours and the front's extremes in both orders, so its crowding distance (the float
// operations of crowding_pass in the same order) and, for whole fronts before the cut, its
// survivor entries: front r starts at survivor entry first(r) + size(0) (rank-0 points
// count twice), members in objective-1 order, a rank-0 point as two adjacent entries; and
// the smallest first objective among them (atomic minimum of order keys).  A value is
// recovered from its key, and equal keys go by place in the list, which is index order: ten
// 32-bit figures a point and a reduction instruction each took 9.5 us for a pool of 4096
// points, (key, index) pairs in 64 bits and shuffles 10.6 us.  CTAs take the points in
// rank order, kFrontWarps at a time, so a CTA's warps share a front, whose members' keys
// the CTA stages in shared memory once (a warp whose point lies in a later front reads
// that front from global memory).  Points of the last front of a peel stopped at the cut
// are never selected and are skipped.  Work: the sum of the squared front sizes instead
// of N^2 per objective.
constexpr int kFrontWarps = 8;

__device__ __forceinline__ float key_value(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// one member's two keys -> the running position, neighbours and extremes of the point.  The
// order is (key, index); members are listed by index, so among equal keys the place in the
// list decides.
struct FrontScan {
    uint32_t me0, me1;
    int place;  // of the point in its front's list
    int below0 = 0, below1 = 0;
    uint32_t lo0 = 0u, hi0 = ~0u, lo1 = 0u, hi1 = ~0u;  // neighbours (0 / ~0: none)
    uint32_t mn0 = ~0u, mx0 = 0u, mn1 = ~0u, mx1 = 0u;  // front extremes
    __device__ __forceinline__ void add(uint32_t k0, uint32_t k1, int j) {
        const bool first = j < place, other = j != place;
        const bool b0 = k0 < me0 || (first && k0 == me0), b1 = k1 < me1 || (first && k1 == me1);
        below0 += b0 ? 1 : 0;
        below1 += b1 ? 1 : 0;
        lo0 = max(lo0, b0 ? k0 : 0u);
        lo1 = max(lo1, b1 ? k1 : 0u);
        hi0 = min(hi0, (other && !b0) ? k0 : ~0u);
        hi1 = min(hi1, (other && !b1) ? k1 : ~0u);
        mn0 = min(mn0, k0), mx0 = max(mx0, k0);
        mn1 = min(mn1, k1), mx1 = max(mx1, k1);
    }
    __device__ __forceinline__ void reduce() {
        constexpr uint32_t all = 0xffffffffu;
        below0 = __reduce_add_sync(all, below0), below1 = __reduce_add_sync(all, below1);
        lo0 = __reduce_max_sync(all, lo0), hi0 = __reduce_min_sync(all, hi0);
        lo1 = __reduce_max_sync(all, lo1), hi1 = __reduce_min_sync(all, hi1);
        mn0 = __reduce_min_sync(all, mn0), mx0 = __reduce_max_sync(all, mx0);
        mn1 = __reduce_min_sync(all, mn1), mx1 = __reduce_max_sync(all, mx1);
    }
};

// one pool point of nsga_front_crowd_kernel (one warp): the scan of its front, then lane
// 0's crowding distance and survivor entries
// A survivor's keys and objectives into the other buffer, at entry q (and q2 >= 0: the
// second entry of a first-front point), by one warp: four 128-bit loads in flight per lane.
__device__ __forceinline__ void copy_survivor(const PopDesc& d, int src_row, int q, int q2, int lane) {
    const int ld4 = d.ld / 4, m = d.m, cur = d.cur;
    const float4* src = reinterpret_cast<const float4*>(d.keys[cur]) + (size_t)src_row * ld4;
    float4* dst = reinterpret_cast<float4*>(d.keys[cur ^ 1]) + (size_t)q * ld4;
    float4* dst2 = (q2 >= 0) ? reinterpret_cast<float4*>(d.keys[cur ^ 1]) + (size_t)q2 * ld4 : nullptr;
    int c = lane;
    for (; c + 96 < ld4; c += 128) {
        const float4 a0 = src[c], a1 = src[c + 32], a2 = src[c + 64], a3 = src[c + 96];
        dst[c] = a0;
        dst[c + 32] = a1;
        dst[c + 64] = a2;
        dst[c + 96] = a3;
        if (dst2) {
            dst2[c] = a0;
            dst2[c + 32] = a1;
            dst2[c + 64] = a2;
            dst2[c + 96] = a3;
        }
    }
    for (; c < ld4; c += 32) {
        const float4 a = src[c];
        dst[c] = a;
        if (dst2) dst2[c] = a;
    }
    if (lane < m) {
        const float v = d.fit[cur][(size_t)src_row * m + lane];
        d.fit[cur ^ 1][(size_t)q * m + lane] = v;
        if (q2 >= 0) d.fit[cur ^ 1][(size_t)q2 * m + lane] = v;
    }
}

__device__ __forceinline__ void front_crowd_point(const PopDesc& d, const int32_t* __restrict__ ft,
                                                  const float2* __restrict__ f2, const int32_t* __restrict__ list,
                                                  const uint2* fkeys, int r0, int lane, int pos, int cut,
                                                  uint32_t* s_min) {
    const int i = __ldg(list + pos);
    const int r = __ldg(d.domcnt + i);
    const int fs = __ldg(ft + 2 + r), size = __ldg(ft + 3 + r) - fs;
    const float2 vi = __ldg(f2 + i);
    FrontScan sc;
    sc.me0 = okey(vi.x);
    sc.me1 = okey(vi.y);
    sc.place = pos - fs;
    if (r == r0) {
        for (int j = lane; j < size; j += 32) {
            const uint2 k = fkeys[j];
            sc.add(k.x, k.y, j);
        }
    } else {
        for (int j = lane; j < size; j += 32) {
            const float2 v = __ldg(f2 + __ldg(list + fs + j));
            sc.add(okey(v.x), okey(v.y), j);
        }
    }
    sc.reduce();  // every lane holds the front's figures
    float cd = 0.0f;
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const int p = o ? sc.below1 : sc.below0;  // position inside the front
        const bool edge = (r == 0) ? (size == 1 || p == 0 || p == size - 1) : (size <= 2 || p == 0 || p == size - 1);
        if (edge) {
            cd = INFINITY;
            continue;
        }
        const float range = __fsub_rn(key_value(o ? sc.mx1 : sc.mx0), key_value(o ? sc.mn1 : sc.mn0));
        if (range > 0.0f) {
            const float vp = key_value(o ? sc.lo1 : sc.lo0), vn = key_value(o ? sc.hi1 : sc.hi0);
            if (r == 0) {
                const float v = key_value(o ? sc.me1 : sc.me0);
                cd = __fadd_rn(__fadd_rn(cd, __fdiv_rn(__fsub_rn(v, vp), range)), __fdiv_rn(__fsub_rn(vn, v), range));
            } else {
                cd = __fadd_rn(cd, __fdiv_rn(__fsub_rn(vn, vp), range));
            }
        }
    }
    if (lane == 0) d.ncdp[i] = cd;
    if (r < cut) {
        const int q = (r == 0) ? 2 * sc.below1 : fs + __ldg(ft + 3) + sc.below1;
        if (lane == 0) {
            d.nsel[q] = i;
            d.nrank[q] = r;
            d.ncd[q] = cd;
            if (r == 0) {
                d.nsel[q + 1] = i;
                d.nrank[q + 1] = r;
                d.ncd[q + 1] = cd;
            }
            atomicMin(s_min, sc.me0);
        }
        copy_survivor(d, i, q, (r == 0) ? q + 1 : -1, lane);
    }
}

__global__ void __launch_bounds__(kFrontWarps * 32) nsga_front_crowd_kernel(PopDesc* dd) {
    dep_wait();
    extern __shared__ uint2 fkeys[];  // [front size]: the staged front's (okey0, okey1)
    __shared__ int s_front[3];        // staged front: rank, first position, size
    __shared__ uint32_t s_min;        // the CTA's smallest first-objective key among survivors
    const PopDesc& d = dd[blockIdx.y];
    if (!select_active(d, 0)) return;
    const int N = 2 * d.P;
    const int32_t* __restrict__ ft = d.nft;
    const int cut = __ldg(ft + 1);
    const int end = (cut >= 0) ? __ldg(ft + 3 + cut) : N;  // positions of the fronts up to the cut
    const int pos0 = blockIdx.x * kFrontWarps;
    if (pos0 >= end) return;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const float2* __restrict__ f2 = reinterpret_cast<const float2*>(d.fit[d.cur]);
    const int32_t* __restrict__ list = d.nlist;
    if (t == 0) {
        const int r0 = __ldg(d.domcnt + __ldg(list + pos0));
        s_front[0] = r0;
        s_front[1] = __ldg(ft + 2 + r0);
        s_front[2] = __ldg(ft + 3 + r0) - s_front[1];
        s_min = 0xFFFFFFFFu;
    }
    __syncthreads();
    const int r0 = s_front[0], fs0 = s_front[1], size0 = s_front[2];
    staged<kFrontWarps * 32, 4>(
        size0, [&](int j) { return __ldg(f2 + __ldg(list + fs0 + j)); },
        [&](int j, float2 v) { fkeys[j] = make_uint2(okey(v.x), okey(v.y)); });
    __syncthreads();
    const int pos = pos0 + w;
    if (pos < end) front_crowd_point(d, ft, f2, list, fkeys, r0, lane, pos, cut, &s_min);
    __syncthreads();
    if (t == 0 && s_min != 0xFFFFFFFFu) atomicMin(d.nfmin, s_min);
}

// Mode 0, over the grid, one warp per member of the cut front: the member's place among
// the front's entries in (crowding descending, index, copy) order, by counting the members
// with a smaller (crowding key, index) (every CTA stages the front's keys), a first-front
// point as two adjacent entries; entries before P - (entries of the whole fronts) become
// survivors, and the warp copies their rows into the other buffer (the front kernel has
// copied the whole fronts' rows).  The population's last CTA (completion counter) then
// finishes the generation: the history entry from the survivors' smallest first objective
// (the atomic minimum of order keys that both kernels feed), the buffer swap and the
// generation count.
__global__ void __launch_bounds__(kFrontWarps * 32) nsga_cut_kernel(PopDesc* dd) {
    dep_wait();
    extern __shared__ unsigned long long ckeys[];  // [cut front size]
    __shared__ uint32_t s_min;
    PopDesc& d = dd[blockIdx.y];
    if (!select_active(d, 0)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) d.advanced = 0;
        return;
    }
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int32_t* __restrict__ ft = d.nft;
    const int cut = __ldg(ft + 1);
    const int fs = __ldg(ft + 2 + cut), nc = __ldg(ft + 3 + cut) - fs;
    const int j0 = blockIdx.x * kFrontWarps;
    if (t == 0) s_min = 0xFFFFFFFFu;
    if (j0 < nc) {  // every CTA reaches the completion count below
        const int mult = (cut == 0) ? 2 : 1;
        const int rb = (cut == 0) ? 0 : fs + __ldg(ft + 3);
        const int take = d.P - rb;
        const int32_t* __restrict__ mem = d.nlist + fs;
        staged<kFrontWarps * 32, 4>(
            nc, [&](int j) { return __ldg(mem + j); },
            [&](int j, int m) { ckeys[j] = ((unsigned long long)cd_key(__ldg(d.ncdp + m)) << 32) | (uint32_t)m; });
        __syncthreads();
        for (int j = j0 + w; j < nc; j += gridDim.x * kFrontWarps) {
            const unsigned long long me = ckeys[j];
            int c = 0;
            for (int k = lane; k < nc; k += 32) c += (ckeys[k] < me) ? 1 : 0;
            c = __reduce_add_sync(0xffffffffu, c);
            const int m = (int)(uint32_t)me, q0 = rb + mult * c;
            if (lane < mult && mult * c + lane < take) {
                const int q = q0 + lane;
                d.nsel[q] = m;
                d.nrank[q] = cut;
                d.ncd[q] = __ldg(d.ncdp + m);
                atomicMin(&s_min, okey(__ldg(d.fit[d.cur] + 2 * m)));
            }
            if (mult * c < take) copy_survivor(d, m, q0, (mult == 2 && 2 * c + 1 < take) ? q0 + 1 : -1, lane);
        }
    }
    __syncthreads();
    if (t == 0) {
        if (s_min != 0xFFFFFFFFu) atomicMin(d.nfmin, s_min);
        __threadfence();
        if (atomicAdd(d.done, 1) == (int)gridDim.x - 1) {
            // +inf when no survivor's first objective is a number; then the minimum's reset
            const uint32_t k = atomicExch(d.nfmin, 0xFFFFFFFFu);
            const uint32_t g = d.gen + 1;
            if (d.history && (int)g < d.hist_cap)
                d.history[g] = (k == 0xFFFFFFFFu) ? INFINITY
                                                  : __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
            d.cur ^= 1;
            d.gen = g;
            d.advanced = 1;
            *d.done = 0;
            __threadfence();
        }
    }
}

// crowding and (mode 0) survivors from the ranks and orders above; one CTA per population
__global__ void __launch_bounds__(kNsgaBlock, 1) nsga_select_kernel(PopDesc* dd, int mode) {
    dep_wait();
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t wt32[32];
    __shared__ float redf[32];
    PopDesc& d = dd[blockIdx.x];
    if (!select_active(d, mode)) return;
    const int t = threadIdx.x;
    const int P = d.P;
    const int N = (mode == 0) ? 2 * P : P;
    const float* f = d.fit[d.cur];
    const SelSmem s = sel_carve(smem, N);
    staged<kNsgaBlock, 8>(2 * N, [&](int i) { return __ldg(f + i); }, [&](int i, float v) { s.obj[i] = v; });
    staged<kNsgaBlock, 4>(N, [&](int i) { return __ldg(d.domcnt + i); },
                          [&](int i, int v) { s.rank[i] = (uint16_t)v; });
    crowding_given<kNsgaBlock>(N, s, d.nord, 2 * P);
    float fmin = INFINITY;
    if (mode == 0) {
        select_given<kNsgaBlock>(N, P, s, d.nsel, d.nrank, d.ncd, &fmin, wt32);
    } else {
        for (int i = t; i < P; i += kNsgaBlock) {
            d.nrank[i] = s.rank[i];
            d.ncd[i] = s.cd[i];
            fmin = fminf(fmin, s.obj[2 * i]);
        }
    }
    fmin = block_min_f(fmin, redf);
    if (t == 0 && d.history) {
        const uint32_t g = (mode == 0) ? d.gen + 1 : d.gen;
        if ((int)g < d.hist_cap) d.history[g] = fmin;
    }
}

// ranks only (op API, any number of objectives): one CTA
__global__ void __launch_bounds__(kNsgaBlock) peel_op_kernel(int N, const uint32_t* S, const int32_t* cnt, int Wmax,
                                                             int32_t* rank) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t wt32[32];
    uint16_t* r16 = reinterpret_cast<uint16_t*>(smem);
    const PeelSmem ps = peel_carve(smem + (((size_t)N * 2 + 15) / 16) * 16, N);
    peel_ranks<kNsgaBlock>(N, S, Wmax, cnt, r16, ps, wt32);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += kNsgaBlock) rank[i] = r16[i];
}

// ensure_minimum_diversity (core/population.hpp:130-182) runs after generation g when
// (g - 1) % interval == 0 (the reference's counter is g - 1).
__device__ __forceinline__ bool div_due(const PopDesc& d) {
    return d.advanced && d.div_interval > 0 && d.gen >= 1u && ((d.gen - 1u) % (uint32_t)d.div_interval) == 0u;
}

// The reference keeps a point when no earlier KEPT point is within distance 0.001 in
// objective space (float differences, squared and summed in double).  near_build_kernel
// records, per point c, which earlier points u < c are that close (bit u of row c of the
// dominance scratch); nsga_diversity_kernel then settles keep / drop in rounds: c is
// dropped as soon as a kept point is near it, kept once every near earlier point is
// settled as dropped.  The result is the reference's greedy in-order pass.
constexpr int kNearWarps = 4, kNearRows = 4;

__global__ void __launch_bounds__(kNearWarps * 32) near_build_kernel(PopDesc* dd) {
    dep_wait();
    extern __shared__ float2 so[];  // [32 * ceil(P / 32)]
    const PopDesc& d = dd[blockIdx.y];
    if (!div_due(d)) return;
    const int P = d.P, W = (P + 31) / 32;
    const int row0 = blockIdx.x * kNearWarps * kNearRows;
    if (row0 >= P) return;
    const float2* o2 = reinterpret_cast<const float2*>(d.fit[d.cur]);
    for (int j = threadIdx.x; j < 32 * W; j += blockDim.x) so[j] = (j < P) ? o2[j] : make_float2(0.0f, 0.0f);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = 0; r < kNearRows; ++r) {
        const int c = row0 + warp * kNearRows + r;
        if (c >= P) break;
        const float2 pc = so[c];
        uint32_t* row = d.domS + (size_t)c * d.domW;
        for (int w = 0; w <= c / 32; ++w) {
            const int u = 32 * w + lane;
            bool near = false;
            if (u < c) {
                const float2 pu = so[u];
                const double d0 = (double)__fsub_rn(pc.x, pu.x);
                const double d1 = (double)__fsub_rn(pc.y, pu.y);
                near = __dsqrt_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1))) < 0.001;
            }
            const uint32_t bits = __ballot_sync(0xffffffffu, near);
            if (lane == 0) row[w] = bits;
        }
    }
}

// Settles the pass (one CTA per population).  When fewer than 70% are kept, the kept rows
// are gathered in order into the other key buffer, which becomes the current one, and
// *nu < P tells the refill and re-rank launches to run; otherwise *nu = P.
__global__ void __launch_bounds__(kNsgaBlock) nsga_diversity_kernel(PopDesc* dd) {
    dep_wait();
    constexpr int WP = kMaxPool / 2 / 32;
    __shared__ uint32_t U[WP], D[WP], Un[WP], Dn[WP];
    __shared__ uint32_t wt32[32];
    PopDesc& d = dd[blockIdx.x];
    const int t = threadIdx.x, P = d.P, W = (P + 31) / 32;
    if (!div_due(d)) {
        if (t == 0) *d.nu = P;
        return;
    }
    for (int w = t; w < W; w += kNsgaBlock) U[w] = D[w] = Un[w] = Dn[w] = 0u;
    __syncthreads();
    // every round settles at least the lowest unsettled point, so P rounds suffice
    for (int round = 0; round <= P; ++round) {
        int open = 0;
        for (int c = t; c < P; c += kNsgaBlock) {
            if ((D[c >> 5] >> (c & 31)) & 1u) continue;
            const uint32_t* row = d.domS + (size_t)c * d.domW;
            const int last = c >> 5;
            bool kept_near = false, unsettled = false;
            for (int w = 0; w <= last; ++w) {
                uint32_t nb = __ldg(row + w);
                if (w == last) nb &= (1u << (c & 31)) - 1u;
                kept_near |= (nb & U[w]) != 0u;
                unsettled |= (nb & ~D[w]) != 0u;
            }
            if (kept_near) {
                atomicOr(&Dn[c >> 5], 1u << (c & 31));
            } else if (!unsettled) {
                atomicOr(&Un[c >> 5], 1u << (c & 31));
                atomicOr(&Dn[c >> 5], 1u << (c & 31));
            } else {
                open = 1;
            }
        }
        __syncthreads();
        for (int w = t; w < W; w += kNsgaBlock) {
            U[w] |= Un[w];
            D[w] |= Dn[w];
        }
        if (!__syncthreads_or(open)) break;
    }
    // kept points in index order -> nsel[0, nu)
    const int pc = (t < W) ? __popc(U[t]) : 0;
    uint32_t nu = 0;
    uint32_t pos = block_exclusive_scan<kNsgaBlock>((uint32_t)pc, wt32, &nu);
    if (t < W)
        for (uint32_t x = U[t]; x; x &= x - 1) d.nsel[pos++] = 32 * t + __ffs(x) - 1;
    __syncthreads();
    const double ratio = (double)nu / (double)P;
    if (!(ratio < 0.70)) {
        if (t == 0) *d.nu = P;
        return;
    }
    // gather the kept rows, in order, into the other buffer and make it current
    const int cur = d.cur, ld4 = d.ld / 4;
    const float4* src = reinterpret_cast<const float4*>(d.keys[cur]);
    float4* dst = reinterpret_cast<float4*>(d.keys[cur ^ 1]);
    const float* fs = d.fit[cur];
    float* fd = d.fit[cur ^ 1];
    const size_t total = (size_t)nu * ld4;
    for (size_t x = t; x < total; x += kNsgaBlock) {
        const int q = (int)(x / ld4), col = (int)(x % ld4);
        dst[x] = src[(size_t)d.nsel[q] * ld4 + col];
    }
    for (int q = t; q < (int)nu; q += kNsgaBlock) {
        fd[2 * q] = fs[2 * d.nsel[q]];
        fd[2 * q + 1] = fs[2 * d.nsel[q] + 1];
    }
    __syncthreads();
    if (t == 0) {
        d.cur = cur ^ 1;
        *d.nu = (int)nu;
    }
}

// ---------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------
int nsga_max_population() { return kMaxPool / 2; }

size_t nsga_select_smem(int maxP) { return sel_smem_bytes(2 * maxP); }

cudaError_t nsga_prepare(int maxP) {
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(nsga_select_kernel), sel_smem_bytes(2 * maxP));
    if (e == cudaSuccess)
        e = raise_smem_limit(reinterpret_cast<const void*>(nsga_order_kernel), (size_t)2 * maxP * 8);
    if (e == cudaSuccess)
        e = raise_smem_limit(reinterpret_cast<const void*>(near_build_kernel), (size_t)((maxP + 31) / 32) * 32 * 8);
    if (e == cudaSuccess)
        e = raise_smem_limit(reinterpret_cast<const void*>(nsga_cut_kernel), (size_t)2 * maxP * 8);
    if (e == cudaSuccess)
        e = raise_smem_limit(reinterpret_cast<const void*>(nsga_front_crowd_kernel), (size_t)2 * maxP * sizeof(uint2));
    return e;
}

// two-objective dominance rows of up to maxN points per population (grid.y)
static cudaError_t launch_dom2(const DomArgs& a, int maxN, int npops, cudaStream_t st) {
    constexpr int RPC = kDom2Rows * kDom2RowWarps;
    const size_t smem = (size_t)((maxN + 31) / 32) * 32 * sizeof(float2);
    cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(dom2_build_kernel), smem);
    if (e != cudaSuccess) return e;
    return launch_dep(dom2_build_kernel, dim3((maxN + RPC - 1) / RPC, npops), dim3(kDom2Warps * 32), smem, st, a);
}

static cudaError_t launch_dom(PopDesc* dd, int npops, int maxN, int only_rebuilt, cudaStream_t st) {
    DomArgs a;
    std::memset(&a, 0, sizeof(a));
    a.dd = dd;
    a.only_rebuilt = only_rebuilt;
    a.dominators = 1;
    return launch_dom2(a, maxN, npops, st);
}

// ranks, crowding and (mode 0) survivors of every population of the group
cudaError_t nsga_enqueue_select(PopDesc* dd, int npops, int maxP, int mode, cudaStream_t st) {
    const int maxN = (mode == 0) ? 2 * maxP : maxP;
    cudaError_t e;
    if (mode == 0)
        e = launch_dep(dom2_pool_kernel, dim3(2 * device_sm_count(), npops), dim3(kSymWarps * 32), 0, st, dd);
    else
        e = launch_dom(dd, npops, maxN, mode == 2 ? 1 : 0, st);
    if (e != cudaSuccess) return e;
    e = launch_peel(dd, npops, maxN, mode, st);
    if (e != cudaSuccess) return e;
    if (mode == 0) {
        // a generation's pool: crowding and whole fronts from each point's own front, then
        // the cut front
        e = launch_dep(nsga_front_crowd_kernel, dim3((maxN + kFrontWarps - 1) / kFrontWarps, npops),
                       dim3(kFrontWarps * 32), (size_t)maxN * sizeof(uint2), st, dd);
        if (e != cudaSuccess) return e;
        // (a cut front is a small part of the pool: two CTAs an SM, that many completion counts)
        const int ctas = std::min((maxN + kFrontWarps - 1) / kFrontWarps, 2 * device_sm_count());
        return launch_dep(nsga_cut_kernel, dim3(ctas, npops), dim3(kFrontWarps * 32),
                          (size_t)maxN * 8, st, dd);
    }
    e = launch_dep(nsga_order_kernel, dim3((maxN + kOrdPerCta - 1) / kOrdPerCta, 2, npops), dim3(kOrdThreads),
                   (size_t)maxN * 8, st, dd, mode);
    if (e != cudaSuccess) return e;
    return launch_dep(nsga_select_kernel, dim3(npops), dim3(kNsgaBlock), sel_smem_bytes(maxN), st, dd, mode);
}

cudaError_t nsga_enqueue_diversity(PopDesc* dd, int npops, int maxP, cudaStream_t st) {
    constexpr int RPC = kNearWarps * kNearRows;
    const size_t smem = (size_t)((maxP + 31) / 32) * 32 * sizeof(float2);
    const cudaError_t e =
        launch_dep(near_build_kernel, dim3((maxP + RPC - 1) / RPC, npops), dim3(kNearWarps * 32), smem, st, dd);
    if (e != cudaSuccess) return e;
    return launch_dep(nsga_diversity_kernel, dim3(npops), dim3(kNsgaBlock), 0, st, dd);
}

int32_t nsga_alloc(PopDesc& d, int P, double mut_rate, int div_interval, int Mn, std::vector<void*>& allocs,
                   size_t* bytes, cudaStream_t stream) {
    const int N = 2 * P;
    const int W = round_up((N + 31) / 32, 4);  // dominance rows of whole 16-byte words
    auto get = [&](size_t b, void** p) -> int32_t {
        int32_t rc = dev_alloc(p, b ? b : 16, stream);
        if (rc != BRKGA_OK) return rc;
        allocs.push_back(*p);
        *bytes += b;
        return BRKGA_OK;
    };
    void* p = nullptr;
    int32_t st;
    if ((st = get((size_t)N * 4, &p)) != BRKGA_OK) return st;
    d.nrank = (int32_t*)p;
    if ((st = get((size_t)N * 4, &p)) != BRKGA_OK) return st;
    d.ncd = (float*)p;
    if ((st = get((size_t)P * 4, &p)) != BRKGA_OK) return st;
    d.nsel = (int32_t*)p;
    if ((st = get((size_t)N * W * 4, &p)) != BRKGA_OK) return st;
    d.domS = (uint32_t*)p;
    if ((st = get((size_t)N * 4, &p)) != BRKGA_OK) return st;
    d.domcnt = (int32_t*)p;
    if ((st = get(16, &p)) != BRKGA_OK) return st;
    d.nu = (int32_t*)p;
    if ((st = get((size_t)2 * N * 4, &p)) != BRKGA_OK) return st;
    d.nord = (int32_t*)p;
    if ((st = get((size_t)(N + 4) * 4, &p)) != BRKGA_OK) return st;
    d.nft = (int32_t*)p;
    if ((st = get((size_t)N * 4, &p)) != BRKGA_OK) return st;
    d.ncdp = (float*)p;
    if ((st = get((size_t)N * 4, &p)) != BRKGA_OK) return st;
    d.nlist = (int32_t*)p;
    if ((st = get(16, &p)) != BRKGA_OK) return st;
    d.nfmin = (uint32_t*)p;
    if (cudaMemsetAsync(d.nfmin, 0xFF, 4, stream) != cudaSuccess) {
        cudaGetLastError();
        return fail(BRKGA_ERR_CUDA, "NSGA-II state initialisation");
    }
    d.domW = W;
    d.Mn = Mn;
    d.mutT = prob_threshold(mut_rate);
    d.div_interval = div_interval;
    return BRKGA_OK;
}

int32_t nsga_setup(NsgaState& s, Population& pop, PopDesc* dd, PopDesc& hdesc, const RowTile& tile, int grid,
                   int groups_per_cta, bool stage) {
    s.dd = dd;
    s.P = pop.sh.Pi;
    s.N = 2 * pop.sh.Pi;
    if (s.P > nsga_max_population())
        return fail(BRKGA_ERR_UNSUPPORTED, "NSGA-II population above " + std::to_string(nsga_max_population()));
    s.n = pop.sh.n;
    s.ld = pop.sh.ld;
    s.kind = pop.pd->kind;
    s.max_points = points_of(*pop.pd);
    s.tile = tile;
    s.grid = grid;
    s.groups_per_cta = groups_per_cta;
    s.stage = stage;
    const double rate = (pop.prm.mutation_rate > 0.0) ? pop.prm.mutation_rate : 5.0 / (double)pop.sh.n;
    int32_t st = nsga_alloc(hdesc, s.P, rate, pop.prm.diversity_interval, pop.sh.Mn, pop.allocs, &pop.bytes,
                            pop.stream);
    if (st != BRKGA_OK) return st;
    s.div_interval = pop.prm.diversity_interval;
    cudaError_t e = cudaStreamSynchronize(pop.stream);
    if (e == cudaSuccess) e = cudaMemcpy(dd, &hdesc, sizeof(PopDesc), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "descriptor upload");
    e = nsga_prepare(s.P);
    if (e != cudaSuccess) return cuda_fail(e, "NSGA-II set-up");
    s.ready = true;
    return BRKGA_OK;
}

void nsga_release(NsgaState& s) { s.ready = false; }

void nsga_set_history(NsgaState& s, float* h, int cap) {
    s.history = h;
    s.hist_cap = cap;
}

static RowLaunch nsga_rows(const NsgaState& s, int mode) {
    RowLaunch L;
    std::memset(&L, 0, sizeof(L));
    L.descs = s.dd;
    L.mode = mode;
    L.ntasks = s.P;
    L.max_n = s.n;
    L.max_points = s.max_points;
    L.stage_xy = s.stage ? 1 : 0;
    L.groups_per_cta = s.groups_per_cta;
    L.gscratch = s.gscratch;
    L.gstride = s.gstride;
    return L;
}

cudaError_t nsga_enqueue_rows(NsgaState& s, int mode, cudaStream_t st) {
    return launch_rows(nsga_rows(s, mode), s.kind, s.tile, s.grid, st);
}

cudaError_t nsga_enqueue_init(NsgaState& s, cudaStream_t st) {
    cudaError_t e = launch_rows(nsga_rows(s, MODE_INIT), s.kind, s.tile, s.grid, st);
    if (e != cudaSuccess) return e;
    return nsga_enqueue_select(s.dd, 1, s.P, 1, st);
}

bool nsga_diversity_due(const NsgaState& s, uint32_t g) {
    return s.div_interval > 0 && g >= 1u && ((g - 1u) % (uint32_t)s.div_interval) == 0u;
}

cudaError_t nsga_enqueue_generation(NsgaState& s, cudaStream_t st, bool with_diversity) {
    // offspring into pool rows [P, 2P) (core/solver.hpp:1019-1032) + their objectives
    cudaError_t e = launch_rows(nsga_rows(s, MODE_NSGA_OFF), s.kind, s.tile, s.grid, st);
    if (e != cudaSuccess) return e;
    // ranks, crowding and survivors of the pool (core/population.hpp:409-517), the
    // survivors' rows into the other buffer and the buffer swap
    if ((e = nsga_enqueue_select(s.dd, 1, s.P, 0, st)) != cudaSuccess) return e;
    if (with_diversity && s.div_interval > 0) {
        // decided on the device: due this generation, and fewer than 70% unique
        if ((e = nsga_enqueue_diversity(s.dd, 1, s.P, st)) != cudaSuccess) return e;
        if ((e = launch_rows(nsga_rows(s, MODE_NSGA_REFILL), s.kind, s.tile, s.grid, st)) != cudaSuccess) return e;
        e = nsga_enqueue_select(s.dd, 1, s.P, 2, st);
    }
    return e;
}

static int32_t read_desc(NsgaState& s, cudaStream_t st, PopDesc* d) {
    cudaError_t e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaMemcpy(d, s.dd, sizeof(PopDesc), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "descriptor read-back");
    if (d->stuck) return fail(BRKGA_ERR_TIMEOUT, "a wait between the launch's CTAs ran out; the population is not valid");
    return BRKGA_OK;
}

int32_t nsga_get_population(NsgaState& s, cudaStream_t st, float* keys, float* obj) {
    PopDesc d;
    int32_t rc = read_desc(s, st, &d);
    if (rc != BRKGA_OK) return rc;
    std::vector<float> hk((size_t)s.P * s.ld);
    cudaError_t e = cudaMemcpy(hk.data(), d.keys[d.cur], hk.size() * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && obj) e = cudaMemcpy(obj, d.fit[d.cur], (size_t)s.P * 2 * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "population read-back");
    if (keys)
        for (int r = 0; r < s.P; ++r) std::memcpy(keys + (size_t)r * s.n, hk.data() + (size_t)r * s.ld, (size_t)s.n * 4);
    return BRKGA_OK;
}

int32_t nsga_set_population(NsgaState& s, cudaStream_t st, const float* keys) {
    PopDesc d;
    int32_t rc = read_desc(s, st, &d);
    if (rc != BRKGA_OK) return rc;
    std::vector<float> hk((size_t)s.P * s.ld, 0.0f);
    for (int r = 0; r < s.P; ++r) std::memcpy(hk.data() + (size_t)r * s.ld, keys + (size_t)r * s.n, (size_t)s.n * 4);
    cudaError_t e = cudaMemcpy(d.keys[d.cur], hk.data(), hk.size() * 4, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_fail(e, "population upload");
    e = launch_rows(nsga_rows(s, MODE_EVAL), s.kind, s.tile, s.grid, st);
    if (e == cudaSuccess) e = nsga_enqueue_select(s.dd, 1, s.P, 1, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(e, "population evaluate");
    return BRKGA_OK;
}

// best = the first-front member with the largest crowding distance (update_best_from_front,
// core/population.hpp:684-698), the first such index on ties
int32_t nsga_get_best(NsgaState& s, cudaStream_t st, float* keys, int32_t* perm, float* obj) {
    PopDesc d;
    int32_t rc = read_desc(s, st, &d);
    if (rc != BRKGA_OK) return rc;
    std::vector<int32_t> hr(s.P);
    std::vector<float> hc(s.P), ho((size_t)s.P * 2);
    cudaMemcpy(hr.data(), d.nrank, (size_t)s.P * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(hc.data(), d.ncd, (size_t)s.P * 4, cudaMemcpyDeviceToHost);
    cudaError_t e = cudaMemcpy(ho.data(), d.fit[d.cur], ho.size() * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "best read-back");
    int best = -1;
    for (int i = 0; i < s.P; ++i)
        if (hr[i] == 0 && (best < 0 || hc[i] > hc[best])) best = i;
    if (best < 0) best = 0;
    if (obj) {
        obj[0] = ho[2 * best];
        obj[1] = ho[2 * best + 1];
    }
    const float* row = d.keys[d.cur] + (size_t)best * s.ld;
    if (keys) {
        e = cudaMemcpy(keys, row, (size_t)s.n * 4, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return cuda_fail(e, "best keys");
    }
    if (perm) {
        // decode on the device with the row kernel (same argsort as the generation step)
        float* tmpf = nullptr;
        int32_t* tmpp = nullptr;
        if (dev_alloc((void**)&tmpf, 16, st) != BRKGA_OK || dev_alloc((void**)&tmpp, (size_t)s.n * 4, st) != BRKGA_OK) {
            dev_free(tmpf, st);
            return fail(BRKGA_ERR_OOM, "decode scratch");
        }
        RowLaunch L;
        std::memset(&L, 0, sizeof(L));
        L.single = d;
        L.single.keys[0] = const_cast<float*>(row);
        L.single.fit[0] = tmpf;
        L.single.cur = 0;
        L.ntasks = 1;
        L.mode = MODE_EVAL;
        L.perm_out = tmpp;
        L.max_n = s.n;
        L.max_points = s.max_points;
        L.stage_xy = s.stage ? 1 : 0;
        L.gscratch = s.gscratch;
        L.gstride = s.gstride;
        e = launch_rows(L, s.kind, s.tile, 1, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = cudaMemcpy(perm, tmpp, (size_t)s.n * 4, cudaMemcpyDeviceToHost);
        dev_free(tmpf, st);
        dev_free(tmpp, st);
        if (e != cudaSuccess) return cuda_fail(e, "best decode");
    }
    return BRKGA_OK;
}

int32_t nsga_get_front(NsgaState& s, cudaStream_t st, float* obj, float* keys, int32_t cap, int32_t* count) {
    PopDesc d;
    int32_t rc = read_desc(s, st, &d);
    if (rc != BRKGA_OK) return rc;
    std::vector<int32_t> hr(s.P);
    std::vector<float> ho((size_t)s.P * 2), hk((size_t)s.P * s.ld);
    cudaMemcpy(hr.data(), d.nrank, (size_t)s.P * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(ho.data(), d.fit[d.cur], ho.size() * 4, cudaMemcpyDeviceToHost);
    cudaError_t e = cudaMemcpy(hk.data(), d.keys[d.cur], hk.size() * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "front read-back");
    int c = 0;
    for (int i = 0; i < s.P; ++i) {
        if (hr[i] != 0) continue;
        if (c < cap) {
            if (obj) {
                obj[2 * c] = ho[2 * i];
                obj[2 * c + 1] = ho[2 * i + 1];
            }
            if (keys) std::memcpy(keys + (size_t)c * s.n, hk.data() + (size_t)i * s.ld, (size_t)s.n * 4);
        }
        ++c;
    }
    *count = c;
    return BRKGA_OK;
}

// ---------------------------------------------------------------------------------------
// Pareto ranks for callers that cannot allocate device memory.  The dominance rows and
// counts live in a file-scope device array of fixed size (every GPU that loads the
// library holds it until the process exits); host code finds its device address with
// cudaGetSymbolAddress once per device, with that device current.
// ---------------------------------------------------------------------------------------
constexpr int kStaticMaxN = 2048;                       // largest point count it accepts
constexpr int kStaticW = (kStaticMaxN + 31) / 32;       // dominance row words
constexpr size_t kStaticWords = (size_t)kStaticMaxN * kStaticW + kStaticMaxN;  // rows + counts (532 KiB)
static __device__ __align__(256) uint32_t g_static_scratch[kStaticWords];

static std::mutex g_static_mu;
static std::map<int, uint32_t*> g_static_addr;  // device -> address of g_static_scratch

// per-device set-up on first use: the array's device address and the peel kernel's
// shared-memory limit (neither allocates device memory)
static int32_t static_scratch(uint32_t** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    std::lock_guard<std::mutex> lk(g_static_mu);
    auto it = g_static_addr.find(dev);
    if (it != g_static_addr.end()) {
        *out = it->second;
        return BRKGA_OK;
    }
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress (static scratch)");
    const size_t smem = (((size_t)kStaticMaxN * 2 + 15) / 16) * 16 + peel_smem_bytes(kStaticMaxN);
    e = raise_smem_limit(reinterpret_cast<const void*>(peel_op_kernel), smem);
    if (e != cudaSuccess) return cuda_fail(e, "peel set-up");
    g_static_addr[dev] = (uint32_t*)ptr;
    *out = (uint32_t*)ptr;
    return BRKGA_OK;
}

// scratch of the operator entry points (grow-only, per device)
static std::mutex g_op_mu;
static std::map<int, std::pair<void*, size_t>> g_op_buf;
static int32_t* g_op_stuck = nullptr;  // a wait in an operator's kernel ran out

static int32_t op_scratch(size_t need, void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (!g_op_stuck) {
        const int32_t st = flag_take(&g_op_stuck);
        if (st != BRKGA_OK) return st;
    }
    auto& b = g_op_buf[dev];
    if (b.second < need) {
        if (b.first) {
            cudaDeviceSynchronize();
            cudaFree(b.first);
        }
        b = {nullptr, 0};
        if ((e = cudaMalloc(&b.first, need)) != cudaSuccess) {
            b.first = nullptr;
            cudaGetLastError();  // a failed allocation must not surface as a later launch's error
            return fail(BRKGA_ERR_OOM, std::string("operator scratch: ") + cudaGetErrorString(e));
        }
        b.second = need;
    }
    *out = b.first;
    return BRKGA_OK;
}

}  // namespace bk

using namespace bk;

extern "C" {

int32_t brkga_pareto_rank_bitmatrix(const float* d_obj, int32_t N, int32_t m, int32_t* d_rank, void* stream) {
    if (!d_obj || !d_rank) return fail(BRKGA_ERR_INVALID, "null argument");
    if (N < 0 || m < 1 || m > 4) return fail(BRKGA_ERR_INVALID, "need N >= 0 and 1 <= m <= 4");
    if (N == 0) return BRKGA_OK;
    if (N > 8192) return fail(BRKGA_ERR_UNSUPPORTED, "more than 8192 points");
    cudaStream_t st = (cudaStream_t)stream;
    const bool rows = N <= kMaxPool;  // ranks by the engine's row peel; larger sets by one CTA's column peel
    const int W = rows ? round_up((N + 31) / 32, 4) : (N + 31) / 32;
    const size_t sbytes = (size_t)N * W * 4, cbytes = (size_t)N * 4;
    const size_t doff = ((sbytes + cbytes + 255) / 256) * 256;  // a descriptor for the cluster peel
    std::lock_guard<std::mutex> lk(g_op_mu);
    void* buf = nullptr;
    int32_t rc = op_scratch(doff + sizeof(PopDesc), &buf);
    if (rc != BRKGA_OK) return rc;
    DomArgs a;
    std::memset(&a, 0, sizeof(a));
    a.obj = d_obj;
    a.rawN = N;
    a.m = m;
    a.S = (uint32_t*)buf;
    a.cnt = (int32_t*)((char*)buf + sbytes);
    a.Wmax = W;
    a.dominators = rows ? 1 : 0;
    if (rows) a.cnt = nullptr;
    cudaError_t e;
    if (m == 2) {
        e = launch_dom2(a, N, 1, st);
    } else {
        dom_build_kernel<<<(N + 7) / 8, 256, 0, st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return cuda_fail(e, "dominance launch");
    if (rows) {
        // as for a population of N rows in mode 1, the ranks straight into the caller's buffer
        PopDesc hd;
        std::memset(&hd, 0, sizeof(hd));
        hd.P = N;
        hd.m = m;
        hd.domS = a.S;
        hd.domW = W;
        hd.domcnt = d_rank;
        hd.stuck_host = g_op_stuck;
        hd.wait_polls = wait_polls();
        PopDesc* dd = reinterpret_cast<PopDesc*>((char*)buf + doff);
        if ((e = cudaMemcpyAsync(dd, &hd, sizeof(hd), cudaMemcpyHostToDevice, st)) != cudaSuccess)
            return cuda_fail(e, "peel descriptor");
        if ((e = launch_peel(dd, 1, N, 1, st)) != cudaSuccess) return cuda_fail(e, "peel launch");
    } else {
        const size_t smem = (((size_t)N * 2 + 15) / 16) * 16 + peel_smem_bytes(N);
        if ((e = raise_smem_limit(reinterpret_cast<const void*>(peel_op_kernel), smem)) != cudaSuccess)
            return cuda_fail(e, "peel set-up");
        peel_op_kernel<<<1, kNsgaBlock, smem, st>>>(N, a.S, a.cnt, W, d_rank);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "peel launch");
    }
    // the scratch is shared by later calls: finish before returning
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(e, "peel");
    if (flag_set(g_op_stuck)) {
        *g_op_stuck = 0;
        return fail(BRKGA_ERR_TIMEOUT, "a wait between the peel's CTAs ran out; the ranks are not valid");
    }
    return BRKGA_OK;
}

int32_t brkga_pareto_rank_noalloc(const float* d_obj, int32_t N, int32_t m, int32_t* d_rank, void* stream) {
    if (!d_obj || !d_rank) return fail(BRKGA_ERR_INVALID, "null argument");
    if (N < 0 || m < 1 || m > 4) return fail(BRKGA_ERR_INVALID, "need N >= 0 and 1 <= m <= 4");
    if (N > kStaticMaxN)
        return fail(BRKGA_ERR_UNSUPPORTED, "brkga_pareto_rank_noalloc takes at most " + std::to_string(kStaticMaxN) +
                                               " points (got " + std::to_string(N) + "); use brkga_pareto_rank");
    if (N == 0) return BRKGA_OK;
    uint32_t* base = nullptr;
    int32_t rc = static_scratch(&base);
    if (rc != BRKGA_OK) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const int W = (N + 31) / 32;
    DomArgs a;
    std::memset(&a, 0, sizeof(a));
    a.obj = d_obj;
    a.rawN = N;
    a.m = m;
    a.S = base;                                        // rows [N][W]: every word is written
    a.cnt = (int32_t*)(base + (size_t)kStaticMaxN * kStaticW);  // counts [N]: every entry is written
    a.Wmax = W;
    dom_build_kernel<<<(N + 7) / 8, 256, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "dominance launch");
    const size_t smem = (((size_t)N * 2 + 15) / 16) * 16 + peel_smem_bytes(N);
    peel_op_kernel<<<1, kNsgaBlock, smem, st>>>(N, a.S, a.cnt, W, d_rank);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "peel launch");
    return BRKGA_OK;
}

int32_t brkga_pareto_rank(const float* d_obj, int32_t N, int32_t m, int32_t* d_rank, void* stream) {
    return brkga_pareto_rank_bitmatrix(d_obj, N, m, d_rank, stream);
}

int32_t brkga_crowding(const float* d_obj, const int32_t* d_rank, int32_t N, int32_t m, float* d_cd, void* stream) {
    if (!d_obj || !d_rank || !d_cd) return fail(BRKGA_ERR_INVALID, "null argument");
    if (m != 2) return fail(BRKGA_ERR_UNSUPPORTED, "crowding kernel handles two objectives");
    if (N < 0 || N > kMaxPool) return fail(BRKGA_ERR_UNSUPPORTED, "N outside [0, 4096]");
    if (N == 0) return BRKGA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    // the engine's crowding: orders by (rank, objective, index) on the grid, then the crowding
    // over them, as for a population of N points in mode 1; scratch from the stream-ordered
    // pool (orders [2][2N], ranks [N], the descriptor), returned behind the launches
    const size_t doff = (((size_t)5 * N * 4 + 255) / 256) * 256;
    void* p = nullptr;
    int32_t rc = dev_alloc(&p, doff + sizeof(PopDesc), st);
    if (rc != BRKGA_OK) return rc;
    PopDesc hd;
    std::memset(&hd, 0, sizeof(hd));
    hd.P = N;
    hd.m = 2;
    hd.fit[0] = const_cast<float*>(d_obj);
    hd.domcnt = const_cast<int32_t*>(d_rank);
    hd.nord = static_cast<int32_t*>(p);
    hd.nrank = static_cast<int32_t*>(p) + 4 * (size_t)N;
    hd.ncd = d_cd;
    PopDesc* dd = reinterpret_cast<PopDesc*>(static_cast<char*>(p) + doff);
    cudaError_t e = nsga_prepare((N + 1) / 2);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dd, &hd, sizeof(hd), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        nsga_order_kernel<<<dim3((N + kOrdPerCta - 1) / kOrdPerCta, 2, 1), kOrdThreads, (size_t)N * 8, st>>>(dd, 1);
        nsga_select_kernel<<<1, kNsgaBlock, sel_smem_bytes(N), st>>>(dd, 1);
        e = cudaGetLastError();
    }
    dev_free(p, st);
    if (e != cudaSuccess) return cuda_fail(e, "crowding launch");
    return BRKGA_OK;
}

}  // extern "C"
