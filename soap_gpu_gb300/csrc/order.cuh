// Order of a grid's cells by a key, for grids of at most ORDER_MAX cells: sorted tiles and
// counted ranks.
//
// A radix sort of some 10^4 keys is ten passes of a few microseconds of work and several
// launches each: latency.  Here a block sorts a tile of ORDER_TILE keys, then a block per
// (tile, other tile) counts, for every key of the one, the other's keys below it: a key's
// rank is the sum of its counts (integer atomics, so the order does not depend on their
// sequence), and the cell goes to that position.  Keys are unique (the cell is their last part).  The counting
// grows with the square of the cells, which sets ORDER_MAX (two radix sorts of the slope and
// the bin: 132, 157, 162, 160 and 175 us for grids of 100, 200, 300, 362 and 500 squared;
// this: 42, 44, 72, 107 and 295 us).
#pragma once
#include "internal.cuh"

constexpr int ORDER_TILE = 2048;
constexpr int ORDER_THREADS = 1024;
constexpr int ORDER_COUNT_THREADS = 256;
constexpr long long ORDER_MAX = 1LL << 17;

// (hi, lo) in lexicographic order; the cell in lo's low 32 bits
struct OrderKey {
    unsigned long long hi, lo;
};

__device__ __forceinline__ bool order_less(unsigned long long ah, unsigned long long al, unsigned long long bh,
                                           unsigned long long bl) {
    return ah < bh || (ah == bh && al < bl);
}

// A warp's 64 keys sorted (bitonic): lane l holds keys l and 32 + l
__device__ __forceinline__ void order_sort64(unsigned long long (&k)[2], int lane) {
#pragma unroll
    for (int lk = 1; lk <= 6; ++lk) {
#pragma unroll
        for (int lj = lk - 1; lj >= 0; --lj) {
            if (lj == 5) {
                const unsigned long long a = k[0], b = k[1];
                k[0] = min(a, b);
                k[1] = max(a, b);
                continue;
            }
            const int j = 1 << lj;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, k[q], j);
                const bool up = (((32 * q + lane) >> lk) & 1) == 0;
                k[q] = (((lane & j) == 0) == up) ? min(k[q], o) : max(k[q], o);
            }
        }
    }
}

// A warp sorts its 64 keys in registers (as order_sort64), then runs
// of 64, 128 ... keys are merged: a key's place is its place in its run plus the count of the
// sibling run's keys below it, found by binary search.
template <typename Key>
__global__ void __launch_bounds__(ORDER_THREADS) k_order_tiles(int gm, Key key, unsigned long long *hi,
                                                               unsigned long long *lo, int *rank) {
    static_assert(ORDER_TILE == 2 * ORDER_THREADS, "two keys per thread");
    __shared__ unsigned long long sh[ORDER_TILE], sl[ORDER_TILE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = blockIdx.x * ORDER_TILE, cnt = min(ORDER_TILE, gm - base);
    unsigned long long kh[2], kl[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int i = 64 * warp + 32 * q + lane;
        OrderKey k{~0ULL, ~0ULL};   // padding sorts last
        if (i < cnt) k = key(base + i);
        kh[q] = k.hi;
        kl[q] = k.lo;
    }
#pragma unroll
    for (int lk = 1; lk <= 6; ++lk) {
#pragma unroll
        for (int lj = lk - 1; lj >= 0; --lj) {
            if (lj == 5) {   // the thread's own pair, ascending
                if (order_less(kh[1], kl[1], kh[0], kl[0])) {
                    const unsigned long long th = kh[0], tl = kl[0];
                    kh[0] = kh[1];
                    kl[0] = kl[1];
                    kh[1] = th;
                    kl[1] = tl;
                }
                continue;
            }
            const int j = 1 << lj;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned long long oh = __shfl_xor_sync(0xffffffffu, kh[q], j);
                const unsigned long long ol = __shfl_xor_sync(0xffffffffu, kl[q], j);
                const bool up = (((32 * q + lane) >> lk) & 1) == 0;   // this key's run ascends
                const bool keep_min = ((lane & j) == 0) == up;
                if (order_less(oh, ol, kh[q], kl[q]) == keep_min) {
                    kh[q] = oh;
                    kl[q] = ol;
                }
            }
        }
    }
    int p[2] = {64 * warp + lane, 64 * warp + 32 + lane};
    for (int run = 64;; run <<= 1) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            sh[p[q]] = kh[q];
            sl[p[q]] = kl[q];
        }
        __syncthreads();
        if (run == ORDER_TILE) break;
        // the sibling run's keys below each of the thread's
        int a[2], s0[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            s0[q] = (p[q] & ~(run - 1)) ^ run;
            a[q] = s0[q];
        }
        for (int w = run >> 1; w > 0; w >>= 1) {   // counts of 0 .. run - 1 keys
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (order_less(sh[a[q] + w - 1], sl[a[q] + w - 1], kh[q], kl[q])) a[q] += w;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (order_less(sh[a[q]], sl[a[q]], kh[q], kl[q])) a[q] += 1;
            p[q] = (p[q] & ~run) + (a[q] - s0[q]);   // both runs begin at p's place in the pair
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < ORDER_TILE / ORDER_THREADS; ++q) {
        const int i = tid + q * ORDER_THREADS;
        if (i >= cnt) continue;
        hi[base + i] = sh[i];
        lo[base + i] = sl[i];
        rank[base + i] = i;
    }
}

static __global__ void __launch_bounds__(ORDER_COUNT_THREADS) k_order_ranks(int gm,
                                                                            const unsigned long long *__restrict__ hi,
                                                                            const unsigned long long *__restrict__ lo,
                                                                            int *rank) {
    constexpr int PER = ORDER_TILE / ORDER_COUNT_THREADS;
    if (blockIdx.x == blockIdx.y) return;   // a tile's own keys: counted by its sort
    __shared__ unsigned long long sh[ORDER_TILE];
    const int tid = threadIdx.x;
    const int tb = blockIdx.x * ORDER_TILE, nt = min(ORDER_TILE, gm - tb);
    const int cb = blockIdx.y * ORDER_TILE, nc = min(ORDER_TILE, gm - cb);
    for (int i = tid; i < nt; i += ORDER_COUNT_THREADS) sh[i] = hi[tb + i];
    unsigned long long k[PER];
    int a[PER], b[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int i = tid + q * ORDER_COUNT_THREADS;
        k[q] = (i < nc) ? hi[cb + i] : 0ULL;
        a[q] = 0;
        b[q] = (i < nc) ? nt : 0;   // nothing to search past the last key
    }
    __syncthreads();
    // the searches of a thread's keys in lock-step, so that their loads overlap
#pragma unroll 1
    for (int w = ORDER_TILE; w > 0; w >>= 1) {
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (a[q] >= b[q]) continue;
            const int m = (a[q] + b[q]) >> 1;
            const unsigned long long v = sh[m];
            const bool less = v < k[q] || (v == k[q] && lo[tb + m] < lo[cb + tid + q * ORDER_COUNT_THREADS]);
            if (less) a[q] = m + 1;
            else b[q] = m;
        }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int i = tid + q * ORDER_COUNT_THREADS;
        if (i < nc) atomicAdd(&rank[cb + i], a[q]);
    }
}

static __global__ void k_order_scatter(int gm, const unsigned long long *__restrict__ lo,
                                       const int *__restrict__ rank, int *order) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < gm) order[rank[i]] = (int)(unsigned)lo[i];
}

namespace soapgb {

// order[r] = the cell of rank r (gm <= ORDER_MAX); hi, lo, rank: work arrays of gm each
template <typename Key>
int order_cells(soapgb_ctx *ctx, long long gm, Key key, unsigned long long *hi, unsigned long long *lo, int *rank,
                int *order) {
    const int nt = (int)((gm + ORDER_TILE - 1) / ORDER_TILE);
    TraceScope ts(ctx, "cell_order");
    k_order_tiles<Key><<<nt, ORDER_THREADS, 0, ctx->stream>>>((int)gm, key, hi, lo, rank);
    SOAP_LAUNCHED(ctx);
    if (nt > 1) {
        k_order_ranks<<<dim3(nt, nt), ORDER_COUNT_THREADS, 0, ctx->stream>>>((int)gm, hi, lo, rank);
        SOAP_LAUNCHED(ctx);
    }
    k_order_scatter<<<(unsigned)((gm + 255) / 256), 256, 0, ctx->stream>>>((int)gm, lo, rank, order);
    SOAP_LAUNCHED(ctx);
    return SOAPGB_OK;
}

}  // namespace soapgb
