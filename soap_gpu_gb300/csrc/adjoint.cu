// Adjoint of the PLAIN64 integration (no counterpart in the reference, which has no gradient
// path).  The outputs are linear in every cube row and in every cell's limb value L:
//   flux += s - I q,  bconv += q - a,  tot += s - I a,   q, s, a = L lerp(row)
// with lerp(row)[j] = row[o] + (row[o+1] - row[o]) w at the owner o of j and
//   w = (l_j - l'_o) / (l'_{o+1} - l'_o) = ((l_j - l_o) / S - l_o f / S) inv[o],
// S = 1 + f = sqrt((1 + b) / (1 - b)), b = delta 1000 / c, inv[o] = 1 / (l_{o+1} - l_o).  With
// alpha = (l_j - l_o) inv[o] and beta = l_o inv[o], which depend on the pixel only,
//   w = alpha / S - beta f / S          dw/ddelta = -(alpha + beta) K,  K = (1000/c) / (S^3 (1-b)^2).
// Given gF, gB, gT (gradients of a scalar w.r.t. flux, bconv, tot), the gradients are
//   rows: source pixel o collects (1 - w) h, source o + 1 collects w h, times L, from the pixels
//     that o owns; h is gF + gT for q_sed, gB - I gF for q_norm, -gB - I gT for spot / facula rows;
//   continuum rows: I = ratio x sed[j], so d/dsed[j] = sum over cells of ratio (-q gF - a gT);
//   limb and velocity, per cell: the sum over j of (its unit-L values) . h and of their
//     derivatives in w times dw/ddelta.
// The spots share I, the faculae's I is (1 + LB) x the row, so for all cells of one row and class
// that have the same owner offset over a tile of pixels each of these sums needs only a few sums over
// the cells, and the limb gradients of the cells only three sums over the tile's pixels.  With f0 a
// shift of the range (its first cell's),
//   sum L w = inv[o] ((l_j - l_o - l_o f0) sum L / S  -  l_o sum (L / S) (f - f0)),
// in which every term is of the size of a weight: in sums of L f / S itself the offset, up to tens of
// pixels, cancels, and differences of prefix sums over a row carry the whole row's rounding (1e-13 of
// a range's weight; summed per tile and centred it is the rounding of single cells, 2e-16).  Cells of
// a row sorted by f have their offsets in ascending ranges, which a tile finds by binary search.
// Cells whose offset changes inside the tile (|v|/c x tile pixels of them) and cells with a Planck
// ratio are evaluated one by one.  Every sum runs in a fixed order, without atomics.
//
// A pixel, cell and phase took about 150 FP64 instructions on a pipe that issues two lanes per
// cycle; a pixel and range of cells takes 20 to 40.
#include <algorithm>
#include <cmath>

#include "internal.cuh"
#include "fir.cuh"
#include "order.cuh"
#include "planck.cuh"

using namespace soapgb;

constexpr int ADJ_MAX_MU = 256;      // mu rows
constexpr int ADJ_THREADS = 256;
constexpr int ADJ_SRC = ADJ_THREADS / 32 * 31;   // source pixels per block of the row gradients
constexpr int ADJ_NB = 64;           // integer boundaries handled at a time
constexpr double ADJ_F_MAX = 0.01;   // largest |f| of the cells taken in ranges (3000 km/s)
constexpr int ADJ_FRAC = 21;         // fraction bits of l u
// Scratch of the lists and of the limb kernel's shares of the pixels: 68 + 16 Q bytes per cell and phase.
// Phases beyond it are taken in groups, whose gradients add up in the phases' order.
constexpr size_t ADJ_SCRATCH = 4ULL << 30;
constexpr int ADJ_CLASS = 3;         // 0 spot, 1 facula, 2 evaluated one by one (Planck ratio, extreme velocity)

struct AdjGeo {
    double f, off, iS, a;   // S - 1, f lambda0 / step, 1 / S, L / S
    double K, L, sig;       // velocity factor, limb, 1 + LB
    double still;           // 1 for v == 0
};
// an entry's weights for the sums over a range
struct AdjEnt {
    double L, a, sig;       // as AdjGeo
};
// for the rounding of the forward's shifted wavelengths (see adj_residue)
struct AdjNoise {
    unsigned long long w;   // |1 - S| 2^(53 + ADJ_FRAC)
    int a, as;              // L / S, negative for S > 1, and (1 + LB) times it, in units of AdjRow's
};
// a row of a class
struct AdjRow {
    int2 zero;              // its entries with f == 0
    double s0, t0;          // their sums of L and (1 + LB) L
    double still0, still1;  // those with v == 0 alone
    double unit, unit_s;    // of AdjNoise's a, as, times 2^-ADJ_FRAC
    int even;               // the weights but zero lie within 2^13: 2^-31 of the largest, of half an
                            // ulp, is then below a weight's rounding
};
// sums over a range's cells, f0 its first cell's f: of L, L / S, (L / S) (f - f0), and with (1 + LB) L
struct AdjSums {
    double f0, s0, s1, s2, t0, t1, t2;
    int zone;               // of adj_residue; 0: an |f| beyond ADJ_W_MAX
};

struct AdjArgs {
    int n, n_eff, n_mu, n_phase, Q;
    long long gm;
    const double *lam, *inv;
    const double *q_norm, *q_sed, *spot_norm, *fac_norm, *spot_sed, *fac_sed;
    const double *temp, *lb;
    double step;
    int solar, t_norm_fac;
    const double *gF, *gB, *gT;
    const AdjGeo *geo;
    // per phase gm entries: the active cells by class, row, f
    const int *cell;
    const double *fb;
    const AdjEnt *ent;
    const AdjNoise *noise;
    const int *seg;     // [phase][class][n_mu + 1] first entry of each row
    const AdjRow *row;  // [phase][2][n_mu]
    int more;           // the outputs hold the sums of the phases before
    double *acc;        // [Q][phase][gm][2] limb and velocity sums per entry
    double *part;       // [n_mu][2][n] continuum sums per row
    double *d_qn, *d_qs, *d_sn, *d_fn;
};

// ---- lists -----------------------------------------------------------------------------
__global__ void k_adj_geo(long long gm, const double *__restrict__ lam, const double *__restrict__ delta_m,
                          const double *__restrict__ limb_m, const double *__restrict__ lb_m,
                          const int *__restrict__ region_m, int n_mu, double step, AdjGeo *__restrict__ geo,
                          unsigned long long *__restrict__ keys, int *__restrict__ vals) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= gm) return;
    const double d = delta_m[k];
    const CellShift cs = soap_cell_shift(d, lam[0], step);
    const double b = d * 1000. / SOAP_C_LIGHT, omb = 1.0 - b;
    AdjGeo g;
    g.f = cs.fbeta + 0.0;   // +0 for no shift
    g.off = cs.off;
    g.iS = 1.0 / cs.sq;
    g.K = (1000. / SOAP_C_LIGHT) / (cs.sq * cs.sq * cs.sq * omb * omb);
    g.L = limb_m[k];
    g.a = g.L * g.iS;
    g.sig = __dadd_rn(1.0, lb_m[k]);
    g.still = d == 0.0 ? 1.0 : 0.0;
    geo[k] = g;
    // by row, then by f (its last 8 bits, 1e-13 of it, are below the ranges' margins)
    const int row = region_m[k];
    keys[k] = ((unsigned long long)((unsigned)row < (unsigned)n_mu ? row : 0) << 56) | (soap_ord64(g.f) >> 8);
    vals[k] = (int)k;
}

// the order's keys, the cell last
struct AdjKey {
    const unsigned long long *keys;
    __device__ __forceinline__ OrderKey operator()(int k) const { return OrderKey{keys[k], (unsigned)k}; }
};

// One block per phase: the active cells in the map's sorted order, class by class, and the
// first entry of every row.  A thread takes ADJ_LIST_ITEMS consecutive cells at a time.
constexpr int ADJ_LIST_ITEMS = 8;

__global__ void __launch_bounds__(1024) k_adj_lists(long long gm, int n_mu, const int *__restrict__ order,
                                                    const double *__restrict__ temp, const double *__restrict__ bi,
                                                    const AdjGeo *__restrict__ geo, const int *__restrict__ region_m,
                                                    int solar, int t_norm_fac, int *__restrict__ cell,
                                                    double *__restrict__ fb, int *__restrict__ seg, int *status) {
    __shared__ int s_warp[ADJ_CLASS][32], s_tot[ADJ_CLASS];
    const int p = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double *pt = temp + (long long)p * gm, *pb = bi + (long long)p * gm;
    int *pc = cell + (long long)p * gm;
    double *pf = fb + (long long)p * gm;
    auto cls = [&](int k) {
        const double t = pb[k];
        if (!(t >= -0.5 && t <= 1.5)) return -1;
        if ((unsigned)region_m[k] >= (unsigned)n_mu) atomicExch(status, 21);
        const double T = pt[k];
        if (!(fabs(geo[k].f) < ADJ_F_MAX)) return 2;
        if (t == 0.0) return (double)(int)T == T ? 0 : 2;
        return solar ? 2 : 1;
    };
    if (threadIdx.x < ADJ_CLASS) s_tot[threadIdx.x] = 0;
    __syncthreads();
    int cnt[ADJ_CLASS] = {0, 0, 0};
    for (long long i = threadIdx.x; i < gm; i += blockDim.x) {
        const int c = cls((int)i);
#pragma unroll
        for (int q = 0; q < ADJ_CLASS; ++q) cnt[q] += c == q;
    }
#pragma unroll
    for (int q = 0; q < ADJ_CLASS; ++q) {
        const int v = __reduce_add_sync(0xffffffffu, cnt[q]);
        if (lane == 0) atomicAdd(&s_tot[q], v);
    }
    __syncthreads();
    int base[ADJ_CLASS] = {0, s_tot[0], s_tot[0] + s_tot[1]};
    for (long long s = 0; s < gm; s += (long long)blockDim.x * ADJ_LIST_ITEMS) {
        const long long i0 = s + (long long)threadIdx.x * ADJ_LIST_ITEMS;
        int k[ADJ_LIST_ITEMS], c[ADJ_LIST_ITEMS];
#pragma unroll
        for (int v = 0; v < ADJ_LIST_ITEMS; ++v) k[v] = i0 + v < gm ? order[i0 + v] : -1;
#pragma unroll
        for (int v = 0; v < ADJ_LIST_ITEMS; ++v) c[v] = k[v] >= 0 ? cls(k[v]) : -1;
        int own[ADJ_CLASS], at[ADJ_CLASS];
#pragma unroll
        for (int q = 0; q < ADJ_CLASS; ++q) {
            own[q] = 0;
#pragma unroll
            for (int v = 0; v < ADJ_LIST_ITEMS; ++v) own[q] += c[v] == q;
            at[q] = own[q];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, at[q], o);
                if (lane >= o) at[q] += t;
            }
            if (lane == 31) s_warp[q][w] = at[q];
        }
        __syncthreads();
        if (w < ADJ_CLASS) {
            int v = s_warp[w][lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            s_warp[w][lane] = v;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < ADJ_CLASS; ++q) {
            at[q] += base[q] + (w ? s_warp[q][w - 1] : 0) - own[q];
            base[q] += s_warp[q][31];
        }
#pragma unroll
        for (int v = 0; v < ADJ_LIST_ITEMS; ++v) {
            if (c[v] < 0) continue;
            const int to = c[v] == 0 ? at[0]++ : c[v] == 1 ? at[1]++ : at[2]++;
            pc[to] = k[v];
            pf[to] = geo[k[v]].f;
        }
        __syncthreads();
    }
    // rows ascend inside a class (the sorted order): first entry of each
    for (int q = threadIdx.x; q < ADJ_CLASS * (n_mu + 1); q += blockDim.x) {
        const int c = q / (n_mu + 1), b = q % (n_mu + 1);
        int lo = c == 0 ? 0 : c == 1 ? s_tot[0] : s_tot[0] + s_tot[1], hi = lo + s_tot[c];
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            const int row = region_m[pc[mid]];
            if (((unsigned)row < (unsigned)n_mu ? row : 0) < b) lo = mid + 1;
            else hi = mid;
        }
        seg[((long long)p * ADJ_CLASS + c) * (n_mu + 1) + b] = lo;
    }
}

constexpr double ADJ_W_MAX = 0x1p-10;   // |f| whose residues adj_residue takes

// a row of a class (block: row, class, phase): its entries' weights and AdjRow
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_entries(long long gm, int n_mu, const int *__restrict__ cell,
                                                             const double *__restrict__ fb,
                                                             const int *__restrict__ seg,
                                                             const AdjGeo *__restrict__ geo, AdjEnt *__restrict__ ent,
                                                             AdjNoise *__restrict__ noise, AdjRow *__restrict__ row) {
    __shared__ int2 s_z;
    __shared__ unsigned long long s_top[2], s_low[2];
    __shared__ double s_v[ADJ_THREADS / 32][4];
    const int b = blockIdx.x, c = blockIdx.y, p = blockIdx.z, t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int *sg = seg + ((long long)p * ADJ_CLASS + c) * (n_mu + 1);
    const int a = sg[b], e = sg[b + 1];
    const int *pc = cell + (long long)p * gm;
    const double *pf = fb + (long long)p * gm;
    AdjEnt *pe = ent + (long long)p * gm;
    AdjNoise *pn = noise + (long long)p * gm;
    if (a == e) return;   // (nothing reads its AdjRow)
    if (t < 2) {   // first entry with f >= 0, first with f > 0
        int lo = a, hi = e;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (t == 0 ? pf[mid] < 0.0 : pf[mid] <= 0.0) lo = mid + 1;
            else hi = mid;
        }
        (t == 0 ? s_z.x : s_z.y) = lo;
        s_top[t] = 0ULL;
        s_low[t] = ~0ULL;
    }
    __syncthreads();
    // the sums of the entries without a shift, and the largest and smallest finite weights but zero
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    unsigned long long top[2] = {0ULL, 0ULL}, low[2] = {~0ULL, ~0ULL};
    for (int k = a + t; k < e; k += ADJ_THREADS) {
        const AdjGeo &g = geo[pc[k]];
        const double s = c == 0 ? 1.0 : g.sig, x[2] = {fabs(g.a), fabs(g.a * s)};
        pe[k] = {g.L, g.a, g.sig};
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (x[q] > 0.0 && x[q] < INFINITY) {
                top[q] = max(top[q], (unsigned long long)__double_as_longlong(x[q]));
                low[q] = min(low[q], (unsigned long long)__double_as_longlong(x[q]));
            }
        if (k < s_z.x || k >= s_z.y) continue;
        v[0] += g.L;
        v[1] = fma(g.L, s, v[1]);
        v[2] = fma(g.still, g.L, v[2]);
        v[3] = fma(g.still, g.L * s, v[3]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (top[q] != 0ULL) {
            atomicMax(&s_top[q], top[q]);
            atomicMin(&s_low[q], low[q]);
        }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (lane == 0) s_v[w][q] = v[q];
    }
    __syncthreads();
    // units that keep the weights below 2^30
    int ex[2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
        ex[q] = min(max((int)(s_top[q] >> 52) - 1022, -900), 1023);   // the largest lies below 2^ex
    if (t == 0) {
        AdjRow r;
        double sum[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            sum[q] = s_v[0][q];
            for (int k = 1; k < ADJ_THREADS / 32; ++k) sum[q] += s_v[k][q];
        }
        r.zero = s_z;
        r.s0 = sum[0];
        r.t0 = sum[1];
        r.still0 = sum[2];
        r.still1 = sum[3];
        r.unit = scalbn(1.0, ex[0] - 30 - ADJ_FRAC);
        r.unit_s = scalbn(1.0, ex[1] - 30 - ADJ_FRAC);
        r.even = 1;
#pragma unroll
        for (int q = 0; q < 2; ++q)   // by the exponents
            if (s_top[q] != 0ULL && (s_low[q] >> 52) + 12 < (s_top[q] >> 52)) r.even = 0;
        row[((long long)p * 2 + c) * n_mu + b] = r;
    }
    for (int k = a + t; k < e; k += ADJ_THREADS) {
        const AdjGeo &g = geo[pc[k]];
        const double u = fabs(g.f), x = g.f > 0.0 ? -g.a : g.a, y = c == 0 ? x : x * g.sig;
        const bool in = u < ADJ_W_MAX && u > 0.0;
        AdjNoise d;
        d.w = in ? (unsigned long long)__double2ll_rn(u * 0x1p+53) << ADJ_FRAC : 0ULL;
        d.a = in && fabs(x) < INFINITY ? __double2int_rn(scalbn(x, 30 - ex[0])) : 0;
        d.as = in && fabs(y) < INFINITY ? __double2int_rn(scalbn(y, 30 - ex[1])) : 0;
        pn[k] = d;
    }
}

// per-interval reciprocals inv[o] = 1 / (l_{o+1} - l_o), o < n_eff - 1
__global__ void k_adj_inv(int n_eff, const double *__restrict__ lam, double *__restrict__ inv) {
    const long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (o < n_eff - 1) inv[o] = 1.0 / (lam[o + 1] - lam[o]);
}

// ---- ranges ----------------------------------------------------------------------------
// Integer boundaries B of one row of a class at a tile, B0, B0 + 1, ...: entries [lo, hi) may
// cross B inside the tile (a fast cell may cross the next ones too: lo of B + 1 then lies below hi of
// B); those between hi of B and lo of B + 1 have the offset c = B + 1 (owner o of pixel j = o + c) at
// every pixel.  A cell's position there is v = f p (source pixels,
// p = o + lambda0 / step) or f p / S (output pixels, p = j + lambda0 / step), ascending in f; the
// margin eps covers the rounding of the reference's positions.
struct AdjRange {
    int lo[ADJ_NB], hi[ADJ_NB];
    AdjSums sum[ADJ_NB];   // over the entries between boundaries k and k + 1
    long long b0, b1;      // first and last boundary
};

template <bool OUT>
__device__ __forceinline__ double adj_pos(double f, double p) {
    return OUT ? f * p / (1.0 + f) : f * p;
}

// the row's boundaries (every thread; false when the row has no entry)
template <bool OUT>
__device__ __forceinline__ void adj_span(const double *__restrict__ fb, int a, int e, double pa, double pb, double eps,
                                         AdjRange &R) {
    if (threadIdx.x == 0) {
        const double f0 = fb[a], f1 = fb[e - 1];
        const double v0 = floor(fmin(adj_pos<OUT>(f0, pa), adj_pos<OUT>(f0, pb)) - eps);
        const double v1 = ceil(fmax(adj_pos<OUT>(f1, pa), adj_pos<OUT>(f1, pb)) + eps);
        const bool sane = fabs(v0) < 1e9 && fabs(v1) < 1e9 && v1 - v0 < 1e6 && pa > 1.0;
        R.b0 = sane ? (long long)v0 : 0;
        R.b1 = sane ? (long long)v1 : -1;   // else every entry by itself
    }
}

// boundaries first .. first + count - 1 by threads 0 .. 2 count - 1 (two binary searches each).
// f p - B d > x, d = 1 + f for output pixels, else 1, is f > (B + x) / (p - B) or (B + x) / p, with
// the tile end p that is the last to satisfy it; the search then compares integer images.
template <bool OUT>
__device__ __forceinline__ void adj_bounds(const double *__restrict__ fb, int a, int e, double pa, double pb, double eps,
                                           long long first, int count, AdjRange &R) {
    const int k = threadIdx.x >> 1;
    if (k >= count) return;
    const double B = (double)(first + k);
    const bool up = threadIdx.x & 1;
    const double x = up ? B + eps : B - eps;
    const double f = x / (((x > 0.0) == up ? pa : pb) - (OUT ? B : 0.0));
    const unsigned long long key = soap_ord64(f);
    int lo = a, hi = e;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const unsigned long long v = soap_ord64(fb[mid]);
        if (up ? v <= key : v < key) lo = mid + 1;
        else hi = mid;
    }
    (up ? R.hi : R.lo)[k] = lo;
}

// sums over the entries [lo, hi) of class c, a warp: every lane's result the same
__device__ __forceinline__ AdjSums adj_sum(const AdjEnt *__restrict__ ent, const double *__restrict__ fb, int c, int lo,
                                           int hi) {
    AdjSums s;
    s.f0 = fb[lo];
    const double u = fmax(fabs(s.f0), fabs(fb[hi - 1]));   // they ascend
    s.zone = u < ADJ_W_MAX ? (int)(u * (double)(1 << ADJ_FRAC)) + 3 : 0;
    s.s0 = s.s1 = s.s2 = s.t0 = s.t1 = s.t2 = 0.0;
    for (int k = lo + (threadIdx.x & 31); k < hi; k += 32) {
        const AdjEnt x = ent[k];
        const double d = fb[k] - s.f0;
        s.s0 += x.L;
        s.s1 += x.a;
        s.s2 = fma(x.a, d, s.s2);
        if (c == 1) {
            const double as = x.a * x.sig;
            s.t0 = fma(x.L, x.sig, s.t0);
            s.t1 += as;
            s.t2 = fma(as, d, s.t2);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        s.s0 += __shfl_xor_sync(0xffffffffu, s.s0, o);
        s.s1 += __shfl_xor_sync(0xffffffffu, s.s1, o);
        s.s2 += __shfl_xor_sync(0xffffffffu, s.s2, o);
        if (c == 1) {
            s.t0 += __shfl_xor_sync(0xffffffffu, s.t0, o);
            s.t1 += __shfl_xor_sync(0xffffffffu, s.t1, o);
            s.t2 += __shfl_xor_sync(0xffffffffu, s.t2, o);
        }
    }
    if (c != 1) {
        s.t0 = s.s0;
        s.t1 = s.s1;
        s.t2 = s.s2;
    }
    return s;
}

// l_j - l_o - l_o f, rounded once (l_j - l_o is exact)
__device__ __forceinline__ double adj_rest(double lj, double lo, double f) { return fma(-lo, f, lj - lo); }

// Walks a row of a class over a tile: group(c, lo, hi, sums) for the entries of one offset (SUMS: with
// their sums), still(row) for those without a shift, single(k) for each of the others.  The calls are
// uniform over the block.
template <bool OUT, bool SUMS, class G, class Z, class S>
__device__ __forceinline__ void adj_walk(const AdjArgs &A, int p, int c, int b, double pa, double pb, double eps,
                                         AdjRange &R, G group, Z still, S single) {
    const int *sg = A.seg + ((long long)p * ADJ_CLASS + c) * (A.n_mu + 1);
    const int a = sg[b], e = sg[b + 1];
    if (a == e) return;
    const double *fb = A.fb + (long long)p * A.gm;
    if (c == 2) {
        for (int k = a; k < e; ++k) single(k);
        return;
    }
    const AdjRow &row = A.row[((long long)p * 2 + c) * A.n_mu + b];
    const int2 z = row.zero;
    __syncthreads();
    adj_span<OUT>(fb, a, e, pa, pb, eps, R);
    __syncthreads();
    const long long b1 = R.b1;
    if (b1 < R.b0) {
        for (int k = a; k < e; ++k)
            if (k < z.x || k >= z.y) single(k);
        if (z.x < z.y) still(row);
        return;
    }
    int done = a;   // entries below it are evaluated
    for (long long first = R.b0;; first += ADJ_NB - 1) {
        const int count = (int)min((long long)ADJ_NB, b1 - first + 1);
        __syncthreads();
        adj_bounds<OUT>(fb, a, e, pa, pb, eps, first, count, R);
        __syncthreads();
        if constexpr (SUMS) {
            const AdjEnt *ent = A.ent + (long long)p * A.gm;
            for (int k = threadIdx.x >> 5; k + 1 < count; k += ADJ_THREADS / 32)
                if (R.hi[k] < R.lo[k + 1]) {
                    const AdjSums x = adj_sum(ent, fb, c, R.hi[k], R.lo[k + 1]);
                    if ((threadIdx.x & 31) == 0) R.sum[k] = x;
                }
            __syncthreads();
        }
        for (int k = 0; k < count; ++k) {
            if (k + 1 < count && R.hi[k] < R.lo[k + 1]) group((int)(first + k + 1), R.hi[k], R.lo[k + 1], R.sum[k]);
            if (k + 1 < count || first + k == b1) {   // a boundary shared by two batches once
                for (int q = max(R.lo[k], done); q < R.hi[k]; ++q)
                    if (q < z.x || q >= z.y) single(q);
                done = max(done, R.hi[k]);
            }
        }
        if (first + count - 1 >= b1) break;
    }
    if (z.x < z.y) still(row);
}

__device__ __forceinline__ int adj_exp(double v) { return (int)(((unsigned)__double2hiint(v) >> 20) & 0x7ffu); }

__device__ __forceinline__ double adj_intensity(const AdjArgs &A, int p, int c, int k, double lj, double ssed,
                                                double fsed) {
    // class 2: the map's temperature and the general ratio; a spot's type is read from the list's class
    const double T = A.temp[(long long)p * A.gm + k];
    return soap_intensity(c, T, A.lb[k], lj, ssed, fsed, A.solar, A.t_norm_fac);
}

// l'_o as the forward rounds it
__device__ __forceinline__ double adj_shifted(double lo, double f) { return __dsub_rn(lo, __dmul_rn(lo, -f)); }

// The forward's l'_o is l_o - rn(l_o u) rounded to ulp(l_o), u = 1 - S: up to half an ulp, 1e-10 of
// a pixel, from S l_o.  The row gradients take the weights of that grid, so that they are the
// transpose of the forward to better than this: the sum over the cells [k0, k1) of L / S times the
// residue.  The fraction bits of the 64-bit product are integers (about 2^20; the two products'
// lower halves are left out, 2^-21 of an ulp on either side), the weights integers of at most 2^30,
// and the sums exact.  Within `zone` of a half, the error of the product and of the reference's rn(l_o
// u), the whole ulps are the FP64 operations' (without it a pixel in some thousands had a cell's
// weight wrong by an ulp of l).  lm: l_o's significand, leading bit at bit 63; TWO: the facula
// weights too.
constexpr int ADJ_HALF = 1 << (ADJ_FRAC - 1);

// the product's low bits, with half an ulp and the zone added: whole ulps from bit ADJ_FRAC on
__device__ __forceinline__ unsigned adj_product(const AdjNoise &c, unsigned long long lm, int zone) {
    const unsigned h = (unsigned)(lm >> 32), l = (unsigned)lm, wh = (unsigned)(c.w >> 32), wl = (unsigned)c.w;
    return h * wh + __umulhi(h, wl) + __umulhi(l, wh) + (unsigned)(ADJ_HALF + 1 + zone);
}

// What the cells near a half among [k0, k1) add where the FP64 operations give an ulp less (a call, off
// the others' path: one in 2^19 / zone cells is near)
static __device__ __noinline__ longlong2 adj_near_half(const AdjNoise *__restrict__ x, const double *__restrict__ fb,
                                                       double lo, unsigned long long lm, int k0, int k1, int zone) {
    longlong2 s = make_longlong2(0, 0);
    for (int k = k0; k < k1; ++k) {
        const AdjNoise c = x[k];
        const unsigned v = adj_product(c, lm, zone);
        if ((v & (2u * ADJ_HALF - 1u)) >= 2u * (unsigned)zone) continue;
        const long long w = __double_as_longlong(lo) - __double_as_longlong(adj_shifted(lo, fb[k]));
        // the difference of the whole ulps, by their low bits: 0 or -1
        const int d = (int)(((unsigned)(w < 0 ? -w : w) - (v >> ADJ_FRAC)) << ADJ_FRAC) >> ADJ_FRAC;
        s.x -= (long long)c.a * (d * (2 * ADJ_HALF));
        s.y -= (long long)c.as * (d * (2 * ADJ_HALF));
    }
    return s;
}

template <bool TWO>
__device__ __forceinline__ void adj_residue(const AdjNoise *__restrict__ x, const double *__restrict__ fb, double lo,
                                            unsigned long long lm, int k0, int k1, int zone, double &r, double &rs) {
    constexpr int PART = 4096, CHUNK = 32;   // 2^12 products below 2^51
    r = rs = 0.0;
    for (int q = k0; q < k1; q += PART) {
        long long s = 0, t = 0;
        const int end = min(k1, q + PART);
        for (int c0 = q; c0 < end; c0 += CHUNK) {
            const int c1 = min(end, c0 + CHUNK);
            unsigned near = ~0u;
#pragma unroll 4
            for (int k = c0; k < c1; ++k) {
                const AdjNoise c = x[k];
                const unsigned f = adj_product(c, lm, zone) & (2u * ADJ_HALF - 1u);
                const int fr = (int)f - (ADJ_HALF + zone);
                near = min(near, f);
                s += (long long)c.a * fr;
                if (TWO) t += (long long)c.as * fr;
            }
            if (near < 2u * (unsigned)zone) {
                const longlong2 fix = adj_near_half(x, fb, lo, lm, c0, c1, zone);
                s += fix.x;
                if (TWO) t += fix.y;
            }
        }
        r += (double)s;
        if (TWO) rs += (double)t;
    }
}

// ---- row gradients -----------------------------------------------------------------------
// Block: ADJ_SRC source pixels of one row, lane l of a warp source o; lane 0 only gives its upper
// share to lane 1.  BC: the bconv gradient alone (gF = gT = 0).  Bound by the FP64 pipe (71 % of
// cycles, some twenty instructions per range and pixel) and the latency of the residues' integer
// chains, so four and three blocks per SM although some registers spill (three
// and two: 0.49 and 0.56 ms for 100 x 100 cells and 50,000 px, BC, and five phases of 200 x 200 and
// 100,000 px; so 0.47 and 0.46).
template <bool BC>
__global__ void __launch_bounds__(ADJ_THREADS, BC ? 4 : 3) k_adj_rows(const __grid_constant__ AdjArgs A,
                                                          const double *__restrict__ bi) {
    __shared__ AdjRange R;
    const int b = blockIdx.y, lane = threadIdx.x & 31, n_eff = A.n_eff;
    const int i0 = blockIdx.x * ADJ_SRC, o = i0 + (threadIdx.x >> 5) * 31 + lane - 1;
    const double *__restrict__ lam = A.lam;
    const double ls = lam[0] / A.step;
    const double pa = (double)(i0 - 1) + ls, pb = (double)(i0 + ADJ_SRC) + ls;
    const double eps = 1.8e-15 * (4.0 * (double)n_eff + 2.0 * ADJ_F_MAX * fabs(ls) + 4.0);
    const bool own = o >= 0 && o <= n_eff - 2;
    const double lo = own ? lam[o] : 0.0, io = own ? A.inv[o] : 0.0, beta = lo * io;
    const int ex = adj_exp(lo);
    const bool noisy = ex > 200 && ex < 1800;   // a wavelength whose ulp is a normal number
    // no shift below ADJ_W_MAX takes l_o out of its binade: 2^-9 of it, 2^11 in the high word, from both ends
    const bool inner = ((unsigned)__double2hiint(lo) & 0xfffffu) - 2048u < (1u << 20) - 4096u;
    const unsigned long long lm = ((unsigned long long)__double_as_longlong(lo) << 11) | 0x8000000000000000ULL;
    const double ulp = noisy ? __hiloint2double((ex - 52) << 20, 0) * io : 0.0;
    double L[4] = {0.0, 0.0, 0.0, 0.0}, U[4] = {0.0, 0.0, 0.0, 0.0};   // q_sed, q_norm, spot, facula: lower, upper
    for (int p = 0; p < A.n_phase; ++p) {
        const long long go = (long long)p * A.n;
        const double *gf = A.gF + go, *gb = A.gB + go, *gt = A.gT + go;
        const AdjNoise *noise = A.noise + (long long)p * A.gm;
        const double *fb = A.fb + (long long)p * A.gm;
        const int *cell = A.cell + (long long)p * A.gm;
#pragma unroll 1
        for (int c = 0; c < ADJ_CLASS; ++c) {
            // shares wl (to o) and w1 (to o + 1; not without `up`, where a gradient that is not finite
            // must not reach it) of pixel j; wls, w1s: with the intensity's factor
            auto add = [&](int j, double wl, double w1, double wls, double w1s, double sed, int type, bool up) {
                const double B = gb[j];
                double q = wl * B, u = w1 * B, al = q, au = u;
                if constexpr (!BC) {
                    const double F = gf[j], T = gt[j], h = F + T, x = sed * F, y = sed * T;
                    L[0] = fma(wl, h, L[0]);
                    if (up) U[0] = fma(w1, h, U[0]);
                    q = fma(-wls, x, q);
                    u = fma(-w1s, x, u);
                    al = fma(wls, y, al);
                    au = fma(w1s, y, au);
                }
                L[1] += q;
                if (type == 0) L[2] -= al;
                else L[3] -= al;
                if (up) {
                    U[1] += u;
                    if (type == 0) U[2] -= au;
                    else U[3] -= au;
                }
            };
            auto sed_at = [&](int type, int j) { return BC ? 0.0 : (type == 0 ? A.spot_sed[j] : A.fac_sed[j]); };
            const AdjRow &row = A.row[((long long)p * 2 + (c < 2 ? c : 0)) * A.n_mu + b];
            adj_walk<false, true>(
                A, p, c, b, pa, pb, eps, R,
                [&](int off, int k0, int k1, const AdjSums &s) {
                    const int j = o + off;
                    if (!own || j < 0 || j >= n_eff) return;
                    const double lj = lam[j];
                    const bool two = !BC && c == 1;
                    double w1, w1s;
                    // |f| below ADJ_W_MAX, and l' in l_o's binade for the range's extreme shifts
                    if (noisy && row.even && s.zone != 0 &&
                        (inner || (adj_exp(fma(lo, s.f0, lo)) == ex && adj_exp(fma(lo, fb[k1 - 1], lo)) == ex))) {
                        const double rest = adj_rest(lj, lo, s.f0);
                        double r, rs;
                        if (two) adj_residue<true>(noise, fb, lo, lm, k0, k1, s.zone, r, rs);
                        else adj_residue<false>(noise, fb, lo, lm, k0, k1, s.zone, r, rs);
                        w1 = fma(io, fma(rest, s.s1, -lo * s.s2), -ulp * (row.unit * r));
                        w1s = two ? fma(io, fma(rest, s.t1, -lo * s.t2), -ulp * (row.unit_s * rs)) : w1;
                    } else {   // the forward's l' cell by cell
                        w1 = w1s = 0.0;
                        for (int k = k0; k < k1; ++k) {
                            const AdjGeo &g = A.geo[cell[k]];
                            const double w = g.a * ((lj - adj_shifted(lo, g.f)) * io);
                            w1 += w;
                            w1s = fma(w, g.sig, w1s);
                        }
                        if (!two) w1s = w1;
                    }
                    add(j, s.s0 - w1, w1, (two ? s.t0 : s.s0) - w1s, w1s, sed_at(c, j), c, true);
                },
                [&](const AdjRow &z) {   // no shift: pixel j is source j
                    if (o < 0 || o >= n_eff) return;
                    const bool end = o == n_eff - 1;   // without an interval above it: the cells at rest only
                    add(o, end ? z.still0 : z.s0, 0.0, end ? z.still1 : z.t0, 0.0, sed_at(c, o), c, false);
                },
                [&](int k) {
                    const AdjGeo &g = A.geo[cell[k]];
                    const int type = c == 2 ? (bi[(long long)p * A.gm + cell[k]] == 0.0 ? 0 : 1) : c;
                    const double sg = c == 1 ? g.sig : 1.0;
                    auto sed_of = [&](int j) {
                        return (!BC && c == 2) ? adj_intensity(A, p, type, cell[k], lam[j], A.spot_sed[j], A.fac_sed[j])
                                               : sed_at(type, j);
                    };
                    if (g.still != 0.0) {
                        if (o >= 0 && o < n_eff) add(o, g.L, 0.0, g.L * sg, 0.0, sed_of(o), type, false);
                        return;
                    }
                    if (!own) return;
                    CellShift cs;
                    cs.fbeta = g.f;
                    cs.off = g.off;
                    const long long ja = max(soap_ceil_pos(o, cs), 0LL), jb = min(soap_ceil_pos(o + 1, cs), (long long)n_eff);
                    const double l1 = adj_shifted(lo, g.f);
                    for (long long j = ja; j < jb; ++j) {
                        const double w1 = g.L * ((lam[j] - l1) * g.iS * io), wl = g.L - w1;
                        add((int)j, wl, w1, wl * sg, w1 * sg, sed_of((int)j), type, true);
                    }
                });
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) L[q] += __shfl_up_sync(0xffffffffu, U[q], 1);
    if (lane != 0 && o < A.n) {
        const long long at = (long long)b * A.n + o;
        const bool in = o < n_eff;
        double *const out[4] = {A.d_qs, A.d_qn, A.d_sn, A.d_fn};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double v = in ? L[q] : 0.0;
            out[q][at] = A.more ? out[q][at] + v : v;
        }
    }
}

// ---- continuum rows ------------------------------------------------------------------------
// Block: 256 output pixels, the cells of one row; per row and class into part, summed afterwards
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_continuum(const __grid_constant__ AdjArgs A,
                                                               const double *__restrict__ bi) {
    __shared__ AdjRange R;
    const int b = blockIdx.y, n_eff = A.n_eff, j0 = blockIdx.x * ADJ_THREADS, j = j0 + threadIdx.x;
    const int cnt = max(1, min(ADJ_THREADS, n_eff - j0));
    const double *__restrict__ lam = A.lam;
    const double ls = lam[0] / A.step, pa = (double)j0 + ls, pb = (double)(j0 + cnt - 1) + ls;
    const double eps = 1.8e-15 * (4.0 * (double)n_eff + 2.0 * ADJ_F_MAX * fabs(ls) + 4.0);
    const double lj = j < n_eff ? lam[j] : 0.0;
    const double *qn = A.q_norm + (long long)b * A.n;
    double sum[2] = {0.0, 0.0};
    for (int p = 0; p < A.n_phase; ++p) {
        const double gf = j < n_eff ? A.gF[(long long)p * A.n + j] : 0.0;
        const double gt = j < n_eff ? A.gT[(long long)p * A.n + j] : 0.0;
        const int *cell = A.cell + (long long)p * A.gm;
#pragma unroll 1
        for (int c = 0; c < ADJ_CLASS; ++c) {
            // -ratio (q gF + a gT): w0 and w1 the cells' sums of ratio L and ratio L w
            auto add = [&](int o, double w0, double w1, int type) {
                const double *an = (type == 0 ? A.spot_norm : A.fac_norm) + (long long)b * A.n;
                const double q0 = qn[o], a0 = an[o];
                double q = w0 * q0, a = w0 * a0;
                if (w1 != 0.0) {
                    q = fma(w1, qn[o + 1] - q0, q);
                    a = fma(w1, an[o + 1] - a0, a);
                }
                const double h = -fma(q, gf, a * gt);
                if (type == 0) sum[0] += h;
                else sum[1] += h;
            };
            adj_walk<true, true>(
                A, p, c, b, pa, pb, eps, R,
                [&](int off, int, int, const AdjSums &s) {
                    const int o = j - off;
                    if (j >= n_eff || o < 0 || o > n_eff - 2) return;
                    const double lo = lam[o];
                    add(o, s.t0, A.inv[o] * fma(adj_rest(lj, lo, s.f0), s.t1, -lo * s.t2), c);
                },
                [&](const AdjRow &z) {
                    if (j < n_eff) add(j, j == n_eff - 1 ? z.still1 : z.t0, 0.0, c);
                },
                [&](int k) {
                    if (j >= n_eff) return;
                    const AdjGeo &g = A.geo[cell[k]];
                    const int type = c == 2 ? (bi[(long long)p * A.gm + cell[k]] == 0.0 ? 0 : 1) : c;
                    const double ratio = c == 1 ? g.sig : c == 2 ? adj_intensity(A, p, type, cell[k], lj, 1.0, 1.0) : 1.0;
                    if (g.still != 0.0) {
                        add(j, ratio * g.L, 0.0, type);
                        return;
                    }
                    CellShift cs;
                    cs.fbeta = g.f;
                    cs.off = g.off;
                    const long long o = soap_owner(j, n_eff, cs);
                    if (o < 0) return;
                    const double lo = lam[o], io = A.inv[o];
                    add((int)o, ratio * g.L, ratio * (g.a * (adj_rest(lj, lo, g.f) * io)), type);
                });
        }
    }
    if (j < A.n) {
        A.part[((long long)b * 2 + 0) * A.n + j] = sum[0];
        A.part[((long long)b * 2 + 1) * A.n + j] = sum[1];
    }
}

__global__ void k_adj_sum_rows(int n, int n_mu, int more, const double *__restrict__ part, double *__restrict__ d_ss,
                               double *__restrict__ d_fs) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double s = more ? d_ss[j] : 0.0, f = more ? d_fs[j] : 0.0;
    for (int b = 0; b < n_mu; ++b) {
        s += part[((long long)b * 2 + 0) * n + j];
        f += part[((long long)b * 2 + 1) * n + j];
    }
    d_ss[j] = s;
    d_fs[j] = f;
}

// ---- limb and velocity ---------------------------------------------------------------------
// Block: one row of one phase over a share of the pixels, tile by tile.  For each offset's cells
// the tile gives three sums over its pixels (six for the faculae, whose intensity factor differs
// from cell to cell): of P, of alpha' Q and of beta Q, P and Q the rows' values and differences
// dotted with h, alpha' = inv[o] (l_j - l_o - l_o f0) with the range's f0; a cell adds
// P + (alpha' Q - (f - f0) beta Q) / S to its limb gradient and -K (alpha' Q + (1 + f0) beta Q) to its
// velocity gradient.
constexpr int ADJ_WARPS = ADJ_THREADS / 32;

template <bool BC>
__global__ void __launch_bounds__(ADJ_THREADS) k_adj_limb(const __grid_constant__ AdjArgs A,
                                                          const double *__restrict__ bi) {
    __shared__ AdjRange R;
    __shared__ double s_v[6][ADJ_THREADS], s_sum[6];
    const int b = blockIdx.x, p = blockIdx.y, n_eff = A.n_eff, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double *__restrict__ lam = A.lam;
    const double ls = lam[0] / A.step;
    const double eps = 1.8e-15 * (4.0 * (double)n_eff + 2.0 * ADJ_F_MAX * fabs(ls) + 4.0);
    const long long ro = (long long)b * A.n, go = (long long)p * A.n;
    const double *qn = A.q_norm + ro, *qs = A.q_sed + ro;
    const double *gf = A.gF + go, *gb = A.gB + go, *gt = A.gT + go;
    const int *cell = A.cell + (long long)p * A.gm;
    double *acc = A.acc + ((long long)blockIdx.z * A.n_phase + p) * A.gm * 2;
    const int tiles = (n_eff + ADJ_THREADS - 1) / ADJ_THREADS;
    const int t0 = (int)((long long)tiles * blockIdx.z / A.Q), t1 = (int)((long long)tiles * (blockIdx.z + 1) / A.Q);
#pragma unroll 1
    for (int c = 0; c < ADJ_CLASS; ++c) {
        const int *sg = A.seg + ((long long)p * ADJ_CLASS + c) * (A.n_mu + 1);
        if (sg[b] == sg[b + 1]) continue;
        // values and differences of the rows at source o dotted with h at pixel j, without (x) and
        // with (y) the intensity factor; last: pixel n_eff - 1 of a cell at rest has no interval
        auto dots = [&](int j, int o, int type, double I, bool last, double &P, double &Qd, double &Ps, double &Qsd) {
            const double *an = (type == 0 ? A.spot_norm : A.fac_norm) + ro;
            const double B = gb[j], q0 = qn[o], a0 = an[o];
            const double eq = last ? 0.0 : qn[o + 1] - q0, ea = last ? 0.0 : an[o + 1] - a0;
            P = B * (q0 - a0);
            Qd = B * (eq - ea);
            Ps = Qsd = 0.0;
            if constexpr (!BC) {
                const double F = gf[j], T = gt[j], h = F + T, s0 = qs[o], x = I * F, y = I * T;
                P = fma(h, s0, P);
                if (!last) Qd = fma(h, qs[o + 1] - s0, Qd);
                Ps = -fma(x, q0, y * a0);
                Qsd = -fma(x, eq, y * ea);
            }
        };
        auto sed_at = [&](int type, int j) { return BC ? 0.0 : (type == 0 ? A.spot_sed[j] : A.fac_sed[j]); };
        for (int t = t0; t < t1; ++t) {
            const int j0 = t * ADJ_THREADS, cnt = min(ADJ_THREADS, n_eff - j0), j = j0 + threadIdx.x;
            const double pa = (double)j0 + ls, pb = (double)(j0 + cnt - 1) + ls;
            // block sums of v[0 .. nv - 1]: warp q sums value q
            auto reduce = [&](double *v, int nv) {
                for (int q = 0; q < nv; ++q) s_v[q][threadIdx.x] = v[q];
                __syncthreads();
                if (w < nv) {
                    double s = s_v[w][lane];
#pragma unroll
                    for (int k = 1; k < ADJ_WARPS; ++k) s += s_v[w][32 * k + lane];
                    for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
                    if (lane == 0) s_sum[w] = s;
                }
                __syncthreads();
                for (int q = 0; q < nv; ++q) v[q] = s_sum[q];
            };
            adj_walk<true, false>(
                A, p, c, b, pa, pb, eps, R,
                [&](int off, int k0, int k1, const AdjSums &) {
                    const double f0 = A.fb[(long long)p * A.gm + k0];
                    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                    const int o = j - off;
                    if (j < n_eff && o >= 0 && o <= n_eff - 2) {
                        double P, Q, Ps, Qsd;
                        dots(j, o, c, sed_at(c, j), false, P, Q, Ps, Qsd);
                        const double lo = lam[o], io = A.inv[o], al = adj_rest(lam[j], lo, f0) * io, be = lo * io;
                        if (c == 0) {
                            P += Ps;
                            Q += Qsd;
                        }
                        v[0] = P;
                        v[1] = al * Q;
                        v[2] = be * Q;
                        v[3] = Ps;
                        v[4] = al * Qsd;
                        v[5] = be * Qsd;
                    }
                    const bool two = !BC && c == 1;
                    reduce(v, two ? 6 : 3);
                    for (int k = k0 + threadIdx.x; k < k1; k += ADJ_THREADS) {
                        const AdjGeo &g = A.geo[cell[k]];
                        double g0 = v[0], g1 = v[1], g2 = v[2];
                        if (two) {
                            g0 = fma(g.sig, v[3], g0);
                            g1 = fma(g.sig, v[4], g1);
                            g2 = fma(g.sig, v[5], g2);
                        }
                        acc[2 * k] += fma(fma(f0 - g.f, g2, g1), g.iS, g0);
                        acc[2 * k + 1] = fma(-g.K, fma(1.0 + f0, g2, g1), acc[2 * k + 1]);
                    }
                },
                [&](const AdjRow &z) {
                    const int k0 = z.zero.x, k1 = z.zero.y;
                    double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
                    double end = 0.0, end_s = 0.0;   // pixel n_eff - 1
                    if (j < n_eff) {
                        double P, Q, Ps, Qsd;
                        const bool last = j == n_eff - 1;
                        dots(j, j, c, sed_at(c, j), last, P, Q, Ps, Qsd);
                        if (!last) {
                            v[0] = P;
                            v[1] = lam[j] * A.inv[j] * Q;
                            v[2] = Ps;
                            v[3] = lam[j] * A.inv[j] * Qsd;
                        } else {
                            end = P;
                            end_s = Ps;
                        }
                    }
                    v[4] = end;
                    v[5] = end_s;
                    reduce(v, 6);
                    for (int k = k0 + threadIdx.x; k < k1; k += ADJ_THREADS) {
                        const AdjGeo &g = A.geo[cell[k]];
                        const double s = c == 0 ? 1.0 : g.sig;
                        acc[2 * k] += fma(s, v[2], v[0]) + g.still * fma(s, v[5], v[4]);
                        acc[2 * k + 1] = fma(-g.K, fma(s, v[3], v[1]), acc[2 * k + 1]);
                    }
                },
                [&](int k) {
                    const AdjGeo &g = A.geo[cell[k]];
                    const int type = c == 2 ? (bi[(long long)p * A.gm + cell[k]] == 0.0 ? 0 : 1) : c;
                    const double s = c == 1 ? g.sig : 1.0;
                    double v[2] = {0.0, 0.0};
                    if (j < n_eff) {
                        CellShift cs;
                        cs.fbeta = g.f;
                        cs.off = g.off;
                        const bool rest = g.still != 0.0, last = rest && j == n_eff - 1;
                        const long long o = rest ? j : soap_owner(j, n_eff, cs);
                        if (o >= 0) {
                            const double lj = lam[j];
                            const double I = (!BC && c == 2) ? adj_intensity(A, p, type, cell[k], lj, A.spot_sed[j], A.fac_sed[j])
                                                             : sed_at(type, j);
                            double P, Q, Ps, Qsd;
                            dots(j, (int)o, type, I, last, P, Q, Ps, Qsd);
                            const double lo = lam[o], io = last ? 0.0 : A.inv[o];
                            const double wt = rest ? 0.0 : adj_rest(lj, lo, g.f) * io * g.iS;
                            const double Qt = fma(s, Qsd, Q);
                            v[0] = fma(wt, Qt, fma(s, Ps, P));
                            v[1] = lj * io * Qt;
                        }
                    }
                    reduce(v, 2);
                    if (threadIdx.x == 0) {
                        acc[2 * k] += v[0];
                        acc[2 * k + 1] = fma(-g.K, v[1], acc[2 * k + 1]);
                    }
                });
            __syncthreads();   // entries are added by different threads from tile to tile
        }
    }
}

// buf[p][cell] of the entries' sums, the shares of the pixels in order
__global__ void k_adj_limb_cells(const __grid_constant__ AdjArgs A, const double *__restrict__ limb_m,
                                 double *__restrict__ buf, double *__restrict__ buf_d) {
    const int p = blockIdx.y, k = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = A.seg[((long long)p * ADJ_CLASS + 2) * (A.n_mu + 1) + A.n_mu];
    if (k >= n) return;
    double s = 0.0, d = 0.0;
    for (int q = 0; q < A.Q; ++q) {
        const double *a = A.acc + ((long long)q * A.n_phase + p) * A.gm * 2 + 2 * (long long)k;
        s += a[0];
        d += a[1];
    }
    const int m = A.cell[(long long)p * A.gm + k];
    buf[(long long)p * A.gm + m] = s;
    buf_d[(long long)p * A.gm + m] = limb_m[m] * d;   // the values carry L
}

// grad_limb[k] = sum over phases, in order, of buf[p][k]
__global__ void k_adj_sum_phases(int n_phase, long long gm, int more, const double *__restrict__ buf, double *out) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= gm) return;
    double s = more ? out[k] : 0.0;
    for (int p = 0; p < n_phase; ++p) s += buf[(long long)p * gm + k];
    out[k] = s;
}

extern "C" int soapgb_phase_integrate_adjoint(soapgb_ctx *ctx, int n, int n_eff, const double *wave, int grid,
                                              int n_phase, const double *temp, const double *bi,
                                              const soapgb_maps *maps, const soapgb_cubes *cubes, double step,
                                              const soapgb_activity *act, const double *g_flux,
                                              const double *g_bconv, const double *g_tot, int mem,
                                              double *grad_q_norm, double *grad_q_sed, double *grad_spot_norm,
                                              double *grad_fac_norm, double *grad_spot_sed, double *grad_fac_sed,
                                              double *grad_limb, double *grad_delta) {
    if (!ctx || !maps || !cubes || !act) return SOAPGB_ERR_ARG;
    if (n < 2 || n_eff < 2 || n_eff > n || grid < 1 || n_phase < 0 || cubes->n_mu < 1 ||
        cubes->n_mu > ADJ_MAX_MU || !(step > 0) || !wave || !temp || !bi || !maps->delta || !maps->limb ||
        !maps->lb || !maps->region || !cubes->q_norm || !cubes->q_sed || !cubes->spot_norm || !cubes->fac_norm ||
        !cubes->spot_sed || !cubes->fac_sed || (!g_flux != !g_tot) || !g_bconv || !grad_q_norm || !grad_q_sed ||
        !grad_spot_norm || !grad_fac_norm || !grad_spot_sed || !grad_fac_sed || !grad_limb || !grad_delta)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_phase_integrate_adjoint: bad arguments");
    SOAP_DEVICE(ctx);
    const long long gm = (long long)grid * grid;
    const int n_mu = cubes->n_mu;
    const size_t cube_b = sizeof(double) * (size_t)n * n_mu, row_b = sizeof(double) * (size_t)n;
    const size_t g_b = sizeof(double) * (size_t)n * std::max(n_phase, 1);
    const size_t map_b = sizeof(double) * (size_t)gm * std::max(n_phase, 1);
    const bool host = (mem == SOAPGB_HOST);
    Workspace ws(ctx);
    int s_wave = ws.add(host ? row_b : 0);
    int s_c[6];
    for (int q = 0; q < 4; ++q) s_c[q] = ws.add(host ? cube_b : 0);
    for (int q = 4; q < 6; ++q) s_c[q] = ws.add(host ? row_b : 0);
    int s_temp = ws.add(host ? map_b : 0), s_bi = ws.add(host ? map_b : 0);
    int s_m[4];
    for (int q = 0; q < 3; ++q) s_m[q] = ws.add(host ? sizeof(double) * gm : 0);
    s_m[3] = ws.add(host ? sizeof(int) * gm : 0);
    int s_g[3];
    for (int q = 0; q < 3; ++q) s_g[q] = ws.add(host ? g_b : 0);
    int s_o[8];
    for (int q = 0; q < 4; ++q) s_o[q] = ws.add(host ? cube_b : 0);
    for (int q = 4; q < 6; ++q) s_o[q] = ws.add(host ? row_b : 0);
    s_o[6] = ws.add(host ? sizeof(double) * gm : 0);
    s_o[7] = ws.add(host ? sizeof(double) * gm : 0);
    // shares of the pixels in the limb kernel: eight blocks per SM over rows, phases and shares (a
    // phase's regions touch about half of the rows)
    const int tiles = (n_eff + ADJ_THREADS - 1) / ADJ_THREADS;
    auto shares = [&](int phases) {
        const int by_blocks = std::min({32, tiles, 8 * std::max(ctx->num_sms, 1) / (n_mu * std::max(phases, 1))});
        const size_t by_scratch = ADJ_SCRATCH / (sizeof(double) * 4 * (size_t)gm * std::max(phases, 1));
        return std::max(1, (int)std::min<size_t>((size_t)std::max(by_blocks, 1), by_scratch));   // half of it
    };
    // phases in a group
    const size_t per_phase = (sizeof(int) + sizeof(double) + sizeof(AdjEnt) + sizeof(AdjNoise) + 4 * sizeof(double)) * (size_t)gm;
    const int group = (int)std::min<size_t>({(size_t)std::max(n_phase, 1), std::max<size_t>(1, ADJ_SCRATCH / per_phase), 65535});
    const int Q = shares(group);
    const size_t pg = (size_t)gm * group, buf_b = sizeof(double) * pg;
    int s_geo = ws.add(sizeof(AdjGeo) * gm);
    int s_key[2], s_val[2];
    for (int q = 0; q < 2; ++q) s_key[q] = ws.add(sizeof(unsigned long long) * gm);
    for (int q = 0; q < 2; ++q) s_val[q] = ws.add(sizeof(int) * gm);
    const bool ranks = gm <= ORDER_MAX;
    const size_t sort_b = ranks ? sizeof(unsigned long long) * gm : fir_sort_temp_bytes(gm);
    int s_sort = ws.add(sort_b);
    int s_cell = ws.add(sizeof(int) * pg), s_fb = ws.add(sizeof(double) * pg), s_ent = ws.add(sizeof(AdjEnt) * pg);
    int s_noise = ws.add(sizeof(AdjNoise) * pg);
    int s_seg = ws.add(sizeof(int) * ADJ_CLASS * (size_t)(n_mu + 1) * group);
    int s_row = ws.add(sizeof(AdjRow) * 2 * (size_t)n_mu * group);
    int s_acc = ws.add(2 * sizeof(double) * pg * Q);
    int s_part = ws.add(g_flux ? 2 * cube_b : 0);
    int s_buf = ws.add(buf_b), s_bufd = ws.add(buf_b);
    // no flux or tot gradients: one zero array stands in for both, and the continuum
    // rows, which enter only flux and tot, get no pass
    const bool bconv_only = (g_flux == nullptr);
    int s_zero = ws.add(bconv_only ? g_b : 0);
    int s_inv = ws.add(row_b);
    int rc = ws.commit();
    if (rc) return rc;
#define STAGE(dst, src, bytes, slot)                                                           \
    dst = (decltype(dst))stage_in(ctx, mem, src, bytes, ws.get<void>(slot), &rc);             \
    if (rc) return rc;
    const double *d_wave, *d_qn, *d_qs, *d_sn, *d_fn, *d_ss, *d_fs, *d_temp, *d_bi, *d_delta, *d_limb, *d_lb;
    const int *d_region;
    const double *d_gf, *d_gb, *d_gt;
    STAGE(d_wave, wave, row_b, s_wave);
    STAGE(d_qn, cubes->q_norm, cube_b, s_c[0]);
    STAGE(d_qs, cubes->q_sed, cube_b, s_c[1]);
    STAGE(d_sn, cubes->spot_norm, cube_b, s_c[2]);
    STAGE(d_fn, cubes->fac_norm, cube_b, s_c[3]);
    STAGE(d_ss, cubes->spot_sed, row_b, s_c[4]);
    STAGE(d_fs, cubes->fac_sed, row_b, s_c[5]);
    STAGE(d_temp, temp, map_b, s_temp);
    STAGE(d_bi, bi, map_b, s_bi);
    STAGE(d_delta, maps->delta, sizeof(double) * gm, s_m[0]);
    STAGE(d_limb, maps->limb, sizeof(double) * gm, s_m[1]);
    STAGE(d_lb, maps->lb, sizeof(double) * gm, s_m[2]);
    STAGE(d_region, maps->region, sizeof(int) * gm, s_m[3]);
    STAGE(d_gf, g_flux, g_b, s_g[0]);
    STAGE(d_gb, g_bconv, g_b, s_g[1]);
    STAGE(d_gt, g_tot, g_b, s_g[2]);
#undef STAGE
    if (bconv_only) {
        SOAP_CUDA(ctx, cudaMemsetAsync(ws.get<void>(s_zero), 0, g_b, ctx->stream));
        d_gf = d_gt = ws.get<double>(s_zero);
    }
    double *o_qn = host ? ws.get<double>(s_o[0]) : grad_q_norm;
    double *o_qs = host ? ws.get<double>(s_o[1]) : grad_q_sed;
    double *o_sn = host ? ws.get<double>(s_o[2]) : grad_spot_norm;
    double *o_fn = host ? ws.get<double>(s_o[3]) : grad_fac_norm;
    double *o_ss = host ? ws.get<double>(s_o[4]) : grad_spot_sed;
    double *o_fs = host ? ws.get<double>(s_o[5]) : grad_fac_sed;
    double *o_lm = host ? ws.get<double>(s_o[6]) : grad_limb;
    double *o_dl = host ? ws.get<double>(s_o[7]) : grad_delta;
    double *d_buf = ws.get<double>(s_buf), *d_bufd = ws.get<double>(s_bufd);
    double *d_inv = ws.get<double>(s_inv);
    if (n_phase == 0) {
        for (double *o : {o_qn, o_qs, o_sn, o_fn})
            SOAP_CUDA(ctx, cudaMemsetAsync(o, 0, cube_b, ctx->stream));
        SOAP_CUDA(ctx, cudaMemsetAsync(o_ss, 0, row_b, ctx->stream));
        SOAP_CUDA(ctx, cudaMemsetAsync(o_fs, 0, row_b, ctx->stream));
        SOAP_CUDA(ctx, cudaMemsetAsync(o_lm, 0, sizeof(double) * gm, ctx->stream));
        SOAP_CUDA(ctx, cudaMemsetAsync(o_dl, 0, sizeof(double) * gm, ctx->stream));
    } else {
        AdjArgs A;
        A.n = n;
        A.n_eff = n_eff;
        A.n_mu = n_mu;
        A.Q = Q;
        A.gm = gm;
        A.lam = d_wave;
        A.inv = d_inv;
        A.q_norm = d_qn;
        A.q_sed = d_qs;
        A.spot_norm = d_sn;
        A.fac_norm = d_fn;
        A.spot_sed = d_ss;
        A.fac_sed = d_fs;
        A.lb = d_lb;
        A.step = step;
        A.solar = act->solar;
        A.t_norm_fac = (int)(act->t_star + act->t_diff_fac + 0.9 - 216.8);
        A.geo = ws.get<AdjGeo>(s_geo);
        A.cell = ws.get<int>(s_cell);
        A.fb = ws.get<double>(s_fb);
        A.ent = ws.get<AdjEnt>(s_ent);
        A.noise = ws.get<AdjNoise>(s_noise);
        A.seg = ws.get<int>(s_seg);
        A.row = ws.get<AdjRow>(s_row);
        A.acc = ws.get<double>(s_acc);
        A.part = ws.get<double>(s_part);
        A.d_qn = o_qn;
        A.d_qs = o_qs;
        A.d_sn = o_sn;
        A.d_fn = o_fn;
        {
            TraceScope ts(ctx, "adjoint_lists");
            k_adj_geo<<<(unsigned)((gm + 127) / 128), 128, 0, ctx->stream>>>(
                gm, d_wave, d_delta, d_limb, d_lb, d_region, n_mu, step, ws.get<AdjGeo>(s_geo),
                ws.get<unsigned long long>(s_key[0]), ws.get<int>(s_val[0]));
            SOAP_LAUNCHED(ctx);
            rc = ranks ? order_cells(ctx, gm, AdjKey{ws.get<unsigned long long>(s_key[0])},
                                     ws.get<unsigned long long>(s_key[1]), ws.get<unsigned long long>(s_sort),
                                     ws.get<int>(s_val[0]), ws.get<int>(s_val[1]))
                       : fir_sort_u64(ctx, gm, ws.get<unsigned long long>(s_key[0]),
                                      ws.get<unsigned long long>(s_key[1]), ws.get<int>(s_val[0]),
                                      ws.get<int>(s_val[1]), ws.get<void>(s_sort), sort_b);
            if (rc) return rc;
            k_adj_inv<<<grid_for(ctx, n_eff, 256), 256, 0, ctx->stream>>>(n_eff, d_wave, d_inv);
            SOAP_LAUNCHED(ctx);
        }
        for (int p0 = 0; p0 < n_phase; p0 += group) {
            const int ph = std::min(group, n_phase - p0);
            const double *p_bi = d_bi + (size_t)p0 * gm;
            A.n_phase = ph;
            A.more = p0 > 0;
            A.temp = d_temp + (size_t)p0 * gm;
            A.gF = d_gf + (size_t)p0 * n;
            A.gB = d_gb + (size_t)p0 * n;
            A.gT = d_gt + (size_t)p0 * n;
            {
                TraceScope ts(ctx, "adjoint_lists");
                k_adj_lists<<<ph, 1024, 0, ctx->stream>>>(gm, n_mu, ws.get<int>(s_val[1]), A.temp, p_bi, A.geo, d_region,
                                                               act->solar, A.t_norm_fac, ws.get<int>(s_cell),
                                                               ws.get<double>(s_fb), ws.get<int>(s_seg), ctx->d_status);
                SOAP_LAUNCHED(ctx);
                k_adj_entries<<<dim3(n_mu, 2, ph), ADJ_THREADS, 0, ctx->stream>>>(
                    gm, n_mu, A.cell, A.fb, A.seg, A.geo, ws.get<AdjEnt>(s_ent), ws.get<AdjNoise>(s_noise),
                    ws.get<AdjRow>(s_row));
                SOAP_LAUNCHED(ctx);
            }
            SOAP_TRACED(ctx, "adjoint_rows",
                        (bconv_only ? k_adj_rows<true> : k_adj_rows<false>)<<<dim3((n + ADJ_SRC - 1) / ADJ_SRC, n_mu),
                                                                              ADJ_THREADS, 0, ctx->stream>>>(A, p_bi));
            SOAP_LAUNCHED(ctx);
            if (bconv_only) {
                SOAP_CUDA(ctx, cudaMemsetAsync(o_ss, 0, row_b, ctx->stream));
                SOAP_CUDA(ctx, cudaMemsetAsync(o_fs, 0, row_b, ctx->stream));
            } else {
                SOAP_TRACED(ctx, "adjoint_continuum",
                            k_adj_continuum<<<dim3((n + ADJ_THREADS - 1) / ADJ_THREADS, n_mu), ADJ_THREADS, 0, ctx->stream>>>(
                                A, p_bi));
                SOAP_LAUNCHED(ctx);
                k_adj_sum_rows<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(n, n_mu, A.more, A.part, o_ss, o_fs);
                SOAP_LAUNCHED(ctx);
            }
            SOAP_CUDA(ctx, cudaMemsetAsync(d_buf, 0, buf_b, ctx->stream));
            SOAP_CUDA(ctx, cudaMemsetAsync(d_bufd, 0, buf_b, ctx->stream));
            SOAP_CUDA(ctx, cudaMemsetAsync(A.acc, 0, 2 * sizeof(double) * pg * Q, ctx->stream));
            SOAP_TRACED(ctx, "adjoint_limb",
                        (bconv_only ? k_adj_limb<true> : k_adj_limb<false>)<<<dim3(n_mu, ph, Q), ADJ_THREADS, 0,
                                                                              ctx->stream>>>(A, p_bi));
            SOAP_LAUNCHED(ctx);
            k_adj_limb_cells<<<dim3((unsigned)((gm + 255) / 256), ph), 256, 0, ctx->stream>>>(A, d_limb, d_buf, d_bufd);
            SOAP_LAUNCHED(ctx);
            k_adj_sum_phases<<<grid_for(ctx, gm, 256), 256, 0, ctx->stream>>>(ph, gm, A.more, d_buf, o_lm);
            SOAP_LAUNCHED(ctx);
            k_adj_sum_phases<<<grid_for(ctx, gm, 256), 256, 0, ctx->stream>>>(ph, gm, A.more, d_bufd, o_dl);
            SOAP_LAUNCHED(ctx);
        }
    }
    if (host) {
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_q_norm, o_qn, cube_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_q_sed, o_qs, cube_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_spot_norm, o_sn, cube_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_fac_norm, o_fn, cube_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_spot_sed, o_ss, row_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_fac_sed, o_fs, row_b, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_limb, o_lm, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_delta, o_dl, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return check_status(ctx, "soapgb_phase_integrate_adjoint");
    }
    return SOAPGB_OK;
}
