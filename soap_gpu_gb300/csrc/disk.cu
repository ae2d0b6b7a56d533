// a3-a7: disk maps and the quiet-star disk integration.
//
// Reference: SOAP_initialize.cu:297-395 (itot) with fast_shift / fast_interp_new /
// fast_sum at :117-176.  The reference launches three kernels per visible cell
// (about 3 x 70,675 launches at G = 300) and scatters each cell into a scratch
// spectrum.  Here one launch sums all cells: every thread owns output pixels and
// gathers, for each cell in iy-major order, the source interval that covers the
// pixel (the interval-owning form of the scatter; see soap_owner()).
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"
#include "fir.cuh"
#include "plain64.cuh"

using namespace soapgb;

// --------------------------------------------------------------------------
// a3: maps.  omega_velo (per iz) and sin(incl) come from the host, computed with
// the same libm calls as the reference's host loop; the rest is exact IEEE
// arithmetic, one rounding per operation.
// --------------------------------------------------------------------------
__global__ void k_disk_maps(int grid, const double *__restrict__ omega_velo, double sin_incl,
                            double delta_grid, double u1, double u2, int n_mu,
                            const double *__restrict__ mu_b, double lb0, double lb1, double lb2,
                            double lb3, double *delta_m, double *limb_m, double *mu_m,
                            int *region_m, double *lb_m) {
    long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long gm = (long long)grid * grid;
    if (k >= gm) return;
    int iy = (int)(k / grid), iz = (int)(k % grid);
    double y = __dadd_rn(-1., __dmul_rn((double)iy, delta_grid));
    double z = __dadd_rn(-1., __dmul_rn((double)iz, delta_grid));
    double delta = __dmul_rn(__dmul_rn(y, omega_velo[iz]), sin_incl);
    double d = -999.0, lm = -999.0, mu = -999.0, lb = -999.0;
    int reg = 0;
    double yz = __dadd_rn(__dmul_rn(y, y), __dmul_rn(z, z));
    if (yz <= 1.) {
        double r = __dsqrt_rn(__dsub_rn(1., yz));
        double om = __dsub_rn(1., r);
        lm = __dsub_rn(__dsub_rn(1., __dmul_rn(u1, om)), __dmul_rn(__dmul_rn(u2, om), om));
        lb = __dadd_rn(__dadd_rn(__dadd_rn(lb0, __dmul_rn(lb1, r)), __dmul_rn(__dmul_rn(lb2, r), r)),
                       __dmul_rn(__dmul_rn(__dmul_rn(lb3, r), r), r));
        reg = n_mu - 1;
        for (int b = 0; b < n_mu - 1; ++b)
            if (r > mu_b[b]) { reg = b; break; }
        d = delta;
        mu = r;
    }
    delta_m[k] = d;
    limb_m[k] = lm;
    mu_m[k] = mu;
    region_m[k] = reg;
    lb_m[k] = lb;
}

// --------------------------------------------------------------------------
// Ordered stream compaction: idx_out[list][...] = positions i (ascending) with
// lo <= key[list][i] <= hi.  One block of 1024 threads per list.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_compact(const double *__restrict__ key, long long key_stride,
                                                  int n, double lo, double hi, int *idx_out,
                                                  int *count_out) {
    const double *kk = key + (long long)blockIdx.x * key_stride;
    int *out = idx_out + (long long)blockIdx.x * n;
    __shared__ int warp_tot[32];
    __shared__ int base;
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int start = 0; start < n; start += blockDim.x) {
        int i = start + threadIdx.x;
        bool p = false;
        if (i < n) {   // lo <= v <= hi by integer compares of the ordered bit patterns
            unsigned long long v = soap_ord64(kk[i]);
            p = (v >= soap_ord64(lo)) && (v <= soap_ord64(hi));
        }
        unsigned m = __ballot_sync(0xffffffffu, p);
        int pre = __popc(m & ((1u << lane) - 1u));
        if (lane == 0) warp_tot[w] = __popc(m);
        __syncthreads();
        if (w == 0) {
            int v = (lane < nw) ? warp_tot[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                int t = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += t;
            }
            warp_tot[lane] = v;
        }
        __syncthreads();
        int woff = (w == 0) ? 0 : warp_tot[w - 1];
        if (p) out[base + woff + pre] = i;
        __syncthreads();
        if (threadIdx.x == 0) base += warp_tot[nw - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) count_out[blockIdx.x] = base;
}

namespace soapgb {
int compact_cells(soapgb_ctx *ctx, int n_lists, int cells_per_list, const double *key, double lo,
                  double hi, int key_stride, int *idx_out, int *count_out) {
    SOAP_TRACED(ctx, "compact", k_compact<<<n_lists, 1024, 0, ctx->stream>>>(key, key_stride, cells_per_list, lo, hi, idx_out,
                                                  count_out));
    SOAP_LAUNCHED(ctx);
    return SOAPGB_OK;
}
}  // namespace soapgb

// --------------------------------------------------------------------------
// a4-a7 plain FP64: per-pixel gather over all visible cells, in map order (plain64.cuh:
// the reference's expression with one IEEE rounding per operation, so the sum is bit-equal
// to a sequential CPU loop over cells).
// --------------------------------------------------------------------------
__device__ __forceinline__ double soap_cell_value(long long j, int n_eff, const double *__restrict__ lam,
                                                  const double *__restrict__ row, double delta,
                                                  double limb, const CellShift &c) {
    if (delta == 0.0) return __dmul_rn(row[j], limb);
    long long i = soap_owner(j, n_eff, c);
    if (i < 0) return 0.0;
    double li = lam[i], li1 = lam[i + 1];
    double ls0 = __dadd_rn(li, __dmul_rn(__dmul_rn(-1.0, li), __dsub_rn(1.0, c.sq)));
    double ls1 = __dadd_rn(li1, __dmul_rn(__dmul_rn(-1.0, li1), __dsub_rn(1.0, c.sq)));
    double s0 = row[i], s1 = row[i + 1];
    double g = __dsub_rn(s1, s0);
    double dd = __dsub_rn(ls1, ls0);
    double t = __dmul_rn(__ddiv_rn(g, dd), __dsub_rn(lam[j], ls0));
    return __dmul_rn(__dadd_rn(s0, t), limb);
}

__global__ void __launch_bounds__(64) k_plain_cells(long long gm, int n_eff, const double *__restrict__ lam,
                                                   const double *__restrict__ delta_m, double step,
                                                   PlainGeo *__restrict__ geo) {
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= gm) return;
    const double l0 = lam[0], l1 = lam[n_eff - 1], d = (l1 - l0) / (double)(n_eff - 1);
    const CellShift c = soap_cell_shift(delta_m[k], l0, step);
    PlainGeo &g = geo[k];
    const double u = __dsub_rn(1.0, c.sq), F = 1.0 + c.fbeta;
    g.sq = c.sq;
    g.fbeta = c.fbeta;
    g.off = c.off;
    g.u = u;
    g.iF = 1.0 / F;
    // the reference's x_i carry an error below 2^-51 (3 n + |off|), the tile's z below
    // 2^-50 (n + |off|); a cell near the speed of light searches per pixel
    g.eps = F > 0.5 ? 1.8e-15 * (4.0 * (double)n_eff + 2.0 * fabs(c.off) + 4.0) : 2.0;
    // exact: u is a multiple of 2^-53 (without a table it is not used)
    const double au = fabs(u);
    g.w = au < 0x1p-10 ? (unsigned long long)__double2ll_rn(au * 0x1p+53) << PL_FRAC : 0ULL;
    g.zone = (long long)(g.w >> 53) + 2;
    pl_table(l0, d, c.sq, u, g.tab[0]);
    if (pl_exp(l1 - l1 * u) == g.tab[0].ex) g.tab[1].ex = -1;
    else pl_table(l1, d, c.sq, u, g.tab[1]);
}

namespace soapgb {
int plain_cells(soapgb_ctx *ctx, long long k0, long long k1, int n_eff, const double *d_wave, const double *d_delta,
                double step, PlainGeo *geo) {
    SOAP_TRACED(ctx, "plain_cells", k_plain_cells<<<(unsigned)((k1 - k0 + 63) / 64), 64, 0, ctx->stream>>>(
                                        k1 - k0, n_eff, d_wave, d_delta + k0, step, geo));
    SOAP_LAUNCHED(ctx);
    return SOAPGB_OK;
}
}  // namespace soapgb

// the term of cell c (one owner offset) at the thread's pixel; in: the pixel has an owner, and lanes
// without one must not send their warp the other way
__device__ __forceinline__ double quiet_term(const PlainRec &c, const PlainPix &px, const PlainVal &va,
                                             const unsigned long long *tab, double lj, bool in) {
    const double ls = pl_shifted(c, px), ls1 = __shfl_down_sync(0xffffffffu, ls, 1);
    int k;
    double X, rise;
    if ((pl_interval(c, lj, ls, ls1, k, X) && px.ok) || !in) rise = pl_rise(c, va, tab[k], k, X);
    else rise = pl_rise_plain(va.g, lj, ls, ls1);
    return __dmul_rn(__dadd_rn(va.s0, rise), c.limb);
}

// the thread's source interval and the row's values there, kept while the cells share both
struct QuietAt {
    PlainPix px;
    PlainVal va;
    int row = -1, m = 0;
    __device__ __forceinline__ void move(const PlainRec &c, int n, int n_eff, int j, const double *__restrict__ lam,
                                         const double *__restrict__ cube) {
        if (c.row == row && c.m == m) return;
        row = c.row;
        m = c.m;
        const int i = min(max(j + m, 0), n_eff - 1);
        px.li = lam[i];
        px.lm = soap_sig(px.li);
        px.ok = pl_load(va, cube + (long long)row * n, i, min(i + 1, n_eff - 1));
    }
};

// a cell without one offset for the tile, or at rest
__device__ __forceinline__ double quiet_value(const PlainRec &c, const PlainGeo &g, int j, int n, int n_eff,
                                              const double *__restrict__ lam, const double *__restrict__ cube) {
    CellShift cs;
    cs.sq = g.sq;
    cs.fbeta = g.fbeta;
    cs.off = g.off;
    return soap_cell_value(j, n_eff, lam, cube + (long long)c.row * n, c.flags == PL_STILL ? 0.0 : 1.0, c.limb, cs);
}

// the record of the cell at a position of the list
__device__ __forceinline__ void quiet_stage(int k, const PlainGeo *__restrict__ geo, const double *__restrict__ delta_m,
                                            const double *__restrict__ limb_m, const int *__restrict__ region_m,
                                            int n_mu, int j0, int cnt, double lmid, PlainRec &rec,
                                            unsigned long long *tab, int *status) {
    int row = region_m[k];
    if ((unsigned)row >= (unsigned)n_mu) {   // mu bin outside the cube: report, use bin 0
        atomicExch(status, 21);
        row = 0;
    }
    pl_stage(geo + k, delta_m[k], limb_m[k], row, j0, cnt, lmid, rec, tab);
}

// A block takes PL_TILE pixels, a thread one, all cells of [k0, k1) in order (geo: of cell k0 on; the
// sums of the cells before k0 in out).  Small blocks: 100,000 px are 10.6 blocks per SM.
__global__ void __launch_bounds__(PL_THREADS) k_quiet_plain64(int n, int n_eff, const double *__restrict__ lam,
                                                              const double *__restrict__ cube,
                                                              const int *__restrict__ n_cells_ptr,
                                                              const int *__restrict__ cells, int k0, int k1,
                                                              const PlainGeo *__restrict__ geo,
                                                              const double *__restrict__ delta_m,
                                                              const double *__restrict__ limb_m,
                                                              const int *__restrict__ region_m, int n_mu,
                                                              double *__restrict__ out, int *status) {
    __shared__ PlainRec s_rec[PL_CHUNK];
    __shared__ unsigned long long s_tab[PL_CHUNK][PL_TAB];
    __shared__ int s_cell[PL_CHUNK];
    const int lane = threadIdx.x & 31;
    const int j0 = blockIdx.x * PL_TILE, j = j0 + (threadIdx.x >> 5) * 31 + lane;
    const int cnt = max(1, min(PL_TILE, n_eff - j0));
    const double lmid = lam[min(j0 + cnt / 2, n_eff - 1)];
    const bool mine = j < n_eff && lane != 31;
    const double lj = lam[min(j, n_eff - 1)];
    double sum = k0 > 0 && mine ? out[j] : 0.0;
    QuietAt at;
    int from, to;
    pl_slab(cells, *n_cells_ptr, k0, k1, from, to);
    geo -= k0;
    for (int c0 = from; c0 < to; c0 += PL_CHUNK) {
        const int nc = min(PL_CHUNK, to - c0);
        __syncthreads();
        if (threadIdx.x < nc) {
            const int k = cells[c0 + threadIdx.x];
            s_cell[threadIdx.x] = k;
            quiet_stage(k, geo, delta_m, limb_m, region_m, n_mu, j0, cnt, lmid, s_rec[threadIdx.x], s_tab[threadIdx.x],
                        status);
        }
        __syncthreads();
        for (int t = 0; t < nc; ++t) {
            const PlainRec c = s_rec[t];
            if (c.flags != PL_CONST) {
                if (mine) sum = __dadd_rn(sum, quiet_value(c, geo[s_cell[t]], j, n, n_eff, lam, cube));
                continue;
            }
            at.move(c, n, n_eff, j, lam, cube);
            const double ls = pl_shifted(c, at.px), ls1 = __shfl_down_sync(0xffffffffu, ls, 1);
            // lanes without a pixel here must not send their warp the other way
            const bool in = mine && (unsigned)(j + c.m) <= (unsigned)(n_eff - 2);
            int k;
            double X, rise;
            if ((pl_interval(c, lj, ls, ls1, k, X) && at.px.ok) || !in) rise = pl_rise(c, at.va, s_tab[t][k], k, X);
            else rise = pl_rise_plain(at.va.g, lj, ls, ls1);
            const double r = __dadd_rn(sum, __dmul_rn(__dadd_rn(at.va.s0, rise), c.limb));
            if (in) sum = r;
        }
    }
    if (lane != 31 && j < n) out[j] = mine ? sum : 0.0;
}

// The same sums where the tiles are too few to fill the chip: a cell's term is a chain of some 800
// cycles, which two warps per tile walk one cell after the other.  Here PQ_WARPS warps share a tile.
// They compute the terms of a chunk of cells into shared memory, in groups taken from a counter,
// while one of them adds up the terms of the chunk before, in the cells' order: the additions stay
// those of the sum above.  100 x 100 cells: 6,000 px 3.38 -> 0.96 ms, 20,000 px 3.64 -> 2.31 ms,
// 37,600 px 3.78 -> 2.82 ms.  Above four tiles per SM the other kernel's warps fill the pipes
// (37,800 px: 4.0 ms; 50,000 px 4.2 ms, here 4.1; 100,000 px of 200 x 200 cells 28.0 ms, here 29.9).
constexpr int PQ_WARPS = 16, PQ_STRIPS = PL_TILE / 31, PQ_CHUNK = 64, PQ_GROUP = 4;
struct PlainQuietSmem {   // chunks, double buffered
    double term[2][PQ_STRIPS][PQ_CHUNK][32];
    unsigned long long tab[2][PQ_CHUNK][PL_TAB];
    PlainRec rec[2][PQ_CHUNK];
    int cell[2][PQ_CHUNK];
    double sum[PQ_STRIPS][32];
    int next[2][PQ_STRIPS];   // jobs taken in a step, per strip
};

__global__ void __launch_bounds__(32 * PQ_WARPS, 2) k_quiet_plain64s(
    int n, int n_eff, const double *__restrict__ lam, const double *__restrict__ cube,
    const int *__restrict__ n_cells_ptr, const int *__restrict__ cells, int k0, int k1, const PlainGeo *__restrict__ geo,
    const double *__restrict__ delta_m, const double *__restrict__ limb_m, const int *__restrict__ region_m, int n_mu,
    double *__restrict__ out, int *status) {
    extern __shared__ __align__(16) unsigned char pq_smem[];
    PlainQuietSmem &sh = *reinterpret_cast<PlainQuietSmem *>(pq_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, strip = warp % PQ_STRIPS;
    const int j0 = blockIdx.x * PL_TILE, j = j0 + strip * 31 + lane;
    const int cnt = max(1, min(PL_TILE, n_eff - j0));
    const double lmid = lam[min(j0 + cnt / 2, n_eff - 1)];
    const bool mine = j < n_eff && lane != 31;
    const double lj = lam[min(j, n_eff - 1)];
    int from, to;
    pl_slab(cells, *n_cells_ptr, k0, k1, from, to);
    cells += from;
    geo -= k0;
    const int n_cells = to - from, n_chunk = (n_cells + PQ_CHUNK - 1) / PQ_CHUNK;
    QuietAt at;
    auto stage = [&](int c) {   // the records of chunk c, by one warp
        const int b = c & 1;
        for (int t = lane; t < min(PQ_CHUNK, n_cells - c * PQ_CHUNK); t += 32) {
            const int k = cells[c * PQ_CHUNK + t];
            sh.cell[b][t] = k;
            quiet_stage(k, geo, delta_m, limb_m, region_m, n_mu, j0, cnt, lmid, sh.rec[b][t], sh.tab[b][t], status);
        }
    };
    if (warp < PQ_STRIPS) sh.sum[warp][lane] = k0 > 0 && mine ? out[j] : 0.0;
    if (threadIdx.x < PQ_STRIPS) sh.next[0][threadIdx.x] = 0;
    if (warp == 0) stage(0);
    // step c: the sum over chunk c - 1, the records of chunk c + 1 (strip 0), the terms of chunk c
    for (int c = 0; c <= n_chunk; ++c) {
        __syncthreads();
        const int b = c & 1;
        if (threadIdx.x < PQ_STRIPS) sh.next[b ^ 1][threadIdx.x] = 0;
        const int nt = c < n_chunk ? min(PQ_CHUNK, n_cells - c * PQ_CHUNK) : 0;
        const int jobs = 2 + (nt + PQ_GROUP - 1) / PQ_GROUP;
        while (true) {
            int job = 0;
            if (lane == 0) job = atomicAdd(&sh.next[b][strip], 1);
            job = __shfl_sync(0xffffffffu, job, 0);
            if (job >= jobs) break;
            if (job == 0) {
                if (c == 0) continue;
                const int np = min(PQ_CHUNK, n_cells - (c - 1) * PQ_CHUNK);
                double sum = sh.sum[strip][lane];
#pragma unroll 4
                for (int t = 0; t < np; ++t) sum = __dadd_rn(sum, sh.term[b ^ 1][strip][t][lane]);
                sh.sum[strip][lane] = sum;
            } else if (job == 1) {
                if (strip == 0 && c + 1 < n_chunk) stage(c + 1);
            } else {
                const int t0 = (job - 2) * PQ_GROUP, t1 = min(t0 + PQ_GROUP, nt);
                for (int t = t0; t < t1; ++t) {
                    const PlainRec r = sh.rec[b][t];
                    double v = 0.0;   // a pixel without an owner adds zero: the sum's bits stay
                    if (r.flags != PL_CONST) {
                        if (mine) v = quiet_value(r, geo[sh.cell[b][t]], j, n, n_eff, lam, cube);
                    } else {
                        at.move(r, n, n_eff, j, lam, cube);
                        const bool in = mine && (unsigned)(j + r.m) <= (unsigned)(n_eff - 2);
                        const double term = quiet_term(r, at.px, at.va, sh.tab[b][t], lj, in);
                        if (in) v = term;
                    }
                    sh.term[b][strip][t][lane] = v;
                }
            }
        }
    }
    __syncthreads();
    if (warp < PQ_STRIPS && lane != 31 && j < n) out[j] = mine ? sh.sum[strip][lane] : 0.0;
}

// --------------------------------------------------------------------------
// host side
// --------------------------------------------------------------------------
namespace soapgb {
void disk_omega_host(const soapgb_star *st, std::vector<double> &ov, double &sin_incl);
int disk_maps_launch(soapgb_ctx *ctx, const soapgb_star *star, int n_mu, const double *d_mu, const double *d_ov,
                     double sin_incl, double *delta, double *limb, double *mu, int *region, double *lb);
}  // namespace soapgb

static void host_omega_velo(const soapgb_star *st, std::vector<double> &ov, double &sin_incl) {
    // SOAP_initialize.cu:308-351, host libm like the reference
    double incl = st->incl * SOAP_PI / 180.;
    double theta_grid = 180.0 / st->grid;
    double omega0 = 360.0 / st->period;
    double omega1 = omega0 * st->omega_ratio;
    ov.resize(st->grid);
    for (int iz = 0; iz < st->grid; ++iz) {
        double theta_z = -90.0 + iz * theta_grid;
        double s = sin(theta_z * SOAP_PI / 180);
        ov[iz] = (omega0 + omega1 * (s * s)) * SOAP_PI / (180 * 24 * 3600) * st->radius_km;
    }
    sin_incl = sin(incl);
}

namespace soapgb {
// the per-row rotation constants of a star's grid (host libm), for disk_maps_launch
void disk_omega_host(const soapgb_star *st, std::vector<double> &ov, double &sin_incl) {
    host_omega_velo(st, ov, sin_incl);
}

// the disk maps of one star from constants already on the device (no host memory read)
int disk_maps_launch(soapgb_ctx *ctx, const soapgb_star *star, int n_mu, const double *d_mu, const double *d_ov,
                     double sin_incl, double *delta, double *limb, double *mu, int *region, double *lb) {
    const int G = star->grid;
    const long long gm = (long long)G * G;
    const double *c = star->lb;
    SOAP_TRACED(ctx, "disk_maps", k_disk_maps<<<grid_for(ctx, gm, 256), 256, 0, ctx->stream>>>(
        G, d_ov, sin_incl, 2. / G, star->u1, star->u2, n_mu, d_mu, c[0], c[1], c[2], c[3], delta, limb, mu, region,
        lb));
    SOAP_LAUNCHED(ctx);
    return SOAPGB_OK;
}
}  // namespace soapgb

extern "C" int soapgb_disk_maps(soapgb_ctx *ctx, const soapgb_star *star, int n_mu,
                                const double *mu_boundary, int mem, soapgb_maps *maps_out) {
    if (!ctx || !star || !maps_out) return SOAPGB_ERR_ARG;
    if (star->grid <= 0 || star->grid > 20000 || n_mu < 1 || (n_mu > 1 && !mu_boundary))
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_disk_maps: bad grid %d / n_mu %d", star->grid, n_mu);
    SOAP_DEVICE(ctx);
    int G = star->grid;
    long long gm = (long long)G * G;
    std::vector<double> ov;
    double sin_incl;
    host_omega_velo(star, ov, sin_incl);
    Workspace ws(ctx);
    int s_ov = ws.add(sizeof(double) * G);
    int s_mu = ws.add(sizeof(double) * (n_mu > 1 ? n_mu - 1 : 1));
    int s_out[5];
    for (int q = 0; q < 5; ++q) s_out[q] = ws.add(mem == SOAPGB_HOST ? sizeof(double) * gm : 0);
    int rc = ws.commit();
    if (rc) return rc;
    double *d_ov = ws.get<double>(s_ov);
    SOAP_CUDA(ctx, cudaMemcpyAsync(d_ov, ov.data(), sizeof(double) * G, cudaMemcpyHostToDevice, ctx->stream));
    const double *d_mu = mu_boundary;
    if (n_mu > 1 && mem == SOAPGB_HOST) {
        d_mu = ws.get<double>(s_mu);
        SOAP_CUDA(ctx, cudaMemcpyAsync((void *)d_mu, mu_boundary, sizeof(double) * (n_mu - 1),
                                       cudaMemcpyHostToDevice, ctx->stream));
    }
    double *o_delta = maps_out->delta, *o_limb = maps_out->limb, *o_mu = maps_out->mu, *o_lb = maps_out->lb;
    int *o_reg = maps_out->region;
    if (mem == SOAPGB_HOST) {
        o_delta = ws.get<double>(s_out[0]);
        o_limb = ws.get<double>(s_out[1]);
        o_mu = ws.get<double>(s_out[2]);
        o_lb = ws.get<double>(s_out[3]);
        o_reg = ws.get<int>(s_out[4]);
    }
    if (!o_delta || !o_limb || !o_mu || !o_lb || !o_reg)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_disk_maps: null map pointer");
    const double *lb = star->lb;
    SOAP_TRACED(ctx, "disk_maps", k_disk_maps<<<grid_for(ctx, gm, 256), 256, 0, ctx->stream>>>(
        G, d_ov, sin_incl, 2. / G, star->u1, star->u2, n_mu, d_mu, lb[0], lb[1], lb[2], lb[3], o_delta, o_limb,
        o_mu, o_reg, o_lb));
    SOAP_LAUNCHED(ctx);
    if (mem == SOAPGB_HOST) {
        SOAP_CUDA(ctx, cudaMemcpyAsync(maps_out->delta, o_delta, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(maps_out->limb, o_limb, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(maps_out->mu, o_mu, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(maps_out->lb, o_lb, sizeof(double) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(maps_out->region, o_reg, sizeof(int) * gm, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return SOAPGB_OK;
}

extern "C" int soapgb_quiet_disk(soapgb_ctx *ctx, int form, int n, int n_eff, const double *wave,
                                 const double *cube, int n_mu, int grid, const double *delta,
                                 const double *limb, const int *region, double step, int mem,
                                 double *sum_out) {
    if (!ctx) return SOAPGB_ERR_ARG;
    if (n < 2 || n_eff < 2 || n_eff > n || n_mu < 1 || grid < 1 || !wave || !cube || !delta || !limb ||
        !region || !sum_out || !(step > 0))
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_quiet_disk: bad arguments (n=%d n_eff=%d)", n, n_eff);
    if (form != SOAPGB_PLAIN64 && form != SOAPGB_FAST64 && form != SOAPGB_FAST32)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_quiet_disk: unknown form %d", form);
    SOAP_DEVICE(ctx);
    long long gm = (long long)grid * grid;
    bool host = (mem == SOAPGB_HOST);
    Workspace ws(ctx);
    int s_wave = ws.add(host ? sizeof(double) * n : 0);
    int s_cube = ws.add(host ? sizeof(double) * (size_t)n * n_mu : 0);
    int s_delta = ws.add(host ? sizeof(double) * gm : 0);
    int s_limb = ws.add(host ? sizeof(double) * gm : 0);
    int s_region = ws.add(host ? sizeof(int) * gm : 0);
    int s_out = ws.add(host ? sizeof(double) * n : 0);
    int s_cells = ws.add(sizeof(int) * gm);
    int s_count = ws.add(sizeof(int));
    FirPlanSizes fp = fir_plan_sizes(form, n, n_mu, gm, false, 1);
    int s_fir = ws.add(fp.bytes);
    int rc = ws.commit();
    if (rc) return rc;
    const double *d_wave = (const double *)stage_in(ctx, mem, wave, sizeof(double) * n, ws.get<void>(s_wave), &rc);
    if (rc) return rc;
    const double *d_cube = (const double *)stage_in(ctx, mem, cube, sizeof(double) * (size_t)n * n_mu, ws.get<void>(s_cube), &rc);
    if (rc) return rc;
    const double *d_delta = (const double *)stage_in(ctx, mem, delta, sizeof(double) * gm, ws.get<void>(s_delta), &rc);
    if (rc) return rc;
    const double *d_limb = (const double *)stage_in(ctx, mem, limb, sizeof(double) * gm, ws.get<void>(s_limb), &rc);
    if (rc) return rc;
    const int *d_region = (const int *)stage_in(ctx, mem, region, sizeof(int) * gm, ws.get<void>(s_region), &rc);
    if (rc) return rc;
    double *d_out = host ? ws.get<double>(s_out) : sum_out;
    int *d_cells = ws.get<int>(s_cells);
    int *d_count = ws.get<int>(s_count);
    if (form == SOAPGB_PLAIN64) {
        // visible cells in map order (limb map is -999 elsewhere)
        rc = compact_cells(ctx, 1, (int)gm, d_limb, -998.0, 1e300, (int)gm, d_cells, d_count);
        if (rc) return rc;
        PlainGeo *geo = ws.get<PlainGeo>(s_fir);
        const int ntile = (n + PL_TILE - 1) / PL_TILE;
        for (long long k0 = 0; k0 < gm; k0 += PL_SLAB) {
            const long long end = std::min(gm, k0 + PL_SLAB);
            const int k1 = end < gm ? (int)end : INT_MAX;
            rc = plain_cells(ctx, k0, end, n_eff, d_wave, d_delta, step, geo);
            if (rc) return rc;
            if (ntile <= 4 * ctx->num_sms) {
                SOAP_CUDA(ctx, soap_allow_smem(k_quiet_plain64s, sizeof(PlainQuietSmem)));
                SOAP_TRACED(ctx, "quiet_plain64",
                            k_quiet_plain64s<<<ntile, 32 * PQ_WARPS, sizeof(PlainQuietSmem), ctx->stream>>>(
                                n, n_eff, d_wave, d_cube, d_count, d_cells, (int)k0, k1, geo, d_delta, d_limb, d_region,
                                n_mu, d_out, ctx->d_status));
            } else {
                SOAP_TRACED(ctx, "quiet_plain64", k_quiet_plain64<<<ntile, PL_THREADS, 0, ctx->stream>>>(
                    n, n_eff, d_wave, d_cube, d_count, d_cells, (int)k0, k1, geo, d_delta, d_limb, d_region, n_mu, d_out,
                    ctx->d_status));
            }
            SOAP_LAUNCHED(ctx);
        }
    } else {
        FirQuietArgs qa;
        qa.n = n;
        qa.n_eff = n_eff;
        qa.wave = d_wave;
        qa.cube = d_cube;
        qa.n_mu = n_mu;
        qa.gm = gm;
        qa.delta = d_delta;
        qa.limb = d_limb;
        qa.region = d_region;
        qa.step = step;
        qa.out = d_out;
        rc = fir_quiet(ctx, form, qa, ws.get<char>(s_fir), fp);
        if (rc) return rc;
    }
    if (host) {
        SOAP_CUDA(ctx, cudaMemcpyAsync(sum_out, d_out, sizeof(double) * n, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return host ? check_status(ctx, "soapgb_quiet_disk") : SOAPGB_OK;
}
