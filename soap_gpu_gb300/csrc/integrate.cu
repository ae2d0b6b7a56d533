// a11-a12: per-phase active-region integration.
//
// Reference: SOAP_integration.cu:392-447 (spot_integrate: a host loop over all
// G*G cells issuing eight FP64 kernels per active cell -- shift, three
// interpolations, intensity, flux/bconv/tot) and :285-323 (the accumulation
// kernels).  Here one launch covers every phase: block (x, p) owns a pixel range
// of phase p and gathers all of the phase's active cells, in map order, into
// register accumulators.
#include <algorithm>
#include <cmath>

#include "internal.cuh"
#include "fir.cuh"
#include "plain64.cuh"
#include "planck.cuh"

using namespace soapgb;

// One cell's interpolation geometry at pixel j (shared by the three cubes).
struct CellAt {
    long long i;   // owner source index, -1 if none
    double dd;     // l'_{i+1} - l'_i
    double dl;     // l_j - l'_i
};

__device__ __forceinline__ CellAt soap_cell_at(long long j, int n_eff, const double *__restrict__ lam,
                                               const CellShift &c) {
    CellAt r;
    r.i = soap_owner(j, n_eff, c);
    r.dd = 0.0;
    r.dl = 0.0;
    if (r.i >= 0) {
        double li = lam[r.i], li1 = lam[r.i + 1];
        double ls0 = __dadd_rn(li, __dmul_rn(__dmul_rn(-1.0, li), __dsub_rn(1.0, c.sq)));
        double ls1 = __dadd_rn(li1, __dmul_rn(__dmul_rn(-1.0, li1), __dsub_rn(1.0, c.sq)));
        r.dd = __dsub_rn(ls1, ls0);
        r.dl = __dsub_rn(lam[j], ls0);
    }
    return r;
}

__device__ __forceinline__ double soap_lerp_at(const CellAt &a, long long j, const double *__restrict__ row,
                                               double delta, double limb) {
    if (delta == 0.0) return __dmul_rn(row[j], limb);
    if (a.i < 0) return 0.0;
    double s0 = row[a.i], s1 = row[a.i + 1];
    double t = __dmul_rn(__ddiv_rn(__dsub_rn(s1, s0), a.dd), a.dl);
    return __dmul_rn(__dadd_rn(s0, t), limb);
}

// one active cell's three rows and intensity
struct PhaseCell {
    int k;          // map index
    int type;       // 0 spot, 1 facula
    int unit;       // 1: the intensity is the continuum row itself, 0: scale x the row, -1: a Planck ratio
    double scale;   // 1 + LB
    PlainFactor by; // the limb factor
};

// the record of active cell k of temperature T and type b
__device__ __forceinline__ PhaseCell phase_cell(int k, double T, double b, const double *__restrict__ lb_m,
                                                const double *__restrict__ limb_m, int solar, int t_norm_fac) {
    PhaseCell a;
    a.k = k;
    a.type = (b == 0.0) ? 0 : 1;
    a.scale = 1.0;
    if (a.type == 0) {
        a.unit = ((double)(int)T == T) ? 1 : -1;
    } else if (solar) {
        a.unit = ((double)t_norm_fac == T) ? 1 : -1;
    } else {
        a.unit = 0;
        a.scale = __dadd_rn(1.0, lb_m[k]);
    }
    a.by = pl_factor(limb_m[k]);
    return a;
}

// The plain form: block (x, p) sums phase p's active cells, in map order, over a tile of
// pixels (plain64.cuh); three rows per cell; the cells [k0, k1), geo of cell k0 on, the sums of those
// before in flux, bconv and tot.  INT: the five products of a cell and pixel on the
// integer pipes (18.4 -> 13 FP64 instructions, 285 -> 440 in all), which pays where the FP64 pipe
// is the bound: 5 phases of 200 x 200 cells and 100,000 px, 8.2 -> 6.1 ms; 11 phases of 151 x 151
// and 60,001 px, 7.0 -> 5.2 ms; at 6.4 blocks per SM 0.340 -> 0.317 ms.  With fewer the pipe waits
// for the chains of the few warps, which the integer products lengthen (5.3 blocks per SM: 0.53 ->
// 0.59 ms; 2.1: 1.45 -> 1.81 ms).
template <bool INT>
__global__ void __launch_bounds__(PL_THREADS) k_phase_plain64(
    int n, int n_eff, const double *__restrict__ lam, const double *__restrict__ q_norm,
    const double *__restrict__ q_sed, const double *__restrict__ spot_norm, const double *__restrict__ fac_norm,
    const double *__restrict__ spot_sed, const double *__restrict__ fac_sed, int max_cells,
    const int *__restrict__ cells, const int *__restrict__ counts, int k0, int k1, const double *__restrict__ temp,
    const double *__restrict__ bi, const PlainGeo *__restrict__ geo, const double *__restrict__ delta_m,
    const double *__restrict__ limb_m, const double *__restrict__ lb_m, const int *__restrict__ region_m,
    long long gm, int solar, int t_star, int t_diff_fac, double *__restrict__ flux, double *__restrict__ bconv,
    double *__restrict__ tot, long long out_stride, int n_mu, int *status) {
    __shared__ PlainRec s_rec[PL_CHUNK];
    __shared__ unsigned long long s_tab[PL_CHUNK][PL_TAB];
    __shared__ PhaseCell s_cell[PL_CHUNK];
    const int p = blockIdx.y, lane = threadIdx.x & 31;
    const int j0 = blockIdx.x * PL_TILE, j = j0 + (threadIdx.x >> 5) * 31 + lane;
    const int cnt = max(1, min(PL_TILE, n_eff - j0));
    const int *pc = cells + (long long)p * max_cells;
    int from, to;
    pl_slab(pc, counts[p], k0, k1, from, to);
    geo -= k0;
    const double *pt = temp + (long long)p * gm;
    const double *pb = bi + (long long)p * gm;
    const double lmid = lam[min(j0 + cnt / 2, n_eff - 1)];
    const int t_norm_fac = (int)(t_star + t_diff_fac + 0.9 - 216.8);
    const bool mine = j < n_eff && lane != 31;
    const int jc = min(j, n_eff - 1);
    const double lj = lam[jc], ssed = spot_sed[jc], fsed = fac_sed[jc];
    const PlainFactor by_s = pl_factor(ssed), by_f = pl_factor(fsed);
    double fx = 0.0, bc = 0.0, tt = 0.0;
    if (k0 > 0 && mine) {
        const long long o = (long long)p * out_stride + j;
        fx = flux[o];
        bc = bconv[o];
        tt = tot[o];
    }
    PlainPix px;
    PlainVal va[3];
    int row_now = -1, m_now = 0, type_now = 0;
    for (int c0 = from; c0 < to; c0 += PL_CHUNK) {
        const int nc = min(PL_CHUNK, to - c0);
        __syncthreads();
        if (threadIdx.x < nc) {
            const int k = pc[c0 + threadIdx.x];
            int row = region_m[k];
            if ((unsigned)row >= (unsigned)n_mu) {   // mu bin outside the cube: report, use bin 0
                atomicExch(status, 21);
                row = 0;
            }
            const PhaseCell a = phase_cell(k, pt[k], pb[k], lb_m, limb_m, solar, t_norm_fac);
            s_cell[threadIdx.x] = a;
            pl_stage(geo + k, delta_m[k], limb_m[k], row, j0, cnt, lmid, s_rec[threadIdx.x], s_tab[threadIdx.x]);
        }
        __syncthreads();
        for (int t = 0; t < nc; ++t) {
            const PlainRec c = s_rec[t];
            const PhaseCell a = s_cell[t];
            const long long off = (long long)c.row * n;
            const double *an = (a.type == 0 ? spot_norm : fac_norm) + off;
            double q, s, v;
            bool fast = false;           // q and v are moderate, or zero where the pixel has no owner
            bool none = false;           // no owner
            if (c.flags != PL_CONST) {   // the pixel itself, or an owner search per pixel
                const PlainGeo &g = geo[a.k];
                CellShift cs;
                cs.sq = g.sq;
                cs.fbeta = g.fbeta;
                cs.off = g.off;
                const double d = c.flags == PL_STILL ? 0.0 : 1.0;
                CellAt at;
                at.i = -1;
                if (d != 0.0) at = soap_cell_at(jc, n_eff, lam, cs);
                q = soap_lerp_at(at, jc, q_norm + off, d, c.limb);
                s = soap_lerp_at(at, jc, q_sed + off, d, c.limb);
                v = soap_lerp_at(at, jc, an, d, c.limb);
            } else {
                if (c.row != row_now || c.m != m_now || a.type != type_now) {
                    row_now = c.row;
                    m_now = c.m;
                    type_now = a.type;
                    const int i = min(max(j + c.m, 0), n_eff - 1), i1 = min(i + 1, n_eff - 1);
                    px.li = lam[i];
                    px.lm = soap_sig(px.li);
                    const bool ok0 = pl_load(va[0], q_norm + off, i, i1), ok1 = pl_load(va[1], q_sed + off, i, i1);
                    px.ok = pl_load(va[2], an, i, i1) && ok0 && ok1;
                }
                const double ls = pl_shifted(c, px), ls1 = __shfl_down_sync(0xffffffffu, ls, 1);
                // lanes without a pixel here must not send their warp the other way
                const bool in = mine && (unsigned)(j + c.m) <= (unsigned)(n_eff - 2);
                int k;
                double X, x[3];
                if ((pl_interval(c, lj, ls, ls1, k, X) && px.ok) || !in) {
                    const unsigned long long rec = s_tab[t][k];
#pragma unroll
                    for (int r = 0; r < 3; ++r) x[r] = pl_rise(c, va[r], rec, k, X);
                } else {
#pragma unroll
                    for (int r = 0; r < 3; ++r) x[r] = pl_rise_plain(va[r].g, lj, ls, ls1);
                }
#pragma unroll
                for (int r = 0; r < 3; ++r) x[r] = __dadd_rn(va[r].s0, x[r]);
                if constexpr (INT) {
                    bool plain = a.by.hi == 0 || !(soap_moderate(x[0], PL_SPAN) && soap_moderate(x[1], PL_SPAN) &&
                                                   soap_moderate(x[2], PL_SPAN));
                    fast = !plain || !in;
                    none = !in;
                    q = pl_mul(x[0], a.by, plain);
                    s = pl_mul(x[1], a.by, plain);
                    v = pl_mul(x[2], a.by, plain);
                    if (plain && in) {
                        q = pl_mul_plain(x[0], c.limb);
                        s = pl_mul_plain(x[1], c.limb);
                        v = pl_mul_plain(x[2], c.limb);
                    }
                } else {
                    q = __dmul_rn(x[0], c.limb);
                    s = __dmul_rn(x[1], c.limb);
                    v = __dmul_rn(x[2], c.limb);
                }
                q = in ? q : 0.0;
                s = in ? s : 0.0;
                v = in ? v : 0.0;
            }
            double I = a.type == 0 ? ssed : fsed, iq, iv;
            if constexpr (INT) {
                PlainFactor by = a.type == 0 ? by_s : by_f;
                if (a.unit == 0) {
                    bool plain = by.hi == 0 || !soap_moderate(a.scale, PL_SPAN);
                    const double f = I;
                    I = pl_mul(a.scale, by, plain);
                    if (plain) I = pl_mul_plain(a.scale, f);
                    by = pl_factor(I);
                } else if (a.unit < 0) {
                    I = soap_intensity(a.type, pt[a.k], lb_m[a.k], lj, ssed, fsed, solar, t_norm_fac);
                    by = pl_factor(I);
                }
                bool plain = !fast || by.hi == 0;
                iq = pl_mul(q, by, plain);
                iv = pl_mul(v, by, plain);
                if (none) iq = iv = 0.0;   // moderate intensity x 0
                if (plain && !(none && by.hi != 0)) {
                    iq = pl_mul_plain(I, q);
                    iv = pl_mul_plain(v, I);
                }
            } else {
                if (a.unit == 0) I = __dmul_rn(a.scale, I);
                else if (a.unit < 0) I = soap_intensity(a.type, pt[a.k], lb_m[a.k], lj, ssed, fsed, solar, t_norm_fac);
                iq = __dmul_rn(I, q);
                iv = __dmul_rn(v, I);
            }
            fx = __dsub_rn(__dadd_rn(fx, s), iq);
            bc = __dsub_rn(__dadd_rn(bc, q), v);
            tt = __dsub_rn(__dadd_rn(tt, s), iv);
        }
    }
    if (lane == 31 || j >= n) return;
    const long long o = (long long)p * out_stride + j;
    flux[o] = mine ? fx : 0.0;
    bconv[o] = mine ? bc : 0.0;
    tot[o] = mine ? tt : 0.0;
}

// The same sums where the blocks are too few to fill the chip: a cell's terms are a chain of some
// 1000 cycles, which a warp per strip of 31 pixels walks one cell after the other.  Here PS_WARPS
// warps share a tile: they compute the five terms of a chunk's cells into shared memory, cell by
// cell from a counter, while one of them per strip adds up the chunk before, in the cells' order
// (as k_quiet_plain64s).  Two blocks fit an SM: up to there one phase of 200 x 200 cells and 6,000 px
// takes 371 us against 813, 150 x 150 and 18,800 px 295 against 421; above (2.1 blocks per SM, two
// waves) 1142 against 1145, at 3.2 692 against 649.
constexpr long long PS_MAX_PER_SM = 2;   // what an SM holds of it
constexpr int PS_WARPS = 8, PS_STRIPS = PL_TILE / 31, PS_CHUNK = 16;
struct PlainPhaseSmem {   // chunks, double buffered
    double term[2][PS_STRIPS][PS_CHUNK][5][32];   // s, I q, q, v, v I
    unsigned long long tab[2][PS_CHUNK][PL_TAB];
    PlainRec rec[2][PS_CHUNK];
    PhaseCell cell[2][PS_CHUNK];
    double sum[PS_STRIPS][3][32];
    int next[2][PS_STRIPS];   // jobs taken in a step, per strip
};

__global__ void __launch_bounds__(32 * PS_WARPS, 2) k_phase_plain64s(
    int n, int n_eff, const double *__restrict__ lam, const double *__restrict__ q_norm,
    const double *__restrict__ q_sed, const double *__restrict__ spot_norm, const double *__restrict__ fac_norm,
    const double *__restrict__ spot_sed, const double *__restrict__ fac_sed, int max_cells,
    const int *__restrict__ cells, const int *__restrict__ counts, int k0, int k1, const double *__restrict__ temp,
    const double *__restrict__ bi, const PlainGeo *__restrict__ geo, const double *__restrict__ delta_m,
    const double *__restrict__ limb_m, const double *__restrict__ lb_m, const int *__restrict__ region_m,
    long long gm, int solar, int t_star, int t_diff_fac, double *__restrict__ flux, double *__restrict__ bconv,
    double *__restrict__ tot, long long out_stride, int n_mu, int *status) {
    extern __shared__ __align__(16) unsigned char ps_smem[];
    PlainPhaseSmem &sh = *reinterpret_cast<PlainPhaseSmem *>(ps_smem);
    const int p = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, strip = warp % PS_STRIPS;
    const int j0 = blockIdx.x * PL_TILE, j = j0 + strip * 31 + lane;
    const int cnt = max(1, min(PL_TILE, n_eff - j0));
    const int *pc = cells + (long long)p * max_cells;
    int from, to;
    pl_slab(pc, counts[p], k0, k1, from, to);
    pc += from;
    geo -= k0;
    const int n_cells = to - from, n_chunk = (n_cells + PS_CHUNK - 1) / PS_CHUNK;
    const double *pt = temp + (long long)p * gm;
    const double *pb = bi + (long long)p * gm;
    const double lmid = lam[min(j0 + cnt / 2, n_eff - 1)];
    const int t_norm_fac = (int)(t_star + t_diff_fac + 0.9 - 216.8);
    const bool mine = j < n_eff && lane != 31;
    const int jc = min(j, n_eff - 1);
    const double lj = lam[jc], ssed = spot_sed[jc], fsed = fac_sed[jc];
    PlainPix px;
    PlainVal va[3];
    int row_now = -1, m_now = 0, type_now = 0;
    auto stage = [&](int c) {   // the records of chunk c, by one warp
        const int b = c & 1, t = lane;
        if (t >= min(PS_CHUNK, n_cells - c * PS_CHUNK)) return;
        const int k = pc[c * PS_CHUNK + t];
        int row = region_m[k];
        if ((unsigned)row >= (unsigned)n_mu) {   // mu bin outside the cube: report, use bin 0
            atomicExch(status, 21);
            row = 0;
        }
        sh.cell[b][t] = phase_cell(k, pt[k], pb[k], lb_m, limb_m, solar, t_norm_fac);
        pl_stage(geo + k, delta_m[k], limb_m[k], row, j0, cnt, lmid, sh.rec[b][t], sh.tab[b][t]);
    };
    auto terms = [&](const PlainRec &c, const PhaseCell &a, const unsigned long long *tab, double(*to)[32]) {
        const long long off = (long long)c.row * n;
        const double *an = (a.type == 0 ? spot_norm : fac_norm) + off;
        double q, s, v;
        if (c.flags != PL_CONST) {   // the pixel itself, or an owner search per pixel
            const PlainGeo &g = geo[a.k];
            CellShift cs;
            cs.sq = g.sq;
            cs.fbeta = g.fbeta;
            cs.off = g.off;
            const double d = c.flags == PL_STILL ? 0.0 : 1.0;
            CellAt at;
            at.i = -1;
            if (d != 0.0) at = soap_cell_at(jc, n_eff, lam, cs);
            q = soap_lerp_at(at, jc, q_norm + off, d, c.limb);
            s = soap_lerp_at(at, jc, q_sed + off, d, c.limb);
            v = soap_lerp_at(at, jc, an, d, c.limb);
        } else {
            if (c.row != row_now || c.m != m_now || a.type != type_now) {
                row_now = c.row;
                m_now = c.m;
                type_now = a.type;
                const int i = min(max(j + c.m, 0), n_eff - 1), i1 = min(i + 1, n_eff - 1);
                px.li = lam[i];
                px.lm = soap_sig(px.li);
                const bool ok0 = pl_load(va[0], q_norm + off, i, i1), ok1 = pl_load(va[1], q_sed + off, i, i1);
                px.ok = pl_load(va[2], an, i, i1) && ok0 && ok1;
            }
            const double ls = pl_shifted(c, px), ls1 = __shfl_down_sync(0xffffffffu, ls, 1);
            // lanes without a pixel here must not send their warp the other way
            const bool in = mine && (unsigned)(j + c.m) <= (unsigned)(n_eff - 2);
            int k;
            double X, x[3];
            if ((pl_interval(c, lj, ls, ls1, k, X) && px.ok) || !in) {
                const unsigned long long rec = tab[k];
#pragma unroll
                for (int r = 0; r < 3; ++r) x[r] = pl_rise(c, va[r], rec, k, X);
            } else {
#pragma unroll
                for (int r = 0; r < 3; ++r) x[r] = pl_rise_plain(va[r].g, lj, ls, ls1);
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) x[r] = __dmul_rn(__dadd_rn(va[r].s0, x[r]), c.limb);
            q = in ? x[0] : 0.0;
            s = in ? x[1] : 0.0;
            v = in ? x[2] : 0.0;
        }
        double I = a.type == 0 ? ssed : fsed;
        if (a.unit == 0) I = __dmul_rn(a.scale, I);
        else if (a.unit < 0) I = soap_intensity(a.type, pt[a.k], lb_m[a.k], lj, ssed, fsed, solar, t_norm_fac);
        to[0][lane] = s;
        to[1][lane] = __dmul_rn(I, q);
        to[2][lane] = q;
        to[3][lane] = v;
        to[4][lane] = __dmul_rn(v, I);
    };
    if (warp < PS_STRIPS) {
        const bool more = k0 > 0 && mine;
        const long long o = (long long)p * out_stride + j;
        sh.sum[warp][0][lane] = more ? flux[o] : 0.0;
        sh.sum[warp][1][lane] = more ? bconv[o] : 0.0;
        sh.sum[warp][2][lane] = more ? tot[o] : 0.0;
    }
    if (threadIdx.x < PS_STRIPS) sh.next[0][threadIdx.x] = 0;
    if (warp == 0) stage(0);
    // step c: the sums over chunk c - 1, the records of chunk c + 1 (strip 0), the terms of chunk c
    for (int c = 0; c <= n_chunk; ++c) {
        __syncthreads();
        const int b = c & 1;
        if (threadIdx.x < PS_STRIPS) sh.next[b ^ 1][threadIdx.x] = 0;
        const int nt = c < n_chunk ? min(PS_CHUNK, n_cells - c * PS_CHUNK) : 0;
        while (true) {
            int job = 0;
            if (lane == 0) job = atomicAdd(&sh.next[b][strip], 1);
            job = __shfl_sync(0xffffffffu, job, 0);
            if (job >= nt + 2) break;
            if (job == 0) {
                if (c == 0) continue;
                const int np = min(PS_CHUNK, n_cells - (c - 1) * PS_CHUNK);
                double fx = sh.sum[strip][0][lane], bc = sh.sum[strip][1][lane], tt = sh.sum[strip][2][lane];
#pragma unroll 2
                for (int t = 0; t < np; ++t) {
                    const double(*x)[32] = sh.term[b ^ 1][strip][t];
                    fx = __dsub_rn(__dadd_rn(fx, x[0][lane]), x[1][lane]);
                    bc = __dsub_rn(__dadd_rn(bc, x[2][lane]), x[3][lane]);
                    tt = __dsub_rn(__dadd_rn(tt, x[0][lane]), x[4][lane]);
                }
                sh.sum[strip][0][lane] = fx;
                sh.sum[strip][1][lane] = bc;
                sh.sum[strip][2][lane] = tt;
            } else if (job == 1) {
                if (strip == 0 && c + 1 < n_chunk) stage(c + 1);
            } else {
                const int t = job - 2;
                const PlainRec r = sh.rec[b][t];
                terms(r, sh.cell[b][t], sh.tab[b][t], sh.term[b][strip][t]);
            }
        }
    }
    __syncthreads();
    if (warp >= PS_STRIPS || lane == 31 || j >= n) return;
    const long long o = (long long)p * out_stride + j;
    flux[o] = mine ? sh.sum[strip][0][lane] : 0.0;
    bconv[o] = mine ? sh.sum[strip][1][lane] : 0.0;
    tot[o] = mine ? sh.sum[strip][2][lane] : 0.0;
}

// float -> double copy without FP64 instructions
__global__ void k_f32_widen(long long count, const float *__restrict__ a, double *__restrict__ out) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = soap_f32_to_f64(a[i]);
}

namespace soapgb {

// Integration on device buffers (all pointers device).  temp/bi: n_phase x gm.
// out_stride: distance between phases in flux/bconv/tot (>= n).
// Outputs are float for the FP32 form (out_f32 must be set), double otherwise.
int integrate_device(soapgb_ctx *ctx, int form, int n, int n_eff, const double *d_wave, int grid, int n_phase,
                     const double *d_temp, const double *d_bi, const soapgb_maps &dm, const soapgb_cubes &dc,
                     double step, const soapgb_activity *act, void *d_flux, void *d_bconv, void *d_tot, int out_f32,
                     long long out_stride, int *d_cells, int *d_counts, char *fir_scratch,
                     const FirPlanSizes &fp) {
    if ((form == SOAPGB_FAST32) != (out_f32 != 0))
        return set_error(ctx, SOAPGB_ERR_ARG, "integration: FP32 outputs go with the FP32 form only");
    long long gm = (long long)grid * grid;
    if (form == SOAPGB_PLAIN64) {
        int rc = compact_cells(ctx, n_phase, (int)gm, d_bi, -0.5, 1.5, (int)gm, d_cells, d_counts);
        if (rc) return rc;
        PlainGeo *geo = (PlainGeo *)fir_scratch;   // PLAIN64 has no plans: its cells' constants stand there
        const dim3 g((n + PL_TILE - 1) / PL_TILE, n_phase);
        const long long blocks = (long long)g.x * g.y;
        const bool few = blocks <= PS_MAX_PER_SM * ctx->num_sms;
        const auto kern = few ? k_phase_plain64s
                              : blocks >= 6LL * ctx->num_sms ? k_phase_plain64<true> : k_phase_plain64<false>;
        const int threads = few ? 32 * PS_WARPS : PL_THREADS;
        const size_t smem = few ? sizeof(PlainPhaseSmem) : 0;
        if (few) SOAP_CUDA(ctx, soap_allow_smem(k_phase_plain64s, smem));
        for (long long k0 = 0; k0 < gm; k0 += PL_SLAB) {
            const long long end = std::min(gm, k0 + PL_SLAB);
            rc = plain_cells(ctx, k0, end, n_eff, d_wave, dm.delta, step, geo);
            if (rc) return rc;
            SOAP_TRACED(ctx, "integrate_plain64", kern<<<g, threads, smem, ctx->stream>>>(
                n, n_eff, d_wave, dc.q_norm, dc.q_sed, dc.spot_norm, dc.fac_norm, dc.spot_sed, dc.fac_sed, (int)gm,
                d_cells, d_counts, (int)k0, end < gm ? (int)end : INT_MAX, d_temp, d_bi, geo, dm.delta, dm.limb, dm.lb,
                dm.region, gm, act->solar, act->t_star, act->t_diff_fac, (double *)d_flux, (double *)d_bconv,
                (double *)d_tot, out_stride, dc.n_mu, ctx->d_status));
            SOAP_LAUNCHED(ctx);
        }
        return SOAPGB_OK;
    }
    FirPhaseArgs a;
    a.n = n;
    a.n_eff = n_eff;
    a.wave = d_wave;
    a.cubes = &dc;
    a.n_phase = n_phase;
    a.temp = d_temp;
    a.bi = d_bi;
    a.delta = dm.delta;
    a.limb = dm.limb;
    a.lb = dm.lb;
    a.region = dm.region;
    a.gm = gm;
    a.step = step;
    a.act = act;
    a.flux = d_flux;
    a.bconv = d_bconv;
    a.tot = d_tot;
    a.out_f32 = out_f32;
    a.out_stride = out_stride;
    return fir_phase(ctx, form, a, fir_scratch, fp);
}

}  // namespace soapgb

extern "C" int soapgb_phase_integrate(soapgb_ctx *ctx, int form, int n, int n_eff, const double *wave, int grid,
                                      int n_phase, const double *temp, const double *bi, const soapgb_maps *maps,
                                      const soapgb_cubes *cubes, double step, const soapgb_activity *act, int mem,
                                      double *flux, double *bconv, double *tot) {
    if (!ctx || !maps || !cubes || !act) return SOAPGB_ERR_ARG;
    if (n < 2 || n_eff < 2 || n_eff > n || grid < 1 || n_phase < 0 || cubes->n_mu < 1 || !(step > 0) || !wave ||
        !temp || !bi || !flux || !bconv || !tot || !maps->delta || !maps->limb || !maps->lb || !maps->region ||
        !cubes->q_norm || !cubes->q_sed || !cubes->spot_norm || !cubes->fac_norm || !cubes->spot_sed ||
        !cubes->fac_sed)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_phase_integrate: bad arguments");
    if (form != SOAPGB_PLAIN64 && form != SOAPGB_FAST64 && form != SOAPGB_FAST32)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_phase_integrate: unknown form %d", form);
    if (n_phase == 0) return SOAPGB_OK;
    SOAP_DEVICE(ctx);
    long long gm = (long long)grid * grid;
    int n_mu = cubes->n_mu;
    size_t cube_b = sizeof(double) * (size_t)n * n_mu;
    bool host = (mem == SOAPGB_HOST);
    Workspace ws(ctx);
    int s_wave = ws.add(host ? sizeof(double) * n : 0);
    int s_c[6];
    for (int q = 0; q < 4; ++q) s_c[q] = ws.add(host ? cube_b : 0);
    for (int q = 4; q < 6; ++q) s_c[q] = ws.add(host ? sizeof(double) * n : 0);
    int s_temp = ws.add(host ? sizeof(double) * gm * n_phase : 0);
    int s_bi = ws.add(host ? sizeof(double) * gm * n_phase : 0);
    int s_m[4];
    for (int q = 0; q < 3; ++q) s_m[q] = ws.add(host ? sizeof(double) * gm : 0);
    s_m[3] = ws.add(host ? sizeof(int) * gm : 0);
    int s_out[3];
    for (int q = 0; q < 3; ++q) s_out[q] = ws.add(host ? sizeof(double) * (size_t)n * n_phase : 0);
    int s_cells = ws.add(sizeof(int) * gm * n_phase);
    int s_counts = ws.add(sizeof(int) * n_phase);
    int s_f32 = ws.add(form == SOAPGB_FAST32 ? sizeof(float) * 3 * (size_t)n * n_phase : 0);
    FirPlanSizes fp = fir_plan_sizes(form, n, n_mu, gm, true, n_phase);
    int s_fir = ws.add(fp.bytes);
    int rc = ws.commit();
    if (rc) return rc;
#define STAGE(dst, src, bytes, slot)                                                           \
    dst = (decltype(dst))stage_in(ctx, mem, src, bytes, ws.get<void>(slot), &rc);             \
    if (rc) return rc;
    const double *d_wave;
    STAGE(d_wave, wave, sizeof(double) * n, s_wave);
    soapgb_cubes dc;
    dc.n_mu = n_mu;
    STAGE(dc.q_norm, cubes->q_norm, cube_b, s_c[0]);
    STAGE(dc.q_sed, cubes->q_sed, cube_b, s_c[1]);
    STAGE(dc.spot_norm, cubes->spot_norm, cube_b, s_c[2]);
    STAGE(dc.fac_norm, cubes->fac_norm, cube_b, s_c[3]);
    STAGE(dc.spot_sed, cubes->spot_sed, sizeof(double) * n, s_c[4]);
    STAGE(dc.fac_sed, cubes->fac_sed, sizeof(double) * n, s_c[5]);
    const double *d_temp, *d_bi;
    STAGE(d_temp, temp, sizeof(double) * gm * n_phase, s_temp);
    STAGE(d_bi, bi, sizeof(double) * gm * n_phase, s_bi);
    soapgb_maps dm;
    const double *cd;
    STAGE(cd, maps->delta, sizeof(double) * gm, s_m[0]);
    dm.delta = (double *)cd;
    STAGE(cd, maps->limb, sizeof(double) * gm, s_m[1]);
    dm.limb = (double *)cd;
    STAGE(cd, maps->lb, sizeof(double) * gm, s_m[2]);
    dm.lb = (double *)cd;
    const int *ci;
    STAGE(ci, maps->region, sizeof(int) * gm, s_m[3]);
    dm.region = (int *)ci;
    dm.mu = nullptr;
#undef STAGE
    double *d_flux = host ? ws.get<double>(s_out[0]) : flux;
    double *d_bconv = host ? ws.get<double>(s_out[1]) : bconv;
    double *d_tot = host ? ws.get<double>(s_out[2]) : tot;
    if (form == SOAPGB_FAST32) {
        float *f32 = ws.get<float>(s_f32);
        size_t pn = (size_t)n * n_phase;
        rc = integrate_device(ctx, form, n, n_eff, d_wave, grid, n_phase, d_temp, d_bi, dm, dc, step, act, f32,
                              f32 + pn, f32 + 2 * pn, 1, n, ws.get<int>(s_cells), ws.get<int>(s_counts),
                              ws.get<char>(s_fir), fp);
        if (rc) return rc;
        double *outs[3] = {d_flux, d_bconv, d_tot};
        for (int q = 0; q < 3; ++q) {
            SOAP_TRACED(ctx, "widen", k_f32_widen<<<grid_for(ctx, (long long)pn, 256), 256, 0, ctx->stream>>>((long long)pn, f32 + q * pn, outs[q]));
            SOAP_LAUNCHED(ctx);
        }
    } else {
        rc = integrate_device(ctx, form, n, n_eff, d_wave, grid, n_phase, d_temp, d_bi, dm, dc, step, act, d_flux,
                              d_bconv, d_tot, 0, n, ws.get<int>(s_cells), ws.get<int>(s_counts), ws.get<char>(s_fir),
                              fp);
        if (rc) return rc;
    }
    if (host) {
        size_t ob = sizeof(double) * (size_t)n * n_phase;
        SOAP_CUDA(ctx, cudaMemcpyAsync(flux, d_flux, ob, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(bconv, d_bconv, ob, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(tot, d_tot, ob, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return host ? check_status(ctx, "soapgb_phase_integrate") : SOAPGB_OK;
}
