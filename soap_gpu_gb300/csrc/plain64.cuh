// The plain form's cell walk, shared by the quiet-disk sum (disk.cu) and the per-phase
// integration (integrate.cu).
//
// Both sum, for every output pixel j and every cell in map order, the reference's expression
//   (S[i] + (S[i+1] - S[i]) / (l'_{i+1} - l'_i) * (l_j - l'_i)) * limb,   l'_i = l_i - l_i u
// (SOAP_initialize.cu:117-176, SOAP_integration.cu:285-323) with one IEEE rounding per
// operation, i the owner interval of j.  GB300's FP64 pipe issues two lanes per cycle and SM,
// the integer pipes 64, so the walk keeps FP64 for what follows the slope (product, sum, limb
// factor, accumulation) and takes the same bits of the rest from integer arithmetic:
//  - the owner.  In exact arithmetic source i sits at x_i = i + i f + off, so i - j is constant
//    over a tile of pixels unless the shift crosses an integer there.  z(j) = -(j f + off) / (1 + f)
//    at the tile's two ends decides: when both lie in (m + eps, m + 1 - eps), eps above the
//    rounding of the reference's x_i, every pixel of the tile has the owner j + m.  The other
//    cells of the tile (about |v|/c x tile pixels of them) search per pixel, as soap_owner does;
//  - rows and wavelengths.  Successive cells of a map row mostly share mu bin and m, so S[i],
//    S[i+1] - S[i] and l_i stay in registers;
//  - l'_i.  In units of ulp(l), l_i is a 53-bit integer and l_i u a product of two integers with
//    21 fraction bits kept; it is subtracted rounded to an integer unless its fraction is so near
//    to one half that the reference's two roundings could go the other way, or the result lies at
//    the binade's lower end, below which the reference rounds to half an ulp (FP64 then).  l'_{i+1}
//    is the next lane's l'_i (a shuffle), a warp's last one serving only for this;
//  - the division.  On a grid of constant step l'_{i+1} - l'_i is one of a few neighbouring
//    integers in units of ulp: the cell's table holds the 64-bit reciprocals of eight of them for
//    soap_quot_bits;
//  - in the integration, the products with the limb factor and the intensities: pl_mul, from the
//    upper half of the significands' product;
//  - l_j - l'_i.  With X = 2^e + (l_j - l'_i), whose bits are an integer sum, slope x difference is
//    fma(slope, X, -slope 2^e), rounded once.
// A cell and pixel takes 4.4 FP64 instructions in the quiet sum (about 60 when every pixel
// searched its owner, shifted two wavelengths and divided) and 13 in the integration.
// 31,417 cells x 100,000 px: 306 -> 28 ms; 5 phases of 200x200 and 100,000 px, three regions:
// 36 -> 6.1 ms.  One pixel per thread: two took 31 ms, and 8.4 against 7.5 ms.  The quiet sum's one
// product stays on the FP64 pipe: with pl_mul 28.6 ms, two cells at a time 28.0 (219 instructions
// against 147, of which 3.6 against 4.4 on the FP64 pipe: issue and the chain then bound it); and the
// integration's three rises as integer products too took 6.5 ms against 6.1.
// What the integers do not cover (another binade, an uneven grid, differences outside the table,
// non-finite or extreme values) takes the reference's operations.  Every path gives the same bits.
#pragma once

#include <climits>

#include "internal.cuh"

constexpr int PL_THREADS = 64;                // two warps, each 31 pixels
constexpr int PL_TILE = PL_THREADS / 32 * 31;
constexpr int PL_CHUNK = PL_THREADS;          // cells staged at a time, one per thread
constexpr int PL_TAB = 8;                     // table entries per cell
constexpr int PL_FRAC = 21;                   // fraction bits of l u
// Cells whose constants are held at a time (0.94 GB).  A larger map is taken in slabs of as many
// cells, each adding to what the ones before left: the sums' order stays, and the workspace does not
// grow with the map's area (90 GB for 20,000 x 20,000 cells).
constexpr long long PL_SLAB = 1LL << 22;

// the table of one binade of l'
struct PlainTab {
    long long base;   // l'_{i+1} - l'_i of entry 0, in ulp
    int ex;           // biased exponent of l', -1: no table
    int qe;           // the slope's biased exponent is the difference's + qe (+ 0 or 1)
    unsigned long long rec[PL_TAB];
};

// a cell's constants, computed once per call and slab; tables for the first and the last wavelength's binade
struct PlainGeo {
    double sq, fbeta, off;   // CellShift
    double u;                // 1 - sq
    double iF, eps;          // 1 / (1 + f), error of x_i
    unsigned long long w;    // |u| 2^(53 + PL_FRAC)
    long long zone;          // error of l u, in its last fraction bit
    PlainTab tab[2];
};

enum : int {
    PL_CONST = 1,   // one owner offset m for the tile
    PL_STILL = 2,   // v == 0: the pixel itself
};

// the cells [k0, k1) of a list in map order as [from, to) of it; k0 = 0 and k1 = INT_MAX: no bound
__device__ __forceinline__ int pl_first(const int *__restrict__ cells, int n, int k) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);
        if (cells[mid] < k) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ void pl_slab(const int *__restrict__ cells, int n, int k0, int k1, int &from, int &to) {
    from = k0 > 0 ? pl_first(cells, n, k0) : 0;
    to = k1 != INT_MAX ? pl_first(cells, n, k1) : n;
}

// a factor of many products
struct PlainFactor {
    unsigned long long sig;   // significand, leading bit at bit 63
    int hi;                   // sign and exponent; 0: not normal or not of moderate size
};

// what a tile needs of a cell
struct PlainRec {
    double u, limb;
    unsigned long long w;
    long long base;
    int m, row;
    int flags, ex;          // ex: biased exponent the integers stand for, -1: none
    int qe, zone;
};

__device__ __forceinline__ int pl_exp(double v) { return (int)((unsigned)__double2hiint(v) >> 20); }

constexpr int PL_SPAN = 200;   // exponents of a product's factors: products of three stay normal

__device__ __forceinline__ PlainFactor pl_factor(double v) {
    PlainFactor f;
    f.sig = soap_sig(v);
    f.hi = soap_moderate(v, PL_SPAN) ? __double2hiint(v) & 0xfff00000 : 0;
    return f;
}

// The bits of a x b (a normal): the upper half of the significands' product holds 53 bits and at
// least ten to round by.  unsure: those are one half as far as they show, so the reference's
// operation decides (one product in 2048).
__device__ __forceinline__ double pl_mul(double a, const PlainFactor &b, bool &unsure) {
    const int ah = __double2hiint(a);
    unsigned long long h = __umul64hi(soap_sig(a), b.sig);
    const int top = (int)(h >> 63);
    if (!top) h += h;
    const unsigned low = (unsigned)h & 0x7ffu;
    unsure = unsure || low == 0x400u;
    const unsigned long long m = (h >> 11) + (low >> 10);
    // exponent - 1: the significand's leading bit adds the one
    const unsigned e = (unsigned)(ah & 0x7ff00000) + (unsigned)(b.hi & 0x7ff00000) - (1024u << 20) + ((unsigned)top << 20);
    return __longlong_as_double(
        (long long)(m + ((unsigned long long)(e | ((unsigned)(ah ^ b.hi) & 0x80000000u)) << 32)));
}

// A call, so that the products of the lanes that need one stay off the others' path.
static __device__ __noinline__ double pl_mul_plain(double a, double b) { return __dmul_rn(a, b); }

// The table of the binade of l (1 - u) around spacings d sq
__device__ __forceinline__ void pl_table(double l, double d, double sq, double u, PlainTab &t) {
    t.ex = -1;
    t.base = 0;
    t.qe = 0;
    const double lp = l - l * u;
    const int ex = pl_exp(lp);
    if (!(lp > 0.0) || ex < 1023 - 200 || ex > 1023 + 200 || !(fabs(u) < 0x1p-10)) return;
    const double cn = d * sq * __hiloint2double((2046 + 52 - ex) << 20, 0);   // in ulp(l')
    if (!(cn > 16.0 && cn < 0x1p51)) return;
    const long long n0 = __double2ll_rn(cn) - PL_TAB / 2;
    const int lz = __clzll(n0);
    if (__clzll(n0 + PL_TAB - 1) != lz) return;
    const double scale = __hiloint2double((1023 + lz - 63) << 20, 0);   // n scale in [1, 2)
    const double nm = __ll2double_rn(n0 + PL_TAB / 2) * scale, rm = 1.0 / nm;
#pragma unroll
    for (int k = 0; k < PL_TAB; ++k) {
        const double nd = nm + (double)(k - PL_TAB / 2) * scale;
        // a Newton step from the middle one's reciprocal leaves (4 / n0)^2
        const double r = n0 >= (1LL << 27) ? fma(rm, fma(-nd, rm, 1.0), rm) : 1.0 / nd;
        t.rec[k] = soap_recip64((unsigned long long)(n0 + k) << lz, r);
    }
    t.base = n0;
    t.ex = ex;
    t.qe = 1023 - ex + lz - 11;
}

// The record of one cell for the tile [j0, j0 + cnt); lmid: a wavelength of the tile
__device__ __forceinline__ void pl_stage(const PlainGeo *__restrict__ geo, double delta, double limb, int row, int j0,
                                         int cnt, double lmid, PlainRec &rec, unsigned long long *tab) {
    const double u = geo->u, f = geo->fbeta, off = geo->off;
    rec.u = u;
    rec.limb = limb;
    rec.w = geo->w;
    rec.zone = (int)geo->zone;
    rec.row = row;
    rec.m = 0;
    rec.flags = 0;
    if (delta == 0.0) rec.flags = PL_STILL;
    const double z0 = -fma((double)j0, f, off) * geo->iF;
    const double z1 = -fma((double)(j0 + cnt - 1), f, off) * geo->iF;
    const double m = floor(z0), hi = m + 1.0 - geo->eps, lo = m + geo->eps;
    if (delta != 0.0 && fabs(z0) < 1e9 && z0 > lo && z0 < hi && z1 > lo && z1 < hi) {
        rec.m = (int)m;
        rec.flags = PL_CONST;
    }
    const int ex = pl_exp(lmid - lmid * u);
    const PlainTab &t = geo->tab[geo->tab[0].ex == ex ? 0 : 1];
    rec.ex = t.ex == ex ? ex : -1;
    rec.base = t.base;
    rec.qe = t.qe;
#pragma unroll
    for (int k = 0; k < PL_TAB; ++k) tab[k] = t.rec[k];
}

// a pixel's source interval and one row's values there
struct PlainPix {
    double li;                 // l_i
    unsigned long long lm;     // its significand
    bool ok;                   // the row differences are zero or normal and of moderate size
};
struct PlainVal {
    double s0, g;              // S[i], S[i+1] - S[i]
    unsigned long long gm;     // the difference's significand
};

// +0 or -0, without the FP64 pipe's compare
__device__ __forceinline__ bool pl_zero(double g) {
    return (((unsigned)__double2hiint(g) << 1) | (unsigned)__double2loint(g)) == 0u;
}

__device__ __forceinline__ bool pl_load(PlainVal &v, const double *__restrict__ row, int i, int i1) {
    v.s0 = row[i];
    v.g = __dsub_rn(row[i1], v.s0);
    v.gm = soap_sig(v.g);
    return pl_zero(v.g) || soap_moderate(v.g, 700);
}

// A call: inlined, the two FP64 instructions would be issued for every cell under a predicate,
// and take their time on the pipe with no lane active.
static __device__ __noinline__ double pl_shifted_plain(double li, double u) { return __dsub_rn(li, __dmul_rn(li, u)); }

// l'_i
__device__ __forceinline__ double pl_shifted(const PlainRec &c, const PlainPix &x) {
    const unsigned long long v = __umul64hi(x.lm, c.w);   // l u in units of ulp 2^-PL_FRAC
    const unsigned fr = ((unsigned)v + (1u << (PL_FRAC - 1)) + (unsigned)c.zone) & ((1u << PL_FRAC) - 1u);
    const long long r = (long long)((v + (1ULL << (PL_FRAC - 1))) >> PL_FRAC);
    const long long b = __double_as_longlong(x.li);
    double ls = __longlong_as_double(__double2hiint(c.u) < 0 ? b + r : b - r);
    // inside the binade: at and just above its power of two (2^32 ulp) the reference's difference may
    // lie below, where it rounds to half an ulp
    const bool inside = (unsigned)__double2hiint(ls) - ((unsigned)c.ex << 20) - 1u < 0xfffffu;
    const bool whole = fr > 2u * (unsigned)c.zone && pl_exp(x.li) == c.ex && inside;
    if (!whole) ls = pl_shifted_plain(x.li, c.u);
    return ls;
}

// the interval's table index and X = 2^e + (l_j - l'_i), false where the integers do not apply
__device__ __forceinline__ bool pl_interval(const PlainRec &c, double lj, double ls0, double ls1, int &k, double &X) {
    const long long b0 = __double_as_longlong(ls0);
    const unsigned long long d = (unsigned long long)(__double_as_longlong(ls1) - b0 - c.base);
    const long long dl = __double_as_longlong(lj) - b0;
    const bool hit = d < (unsigned long long)PL_TAB && pl_exp(ls0) == c.ex && pl_exp(ls1) == c.ex &&
                     pl_exp(lj) == c.ex && dl >= 0;
    k = hit ? (int)d : 0;
    X = __longlong_as_double(dl + ((long long)c.ex << 52));
    return hit;
}

// slope x (l_j - l'_i) in integers: rec = floor(2^127 / n) of the interval n
__device__ __forceinline__ double pl_rise(const PlainRec &c, const PlainVal &v, unsigned long long rec, int k,
                                          double X) {
    const unsigned long long bits =
        soap_quot_bits(v.g, v.gm, rec, (unsigned long long)(c.base + k), c.qe - 1012 + c.ex, c.qe);
    const double slope = __longlong_as_double((long long)bits);
    const double scaled = __longlong_as_double((long long)((bits + ((unsigned long long)(long long)(c.ex - 1023) << 52)) ^
                                                           0x8000000000000000ULL));   // -slope 2^e
    const double t = __fma_rn(slope, X, scaled);
    return pl_zero(v.g) ? v.g : t;   // flat continuum
}

// ... by the reference's operations (a call, as pl_shifted_plain)
static __device__ __noinline__ double pl_rise_plain(double g, double lj, double ls0, double ls1) {
    return __dmul_rn(__ddiv_rn(g, __dsub_rn(ls1, ls0)), __dsub_rn(lj, ls0));
}

namespace soapgb {
// the constants of the map's cells [k0, k1), geo[k1 - k0]
int plain_cells(soapgb_ctx *ctx, long long k0, long long k1, int n_eff, const double *d_wave, const double *d_delta,
                double step, PlainGeo *geo);
}  // namespace soapgb
