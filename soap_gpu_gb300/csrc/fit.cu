// a17-a18: Gaussian fit of the CCF and its bisector, batched.
//
// Reference: BIS_FIT2.cpp:31-81 (model and analytic Jacobian), :97-192 (GSL
// multifit_nlinear trust region with default parameters: Levenberg-Marquardt,
// More scaling, xtol = gtol = 1e-8, ftol = 0, max_iter = 10000) and :214-317
// (bisector on 91 depths, span).  The reference spawns one BIS_FIT2 process per
// spectrum and exchanges text files with it.  Here one block of two warps fits one
// spectrum: the threads evaluate residuals and Jacobian rows, shuffles and shared
// memory reduce J^T J and J^T f, and every thread solves the 4x4 damped normal
// equations redundantly (no divergence).
// What bounds it is the FP64 pipe's latency and rate (half a lane per cycle in each
// of an SM's four partitions): a few hundred spectra put about one warp on each
// partition, so an iteration costs its FP64 instructions in a row.  Hence two warps
// per spectrum, reciprocals instead of divisions inside an iteration, sixteen sums
// reduced together (16 additions per warp instead of 5 each), and index searches by
// integer images instead of serial loops of FP64 compares: 303 CCFs of 161 velocities
// 478 -> 150 us.  Damping follows Nielsen's rule as in GSL
// (mu *= max(1/3, 1-(2 rho-1)^3) on acceptance, mu *= nu, nu *= 2 on rejection).
// All iteration loops are bounded.
#include <cmath>

#include "internal.cuh"

using namespace soapgb;

constexpr int FIT_THREADS = 64;    // the fit's threads per spectrum
constexpr int ADJ_THREADS = 128;   // its adjoint's
#define FIT_DEPTHS 91
constexpr size_t FIT_SMEM_MAX = 48 * 1024;   // bisector arrays kept in shared memory up to here

// Sums of v[0 .. 15] over the block in a fixed order, the same bits in every thread's tot[]: a
// warp's lanes halve the values they hold as they halve the lanes that hold them.
struct BlockSums {
    double part[ADJ_THREADS / 32][16], tot[16];
};
__device__ __forceinline__ void block_sum16(double (&v)[16], BlockSums &s) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16, h = 8; o > 1; o >>= 1, h >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < h; ++q) {
            const double give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    __syncthreads();
    if (!(lane & 1)) s.part[w][lane >> 1] = v[0];
    __syncthreads();
    if (threadIdx.x < 16) {
        double t = s.part[0][threadIdx.x];
        for (int k = 1; k < nw; ++k) t += s.part[k][threadIdx.x];
        s.tot[threadIdx.x] = t;
    }
    __syncthreads();
}

// index of the block's largest key, the first at ties (every thread; s: two words)
__device__ __forceinline__ int block_argmax(unsigned long long key, int i, unsigned long long *s_key, int *s_idx) {
    __syncthreads();
    if (threadIdx.x == 0) {
        *s_key = 0ULL;
        *s_idx = 0x7fffffff;
    }
    __syncthreads();
    if (key) atomicMax(s_key, key);
    __syncthreads();
    if (key && key == *s_key) atomicMin(s_idx, i);
    __syncthreads();
    return *s_idx;
}

__device__ __forceinline__ double gauss_sigma(double fwhm) { return fwhm / 2 / sqrt(2 * log(2.0)); }

// solve (A) x = b (4x4 SPD) by Cholesky, the diagonal as reciprocals; false if not positive definite
__device__ __forceinline__ bool chol4(const double *A, const double *b, double *x) {
    double L[16], r[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j <= i; j++) {
            double s = A[i * 4 + j];
#pragma unroll
            for (int k = 0; k < j; k++) s -= L[i * 4 + k] * L[j * 4 + k];
            if (i == j) {
                if (!(s > 0)) return false;
                r[i] = rsqrt(s);
            } else {
                L[i * 4 + j] = s * r[j];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        double s = b[i];
#pragma unroll
        for (int k = 0; k < i; k++) s -= L[i * 4 + k] * y[k];
        y[i] = s * r[i];
    }
#pragma unroll
    for (int i = 3; i >= 0; i--) {
        double s = y[i];
#pragma unroll
        for (int k = i + 1; k < 4; k++) s -= L[k * 4 + i] * x[k];
        x[i] = s * r[i];
    }
    return true;
}

__global__ void __launch_bounds__(FIT_THREADS) k_gauss_bis(int n_spec, int n, const double *__restrict__ xin,
                                                           const double *__restrict__ yall,
                                                           const double *__restrict__ errall,
                                                           double *__restrict__ model, double *__restrict__ par,
                                                           double *__restrict__ depth_out,
                                                           double *__restrict__ bis_out, int *__restrict__ iters,
                                                           double *__restrict__ scratch) {
    extern __shared__ __align__(16) double sm_fit[];
    __shared__ BlockSums sums;
    __shared__ unsigned long long s_key;
    __shared__ int s_idx;
    __shared__ double s_bis[FIT_DEPTHS];
    const int s = blockIdx.x, t = threadIdx.x;
    const double *y = yall + (long long)s * n;
    const double *err = errall ? errall + (long long)s * n : nullptr;
    const double x00 = xin[0];
    auto x = [&](int i) { return xin[i] - x00; };   // rebased velocities
    const double s2l = 2 * sqrt(2 * log(2.0));
    // initial guess, BIS_FIT2.cpp:155-160: the first largest |y - c|
    double c = (y[0] + y[n - 1]) / 2;
    double fwhm = (x(n - 1) - x(0)) / 5.;
    double k = 0., x0 = x(n / 2);
    {
        unsigned long long key = 0ULL;
        int at = 0;
        for (int i = t; i < n; i += FIT_THREADS) {
            const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(y[i] - c));
            if (v > key && v <= 0x7ff0000000000000ULL) {   // (a NaN is not larger than anything)
                key = v;
                at = i;
            }
        }
        const int best = block_argmax(key, at, &s_key, &s_idx);
        if (best < n) {
            k = y[best] - c;
            x0 = x(best);
        }
    }
    double p[4] = {c, k, x0, fwhm};
    double D[4] = {0, 0, 0, 0};
    double mu = 0.0, nu = 2.0;
    double dx[4] = {0, 0, 0, 0};
    int status = -1;
    const double xtol = 1e-8, gtol = 1e-8;
    for (int iter = 0; iter <= 10000; ++iter) {
        // J^T J, J^T f, phi at p
        const double is = s2l / p[3], is2 = is * is, h = 0.5 * is2;   // 1 / sigma, 1 / sigma^2
        const double f2 = p[1] * is2, f3 = f2 * is / s2l;             // of J[2], J[3]
        double v[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = 0.0;
        for (int i = t; i < n; i += FIT_THREADS) {
            const double inv = err ? 1.0 / err[i] : 1.0;
            const double d = x(i) - p[2];
            const double e = exp(-d * d * h);
            const double f = (p[0] + p[1] * e - y[i]) * inv;
            const double ed = e * inv * d;
            const double J[4] = {inv, e * inv, f2 * ed, f3 * ed * d};
            int q = 0;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                v[10 + a] += J[a] * f;
#pragma unroll
                for (int b = a; b < 4; ++b) v[q++] += J[a] * J[b];
            }
            v[14] += f * f;
        }
        block_sum16(v, sums);
        double A[16], g[4];
        {
            int q = 0;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                g[a] = sums.tot[10 + a];
#pragma unroll
                for (int b = a; b < 4; ++b) { A[a * 4 + b] = A[b * 4 + a] = sums.tot[q]; ++q; }
            }
        }
        const double phi = sums.tot[14];
        if (iter == 0) {
            double mx = 0.0;
            for (int a = 0; a < 4; ++a) {
                D[a] = sqrt(A[a * 5]);
                if (D[a] == 0.0) D[a] = 1.0;
                const double r = sqrt(A[a * 5]) / D[a];
                mx = fmax(mx, r * r);
            }
            mu = 1e-3 * mx;
        } else {
            for (int a = 0; a < 4; ++a) D[a] = fmax(D[a], sqrt(A[a * 5]));
            // convergence tests after an accepted step (GSL multifit_nlinear_test)
            bool xok = true;
            for (int a = 0; a < 4; ++a)
                if (fabs(dx[a]) > xtol * (fabs(p[a]) + xtol)) xok = false;
            double gn = 0.0;
            for (int a = 0; a < 4; ++a) gn = fmax(gn, fabs(g[a] * fmax(fabs(p[a]), 1.0)));
            if (xok || gn <= gtol * fmax(0.5 * phi, 1.0)) { status = iter; break; }
            if (iter == 10000) break;
        }
        // inner loop: find an acceptable step (at most 16 consecutive rejections)
        bool accepted = false;
        int bad = 0;
        while (!accepted && bad <= 15) {
            double M[16], rhs[4];
            for (int q = 0; q < 16; ++q) M[q] = A[q];
            for (int a = 0; a < 4; ++a) { M[a * 5] += mu * D[a] * D[a]; rhs[a] = -g[a]; }
            if (!chol4(M, rhs, dx)) { mu *= nu; nu *= 2; ++bad; continue; }
            double pt[4];
            for (int a = 0; a < 4; ++a) pt[a] = p[a] + dx[a];
            // residual sum of squares at pt
            const double ht = 0.5 * (s2l / pt[3]) * (s2l / pt[3]);
            double acc = 0.0;
            for (int i = t; i < n; i += FIT_THREADS) {
                const double d = x(i) - pt[2];
                double f = pt[0] + pt[1] * exp(-d * d * ht) - y[i];
                if (err) f /= err[i];
                acc += f * f;
            }
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            __syncthreads();
            if ((t & 31) == 0) sums.part[t >> 5][0] = acc;
            __syncthreads();
            const double phit = sums.part[0][0] + sums.part[1][0];
            double jdx = 0.0;   // ||J dx||^2 = dx^T (J^T J) dx
            for (int a = 0; a < 4; ++a)
                for (int b = 0; b < 4; ++b) jdx += dx[a] * A[a * 4 + b] * dx[b];
            double mud = 0.0;
            for (int a = 0; a < 4; ++a) mud += mu * D[a] * D[a] * dx[a] * dx[a];
            double pred = jdx + 2 * mud;
            double rho = (pred > 0 && phit < phi) ? (phi - phit) / pred : -1.0;
            if (rho > 0) {
                accepted = true;
                double r = 2 * rho - 1;
                double fac = 1 - r * r * r;
                mu *= fmax(fac, 1.0 / 3.0);
                nu = 2;
                for (int a = 0; a < 4; ++a) p[a] = pt[a];
            } else {
                mu *= nu;
                nu *= 2;
                ++bad;
            }
        }
        if (!accepted) {
            // no acceptable step: converged if the last (rejected) step already
            // meets the tolerances, as GSL's driver tests it after ENOPROG
            bool xok = true;
            for (int a = 0; a < 4; ++a)
                if (fabs(dx[a]) > xtol * (fabs(p[a]) + xtol)) xok = false;
            double gn = 0.0;
            for (int a = 0; a < 4; ++a) gn = fmax(gn, fabs(g[a] * fmax(fabs(p[a]), 1.0)));
            status = (xok || gn <= gtol * fmax(0.5 * phi, 1.0)) ? iter + 1 : -1;
            break;
        }
    }
    c = p[0]; k = p[1]; x0 = p[2]; fwhm = p[3];
    {
        const double is = s2l / fwhm, h = 0.5 * is * is;
        for (int i = t; i < n; i += FIT_THREADS) {
            const double d = x(i) - x0;
            model[(long long)s * n + i] = c + k * exp(-d * d * h);
        }
    }
    // bisector, BIS_FIT2.cpp:214-268
    double *norm = scratch ? scratch + (long long)s * 4 * n : sm_fit;
    double *p0 = norm + n, *p1 = norm + 2 * n, *p2 = norm + 3 * n;
    const double sig_b = fwhm / 2. / pow(2. * log(2.), .5), ss = sig_b * sig_b, iss = 1.0 / ss;
    const double v0 = x0 + x00;
    unsigned long long key = 0ULL;
    int at = 0;
    const double nk = -c / k;
    for (int i = t; i < n; i += FIT_THREADS) {
        const double v = nk * (1. - y[i] / c);
        norm[i] = v;
        const unsigned long long w = v == v ? soap_ord64(v + 0.0) : 0ULL;
        if (w > key) {
            key = w;
            at = i;
        }
    }
    if (t == 0) { p0[n - 1] = 0.0; p1[n - 1] = 0.0; p2[n - 1] = 0.0; }   // never set by the loop below
    int ind_max = block_argmax(key, at, &s_key, &s_idx);   // (its barriers publish norm)
    if (ind_max >= n || norm[0] != norm[0]) ind_max = 0;   // nothing is larger than a NaN
    for (int i = t; i < n - 1; i += FIT_THREADS) {
        const double vr = (xin[i] + xin[i + 1]) / 2.;
        const double dd = vr - v0, u = dd * dd * iss;
        const double e = exp(-0.5 * u);
        const double dC = -dd * iss * e;
        const double d2C = (u - 1) * iss * e;
        const double q2 = -d2C / (dC * dC * dC) / 2.;
        const double a0 = norm[i], a1 = norm[i + 1];
        const double q1 = (xin[i + 1] - xin[i] - q2 * (a1 * a1 - a0 * a0)) / (a1 - a0);
        p2[i] = q2;
        p1[i] = q1;
        p0[i] = xin[i] - q1 * a0 - q2 * (a0 * a0);
    }
    __syncthreads();
    double *bo = bis_out + (long long)s * FIT_DEPTHS;
    for (int q = t; q < FIT_DEPTHS; q += FIT_THREADS) {
        const double dep = (double)(q + 5) / 100;
        int i_b = ind_max, i_r = ind_max;
        while ((norm[i_b] > dep) && (i_b > 1)) i_b--;
        while ((norm[i_r + 1] > dep) && (i_r < (n - 2))) i_r++;
        double b = (p0[i_b] + p0[i_r]) + (p1[i_b] + p1[i_r]) * dep + (p2[i_b] + p2[i_r]) * (dep * dep);
        b /= 2.;
        bo[q] = b;
        s_bis[q] = b;
        depth_out[(long long)s * FIT_DEPTHS + q] = 1.0 - fabs(k) * dep;
    }
    __syncthreads();
    if (t == 0) {
        // span in the reference's summation order, BIS_FIT2.cpp:256-268: depths 0.1 to 0.4 and
        // 0.6 to 0.9, the hundredths 10 .. 40 and 60 .. 90
        double top = 0.0, bottom = 0.0;
        for (int q = 10; q <= 40; ++q) top += s_bis[q - 5];
        for (int q = 60; q <= 90; ++q) bottom += s_bis[q - 5];
        double *pp = par + (long long)s * 5;
        pp[0] = c;
        pp[1] = fabs(k);
        pp[2] = top / 31 - bottom / 31;
        pp[3] = v0;
        pp[4] = fwhm;
        if (iters) iters[s] = status;
    }
}

extern "C" int soapgb_gauss_bis(soapgb_ctx *ctx, int n_spec, int n, const double *x, const double *y,
                                const double *err, int mem, double *model, double *par, double *depth, double *bis,
                                int *iters) {
    if (!ctx) return SOAPGB_ERR_ARG;
    if (n_spec < 0 || n < 8 || !x || !y || !model || !par || !depth || !bis)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_gauss_bis: bad arguments");
    if (n_spec == 0) return SOAPGB_OK;
    SOAP_DEVICE(ctx);
    bool host = (mem == SOAPGB_HOST);
    Workspace ws(ctx);
    int s_x = ws.add(host ? sizeof(double) * n : 0);
    int s_y = ws.add(host ? sizeof(double) * (size_t)n * n_spec : 0);
    int s_e = ws.add(host && err ? sizeof(double) * (size_t)n * n_spec : 0);
    int s_model = ws.add(host ? sizeof(double) * (size_t)n * n_spec : 0);
    int s_par = ws.add(host ? sizeof(double) * 5 * n_spec : 0);
    int s_dep = ws.add(host ? sizeof(double) * FIT_DEPTHS * n_spec : 0);
    int s_bis = ws.add(host ? sizeof(double) * FIT_DEPTHS * n_spec : 0);
    int s_it = ws.add(host && iters ? sizeof(int) * n_spec : 0);
    // the bisector's arrays: shared memory, or scratch for long CCFs
    const size_t bis_b = sizeof(double) * 4 * (size_t)n;
    const bool in_smem = bis_b <= FIT_SMEM_MAX - 4096;
    int s_scr = ws.add(in_smem ? 0 : bis_b * n_spec);
    int rc = ws.commit();
    if (rc) return rc;
    const double *d_x = (const double *)stage_in(ctx, mem, x, sizeof(double) * n, ws.get<void>(s_x), &rc);
    if (rc) return rc;
    const double *d_y = (const double *)stage_in(ctx, mem, y, sizeof(double) * (size_t)n * n_spec, ws.get<void>(s_y), &rc);
    if (rc) return rc;
    const double *d_e = (const double *)stage_in(ctx, mem, err, err ? sizeof(double) * (size_t)n * n_spec : 0, ws.get<void>(s_e), &rc);
    if (rc) return rc;
    double *d_model = host ? ws.get<double>(s_model) : model;
    double *d_par = host ? ws.get<double>(s_par) : par;
    double *d_dep = host ? ws.get<double>(s_dep) : depth;
    double *d_bis = host ? ws.get<double>(s_bis) : bis;
    int *d_it = iters ? (host ? ws.get<int>(s_it) : iters) : nullptr;
    SOAP_TRACED(ctx, "gauss_bis", k_gauss_bis<<<n_spec, FIT_THREADS, in_smem ? bis_b : 0, ctx->stream>>>(
        n_spec, n, d_x, d_y, d_e, d_model, d_par, d_dep, d_bis, d_it, in_smem ? nullptr : ws.get<double>(s_scr)));
    SOAP_LAUNCHED(ctx);
    if (host) {
        SOAP_CUDA(ctx, cudaMemcpyAsync(model, d_model, sizeof(double) * (size_t)n * n_spec, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(par, d_par, sizeof(double) * 5 * n_spec, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(depth, d_dep, sizeof(double) * FIT_DEPTHS * n_spec, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaMemcpyAsync(bis, d_bis, sizeof(double) * FIT_DEPTHS * n_spec, cudaMemcpyDeviceToHost, ctx->stream));
        if (iters) SOAP_CUDA(ctx, cudaMemcpyAsync(iters, d_it, sizeof(int) * n_spec, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    }
    return host ? check_status(ctx, "soapgb_gauss_bis") : SOAPGB_OK;
}

// ---------------------------------------------------------------------------
// Adjoint of the Gaussian fit (the differentiable form; the reference has no
// gradient path).  At the fitted optimum theta = (c, k, x0, fwhm) of
// Phi = sum_i f_i^2, f_i = (G(x_i; theta) - y_i) / err_i, the stationarity condition
// sum_i f_i df_i/dtheta = 0 gives, by the implicit function theorem,
//   H dtheta/dy_j = grad G_j / err_j^2,   H = sum_i (J_i J_i^T + f_i Hess f_i)
// so dL/dy_j = (grad G_j . z) / err_j^2 with H z = dL/dtheta.  The second derivatives
// of G = c + k e, e = exp(-d^2 / 2 s^2), d = x - x0, s = a fwhm, a = 1 / (2 sqrt(2 ln 2)):
//   G_k,x0 = e d / s^2          G_k,fwhm = a e d^2 / s^3
//   G_x0,x0 = k e (d^2 / s^4 - 1 / s^2)
//   G_x0,fwhm = a k e d (d^2 / s^5 - 2 / s^3)
//   G_fwhm,fwhm = a^2 k e d^2 (d^2 / s^6 - 3 / s^4)   (all c terms vanish).
// The fitted outputs give c, |k|, v0 = x0 + x[0] and fwhm; the sign of k is that of
// the model's largest excursion from c.  One block per spectrum, fixed reduction order.
// ---------------------------------------------------------------------------
// 4x4 solve by Gaussian elimination with partial pivoting; false when singular
__device__ bool solve4(double *A, double *b, double *z) {
    for (int c = 0; c < 4; ++c) {
        int piv = c;
        for (int r = c + 1; r < 4; ++r)
            if (fabs(A[r * 4 + c]) > fabs(A[piv * 4 + c])) piv = r;
        if (!(fabs(A[piv * 4 + c]) > 0.0)) return false;
        if (piv != c) {
            for (int q = 0; q < 4; ++q) { double t = A[c * 4 + q]; A[c * 4 + q] = A[piv * 4 + q]; A[piv * 4 + q] = t; }
            double t = b[c]; b[c] = b[piv]; b[piv] = t;
        }
        for (int r = c + 1; r < 4; ++r) {
            double f = A[r * 4 + c] / A[c * 4 + c];
            for (int q = c; q < 4; ++q) A[r * 4 + q] -= f * A[c * 4 + q];
            b[r] -= f * b[c];
        }
    }
    for (int r = 3; r >= 0; --r) {
        double t = b[r];
        for (int q = r + 1; q < 4; ++q) t -= A[r * 4 + q] * z[q];
        z[r] = t / A[r * 4 + r];
    }
    return true;
}

__global__ void __launch_bounds__(ADJ_THREADS) k_gauss_fit_adj(int n_spec, int n, const double *__restrict__ x,
                                                               const double *__restrict__ yall,
                                                               const double *__restrict__ errall,
                                                               const double *__restrict__ model,
                                                               const double *__restrict__ par,
                                                               const double *__restrict__ gpar,
                                                               double *__restrict__ grad_y,
                                                               double *__restrict__ scratch, int *status) {
    extern __shared__ __align__(16) double sm_fit[];
    __shared__ BlockSums sums;
    __shared__ unsigned long long s_key;
    __shared__ int s_idx;
    const int s = blockIdx.x, tid = threadIdx.x;
    const double *y = yall + (long long)s * n;
    const double *err = errall ? errall + (long long)s * n : nullptr;
    const double *mo = model + (long long)s * n;
    const double *pp = par + (long long)s * 5;
    const double *gp = gpar + (long long)s * 5;
    double *gy = grad_y + (long long)s * n;
    double *norm = scratch ? scratch + (long long)s * n : sm_fit;
    const double c = pp[0], v0 = pp[3], fwhm = pp[4];
    // sign of k: the model's largest excursion from c (first index at ties)
    unsigned long long key = 0ULL;
    int at = 0;
    for (int i = tid; i < n; i += ADJ_THREADS) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(fabs(mo[i] - c));
        if (v + 1 > key && v <= 0x7ff0000000000000ULL) {
            key = v + 1;
            at = i;
        }
    }
    const int top = block_argmax(key, at, &s_key, &s_idx);
    const double sgn = (top >= n || mo[top] - c >= 0.0) ? 1.0 : -1.0;
    const double k = sgn * pp[1];
    const double a = gauss_sigma(1.0);
    const double is = 1.0 / gauss_sigma(fwhm), is2 = is * is, is3 = is2 * is, is4 = is2 * is2;
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = 0.0;
    for (int i = tid; i < n; i += ADJ_THREADS) {
        const double inv = err ? 1.0 / err[i] : 1.0;
        const double d = x[i] - v0, d2 = d * d, u = d2 * is2;
        const double e = exp(-0.5 * u);
        const double f = (c + k * e - y[i]) * inv;
        const double G[4] = {1.0, e, k * e * d * is2, k * e * d2 * a * is3};
        double S[10];   // second derivatives, upper triangle row-major
        S[0] = 0.0; S[1] = 0.0; S[2] = 0.0; S[3] = 0.0;
        S[4] = 0.0;
        S[5] = e * d * is2;
        S[6] = a * e * d2 * is3;
        S[7] = k * e * is2 * (u - 1.0);
        S[8] = a * k * e * d * is3 * (u - 2.0);
        S[9] = a * a * k * e * d2 * is4 * (u - 3.0);
        int t = 0;
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = p; q < 4; ++q, ++t) v[t] += inv * inv * G[p] * G[q] + f * inv * S[t];
    }
    block_sum16(v, sums);
    double H[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) H[q] = sums.tot[q];
    double A[16], b[4] = {gp[0], gp[1] * sgn, gp[3], gp[4]}, z[4] = {0, 0, 0, 0};
    // --- the bisector span (BIS_FIT2.cpp:214-268).  Per depth the forward picks the
    // intervals i_b, i_r where the normalised CCF a_i = (y_i - c) / k crosses it (held fixed
    // here: a discrete choice) and evaluates on each the quadratic inverse
    //   P_i(d) = x_i + dx_i (d - a_i) / (a_{i+1} - a_i) + q2_i (d - a_i)(d - a_{i+1}),
    // the closed form of its p0 + p1 d + p2 d^2, with q2_i = -C''/(2 C'^3) of the fitted
    // Gaussian at the interval's middle.  The span is the mean of the bisector over depths
    // 0.1-0.4 minus its mean over 0.6-0.9; its gradient reaches y directly (a_i) and through
    // the fit's parameters (c, k in a_i; v0, sigma in q2_i), the latter added to b.
    __shared__ int sp_ib[FIT_DEPTHS], sp_ir[FIT_DEPTHS];
    __shared__ double sp_d[FIT_DEPTHS][4];
    const double gs = gp[2];
    if (gs != 0.0) {   // uniform for the block
        const double nk = -c / k, ik = 1.0 / k;
        key = 0ULL;
        at = 0;
        for (int i = tid; i < n; i += ADJ_THREADS) {
            const double w = nk * (1. - y[i] / c);   // the forward's expression
            norm[i] = w;
            const unsigned long long o = w == w ? soap_ord64(w + 0.0) : 0ULL;
            if (o > key) {
                key = o;
                at = i;
            }
        }
        int ind_max = block_argmax(key, at, &s_key, &s_idx);   // (its barriers publish norm)
        if (ind_max >= n) ind_max = n - 1;
        const double sig_b = fwhm / 2. / pow(2. * log(2.), .5), ss = sig_b * sig_b, iss = 1.0 / ss, iss2 = iss * iss;
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = 0.0;   // first four: d span / d (c, k, v0, ss)
        for (int t = tid; t < FIT_DEPTHS; t += ADJ_THREADS) {
            const double dep = (double)(t + 5) / 100;
            // depths 0.1 to 0.4 and 0.6 to 0.9: 31 each
            const double w = t >= 5 && t <= 35 ? 1.0 / 31 : t >= 55 && t <= 85 ? -1.0 / 31 : 0.0;
            int i_b = ind_max, i_r = min(ind_max, n - 2);
            while ((norm[i_b] > dep) && (i_b > 1)) i_b--;
            while ((norm[i_r + 1] > dep) && (i_r < (n - 2))) i_r++;
            sp_ib[t] = i_b;
            sp_ir[t] = i_r;
#pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                const int i = min(side ? i_r : i_b, n - 2);
                const double a0 = norm[i], a1 = norm[i + 1], dx = x[i + 1] - x[i], iden = 1.0 / (a1 - a0);
                const double dd = (x[i] + x[i + 1]) / 2. - v0, u = dd * dd * iss;
                const double e = exp(-0.5 * u);
                const double dC = -dd * iss * e, d2C = (u - 1) * iss * e;
                const double idC = 1.0 / dC, ic3 = idC * idC * idC, ic4 = ic3 * idC;
                const double q2 = -0.5 * d2C * ic3;
                const double d3C = e * dd * (3. - u) * iss2;
                const double dCs = dd * e * iss2 * (1. - 0.5 * u);
                const double d2Cs = e * iss2 * ((1. - 2. * u) + (u - 1.) * 0.5 * u);
                const double q2_dd = -0.5 * (d3C * ic3 - 3. * d2C * d2C * ic4);
                const double q2_ss = -0.5 * (d2Cs * ic3 - 3. * d2C * dCs * ic4);
                const double h = 0.5 * w, dxi = dx * iden * iden;
                const double pa0 = h * (dep - a1) * (dxi - q2);
                const double pa1 = -h * (dep - a0) * (dxi + q2);
                const double pq2 = h * (dep - a0) * (dep - a1);
                sp_d[t][2 * side] = pa0;
                sp_d[t][2 * side + 1] = pa1;
                v[0] += -(pa0 + pa1) * ik;
                v[1] += -(pa0 * a0 + pa1 * a1) * ik;
                v[2] += -pq2 * q2_dd;   // dd = vr - v0
                v[3] += pq2 * q2_ss;
            }
        }
        block_sum16(v, sums);   // (its barriers publish sp_ib, sp_ir and sp_d)
        b[0] += gs * sums.tot[0];
        b[1] += gs * sums.tot[1];
        b[2] += gs * sums.tot[2];
        b[3] += gs * sums.tot[3] * 2. * ss / fwhm;   // ss = (fwhm / 2 sqrt(2 ln 2))^2
    }
    {
        int t = 0;
        for (int p = 0; p < 4; ++p)
            for (int q = p; q < 4; ++q, ++t) { A[p * 4 + q] = H[t]; A[q * 4 + p] = H[t]; }
    }
    if (!solve4(A, b, z)) {
        if (tid == 0) atomicExch(status, SOAPGB_ST_FIT_SINGULAR);
        for (int q = 0; q < 4; ++q) z[q] = 0.0;
    }
    for (int i = tid; i < n; i += ADJ_THREADS) {
        const double inv = err ? 1.0 / err[i] : 1.0;
        const double d = x[i] - v0, d2 = d * d;
        const double e = exp(-0.5 * d2 * is2);
        double g = inv * inv * (z[0] + e * z[1] + (k * e * d * is2) * z[2] + (k * e * d2 * a * is3) * z[3]);
        if (gs != 0.0) {   // the span's direct dependence on y_i (through a_i), depths in order
            double dir = 0.0;
            for (int t = 0; t < FIT_DEPTHS; ++t) {
                const int ib = sp_ib[t], ir = sp_ir[t];
                if (ib == i) dir += sp_d[t][0];
                if (ib + 1 == i) dir += sp_d[t][1];
                if (ir == i) dir += sp_d[t][2];
                if (ir + 1 == i) dir += sp_d[t][3];
            }
            g += gs * dir / k;
        }
        gy[i] = g;
    }
}

extern "C" int soapgb_gauss_fit_adjoint(soapgb_ctx *ctx, int n_spec, int n, const double *x, const double *y,
                                        const double *err, const double *model, const double *par,
                                        const double *g_par, int mem, double *grad_y) {
    if (!ctx) return SOAPGB_ERR_ARG;
    if (n_spec < 0 || n < 8 || !x || !y || !model || !par || !g_par || !grad_y)
        return set_error(ctx, SOAPGB_ERR_ARG, "soapgb_gauss_fit_adjoint: bad arguments");
    if (n_spec == 0) return SOAPGB_OK;
    SOAP_DEVICE(ctx);
    const bool host = (mem == SOAPGB_HOST);
    const size_t sb = sizeof(double) * (size_t)n * n_spec, pb = sizeof(double) * 5 * (size_t)n_spec;
    Workspace ws(ctx);
    int s_x = ws.add(host ? sizeof(double) * n : 0);
    int s_y = ws.add(host ? sb : 0), s_e = ws.add(host && err ? sb : 0), s_m = ws.add(host ? sb : 0);
    int s_p = ws.add(host ? pb : 0), s_g = ws.add(host ? pb : 0), s_o = ws.add(host ? sb : 0);
    const bool in_smem = sizeof(double) * (size_t)n <= FIT_SMEM_MAX - 8192;   // the normalised CCF
    int s_scr = ws.add(in_smem ? 0 : sb);
    int rc = ws.commit();
    if (rc) return rc;
#define STAGE(dst, src, bytes, slot)                                                  \
    dst = (const double *)stage_in(ctx, mem, src, bytes, ws.get<void>(slot), &rc);   \
    if (rc) return rc;
    const double *d_x, *d_y, *d_e, *d_m, *d_p, *d_g;
    STAGE(d_x, x, sizeof(double) * n, s_x);
    STAGE(d_y, y, sb, s_y);
    STAGE(d_e, err, err ? sb : 0, s_e);
    STAGE(d_m, model, sb, s_m);
    STAGE(d_p, par, pb, s_p);
    STAGE(d_g, g_par, pb, s_g);
#undef STAGE
    double *d_o = host ? ws.get<double>(s_o) : grad_y;
    SOAP_TRACED(ctx, "gauss_fit_adjoint",
                k_gauss_fit_adj<<<n_spec, ADJ_THREADS, in_smem ? sizeof(double) * n : 0, ctx->stream>>>(
                    n_spec, n, d_x, d_y, d_e, d_m, d_p, d_g, d_o, in_smem ? nullptr : ws.get<double>(s_scr),
                    ctx->d_status));
    SOAP_LAUNCHED(ctx);
    if (host) {
        SOAP_CUDA(ctx, cudaMemcpyAsync(grad_y, d_o, sb, cudaMemcpyDeviceToHost, ctx->stream));
        SOAP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return check_status(ctx, "soapgb_gauss_fit_adjoint");
    }
    return SOAPGB_OK;
}
