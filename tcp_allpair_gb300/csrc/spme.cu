// spme.cu -- reciprocal-space sums: smooth PME (Force_SPME4, force.f90:652-929,
// generalised to B-spline order 4..8) and the plain Ewald k-sum.
//
// Mesh layout: Q[iz][iy][ix] (ix fastest, the Fortran order of Q(ix,iy,iz)),
// FP64.  Cubic meshes of 32, 48, 64, 96 or 128 points a side are spread and
// convolved by spme_fft.cu; for the others the 3-D FFT is cuFFT D2Z / Z2D on
// that layout (the only library call of the path), with the influence multiply
// and energy reduction of this file between.  Spreading (cell-sorted and
// atomic-free) and force gather: spme_chain.cu.
// In the compensated-FP32 mode the charge mesh is summed in two-float FP32
// and written as FP32 for R2C / C2R transforms, the influence multiply
// (energy summed in FP64) and the force gather: on GB300 FP64 runs at 1/64 of
// the FP32 rate, which makes a 128^3 FP64 transform compute-bound.
// TCP_PREC_FP32C_R64 keeps the FP32C real-space sum and runs this chain in
// FP64 as in TCP_PREC_FP64.
//
// Normalisation: both transforms are unnormalised, so the real mesh after the
// inverse transform is phi = K^3 Qfin of the reference; its 1/K^3 (FFTE
// iopt=+1) and K^3 (force.f90:864-865) cancel, giving
//   Um = eps/(2 pi V) sum_m theta(m) B(m) |S(m)|^2          (force.f90:921)
//   F_i = -eps/(pi V) sum_k dQ(k)/dx_i phi(k)              (force.f90:882-887)
#include <algorithm>
#include <cmath>
#include <functional>
#include <vector>

#include "device_util.cuh"
#include "spme_chain.cuh"
#include "tcp_internal.h"

namespace tcp {

// Qk *= theta B; energy partial sum_m w_m theta B |Qk|^2 (w = 2 for the
// kx columns that stand for a conjugate pair in the half spectrum).
__global__ void spme_influence_kernel(cufftDoubleComplex *__restrict__ Qk, const double *__restrict__ infl,
                                      long total, int Kh, int K1, double *__restrict__ epart, bool energy) {
    __shared__ double red[32];
    double e = 0.0;
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
        const double g = infl[idx];
        cufftDoubleComplex z = Qk[idx];
        if (energy) {
            const int kx = (int)(idx % Kh);
            const double wgt = (kx == 0 || (2 * kx == K1)) ? 1.0 : 2.0;
            e += wgt * g * (z.x * z.x + z.y * z.y);
        }
        z.x *= g;
        z.y *= g;
        Qk[idx] = z;
    }
    if (energy) {
        const double t = block_sum(e, red);
        if (threadIdx.x == 0) epart[blockIdx.x] = t;
    }
}

// FP32C influence multiply.  Energy terms are summed in FP32 per thread (a
// few elements each) and in FP64 across threads and blocks.  The half-spectrum
// column kx of element idx advances by the grid stride modulo Kh, so no
// division runs per element.
__global__ void spme_influence_f_kernel(cufftComplex *__restrict__ Qk, const float *__restrict__ infl, int total,
                                        int Kh, int K1, double *__restrict__ epart, bool energy) {
    __shared__ double red[32];
    float e = 0.0f;
    const int stride = gridDim.x * blockDim.x;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    int kx = idx % Kh;
    const int dkx = stride % Kh;
    for (; idx < total; idx += stride) {
        const float g = infl[idx];
        cufftComplex z = Qk[idx];
        if (energy) {
            const float wgt = (kx == 0 || (2 * kx == K1)) ? 1.0f : 2.0f;
            e = fmaf(wgt * g, fmaf(z.x, z.x, z.y * z.y), e);
        }
        z.x *= g;
        z.y *= g;
        Qk[idx] = z;
        kx += dkx;
        if (kx >= Kh) kx -= Kh;
    }
    if (energy) {
        const double t = block_sum((double)e, red);
        if (threadIdx.x == 0) epart[blockIdx.x] = t;
    }
}

// ---- plain Ewald k-sum ------------------------------------------------------
// S(m) = sum_j q_j exp(2 pi i m.x_j) and the forces, by the product form
// exp(2 pi i m.x) = ex[n1] ey[n2] ez[n3] of one phase factor per particle, axis
// and index instead of a sine and cosine per particle and k-vector, and over
// the half space n1 >= 0 (S(-m) is the conjugate; n1 > 0 counts twice).  Bound:
// the FP64 pipe, about 5 operations per (k, j) for S and 7 per (k, i) for the
// forces, one complex factor ey ez serving all n1 of a column (n2, n3).  N =
// 1,024, |n|^2 <= 64 (2,108 vectors): 74 us for the whole sum, 2,922 us with
// sincos per term and the force kernel on N/128 CTAs.
//
// Items: a column (n2, n3) with up to kEwN1 consecutive n1, columns with the
// longest n1 range first, so that the lanes of a warp run equally far.
constexpr int kEwN1 = 9;
constexpr int kEwThreads = 256;
constexpr int kEwPart = 8;        // particles whose phases a CTA holds at a time

struct EwArgs {
    const double *x;
    int nel, n;
    double q0, q1;
    double iL[3];
    int nm;               // largest index
    int nitem;
    const int4 *item;     // n2, n3, first n1, n1 count
    const double *th;     // [kEwN1][nitem]: theta(m), doubled for n1 > 0, 0 outside the sphere
    double2 *part;        // [CTA][kEwN1][nitem] partial S
    double2 *Z;           // [kEwN1][nitem]: th conj(S)
    double *epart;
    int nblk, per;        // CTAs of the S kernel, particles per CTA
};

// exp(2 pi i n u) with n u reduced to the nearest integer first (exact for the
// leading part of the product, so the phase error does not grow with n)
__device__ __forceinline__ double2 ew_phase(int n, double u) {
    const double p = n * u, e = fma((double)n, u, -p);
    const double f = (p - rint(p)) + e;
    double s, c;
    sincospi(2.0 * f, &s, &c);
    return make_double2(c, s);
}

// partial S over the particles of this CTA, one item per thread (grid.y groups of items)
__global__ void __launch_bounds__(kEwThreads) ewald_sfac_kernel(const EwArgs a) {
    extern __shared__ double2 ph[];               // [3][nm + 1][kEwPart]
    __shared__ double sq[kEwPart];
    const int np = a.nm + 1;
    const int it = blockIdx.y * kEwThreads + threadIdx.x;
    const int4 im = it < a.nitem ? a.item[it] : make_int4(0, 0, 0, 0);
    const int i2 = abs(im.x), i3 = abs(im.y);
    const double s2 = im.x < 0 ? -1.0 : 1.0, s3 = im.y < 0 ? -1.0 : 1.0;
    const int cnt = __reduce_max_sync(0xffffffffu, im.w);
    double2 S[kEwN1];
#pragma unroll
    for (int k = 0; k < kEwN1; ++k) S[k] = make_double2(0.0, 0.0);
    const int j0 = blockIdx.x * a.per, j1 = min(a.n, j0 + a.per);
    for (int jb = j0; jb < j1; jb += kEwPart) {
        const int nj = min(kEwPart, j1 - jb);
        __syncthreads();
        for (int k = threadIdx.x; k < 3 * np * nj; k += kEwThreads) {
            const int j = k % nj, r = k / nj, n = r % np, d = r / np;
            ph[(d * np + n) * kEwPart + j] = ew_phase(n, a.x[(size_t)d * a.n + jb + j] * a.iL[d]);
        }
        if (threadIdx.x < nj) sq[threadIdx.x] = jb + (int)threadIdx.x < a.nel ? a.q0 : a.q1;
        __syncthreads();
        for (int j = 0; j < nj; ++j) {
            const double2 ey = ph[(np + i2) * kEwPart + j], ez = ph[(2 * np + i3) * kEwPart + j];
            const double q = sq[j], yr = q * ey.x, yi = (q * s2) * ey.y, zi = s3 * ez.y;
            const double er = fma(yr, ez.x, -yi * zi), ei = fma(yr, zi, yi * ez.x);
            const double2 *ex = ph + im.z * kEwPart + j;
#pragma unroll
            for (int k = 0; k < kEwN1; ++k)
                if (k < cnt) {
                    const double2 e = ex[min(k, np - 1 - im.z) * kEwPart];
                    S[k].x = fma(er, e.x, fma(-ei, e.y, S[k].x));
                    S[k].y = fma(er, e.y, fma(ei, e.x, S[k].y));
                }
        }
    }
    if (it < a.nitem) {
        double2 *o = a.part + (size_t)blockIdx.x * kEwN1 * a.nitem + it;
#pragma unroll
        for (int k = 0; k < kEwN1; ++k) o[(size_t)k * a.nitem] = S[k];
    }
}

// Z = th conj(S), S the sum of the partials (a warp per eight vectors: lanes
// over the CTAs' partials would stride by whole arrays), and the energy
// partials sum th |S|^2 per CTA
__global__ void __launch_bounds__(kEwThreads) ewald_sum_kernel(const EwArgs a) {
    __shared__ double2 sm[kEwThreads];
    __shared__ double red[32];
    const int total = kEwN1 * a.nitem;
    const int v = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.x * 32 + v;   // 32 vectors, 8 slices
    double sr = 0.0, si = 0.0;
    if (k < total)
        for (int b = w; b < a.nblk; b += kEwThreads / 32) {
            const double2 z = a.part[(size_t)b * total + k];
            sr += z.x;
            si += z.y;
        }
    sm[threadIdx.x] = make_double2(sr, si);
    __syncthreads();
    double e = 0.0;
    if (w == 0 && k < total) {
        sr = si = 0.0;
        for (int b = 0; b < kEwThreads / 32; ++b) {
            sr += sm[b * 32 + v].x;
            si += sm[b * 32 + v].y;
        }
        const double t = a.th[k];
        a.Z[k] = make_double2(t * sr, -t * si);
        e = t * fma(sr, sr, si * si);
    }
    e = block_sum(e, red);
    if (threadIdx.x == 0) a.epart[blockIdx.x] = e;
}

// F_i = (2 eps q_i / V) sum_m theta m Im(conj(S) e^{i phase}); a warp per
// particle, lanes over the items, so every particle count fills the SMs and
// the sum over k-vectors ends in one warp reduction.  The last CTA adds up the
// energy partials.
__global__ void __launch_bounds__(kEwThreads) ewald_force_kernel(const EwArgs a, double coef,
                                                                 double *__restrict__ frec, int npart, double escale,
                                                                 double *__restrict__ um) {
    extern __shared__ double2 ph[];               // [warps][3][nm + 1]
    __shared__ double red[32];
    if (blockIdx.x == gridDim.x - 1) {
        double e = 0.0;
        for (int k = threadIdx.x; um && k < npart; k += kEwThreads) e += a.epart[k];
        e = block_sum(e, red);
        if (um && threadIdx.x == 0) *um = e * escale;
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, np = a.nm + 1;
    const int i = blockIdx.x * (kEwThreads / 32) + warp;
    if (i >= a.n) return;                         // warp-uniform
    double2 *p = ph + (size_t)warp * 3 * np;
    for (int k = lane; k < 3 * np; k += 32) p[k] = ew_phase(k % np, a.x[(size_t)(k / np) * a.n + i] * a.iL[k / np]);
    __syncwarp();
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int it = lane; it < a.nitem; it += 32) {
        const int4 im = a.item[it];
        double tr = 0.0, ti = 0.0, xr = 0.0, xi = 0.0;   // sum t_k, sum k t_k (as the sum of the suffix sums)
        for (int k = im.w - 1; k >= 0; --k) {
            const double2 z = a.Z[(size_t)k * a.nitem + it], e = p[im.z + k];
            tr = fma(z.x, e.x, fma(-z.y, e.y, tr));
            ti = fma(z.x, e.y, fma(z.y, e.x, ti));
            if (k > 0) {
                xr += tr;
                xi += ti;
            }
        }
        if (im.z) {
            xr = fma((double)im.z, tr, xr);
            xi = fma((double)im.z, ti, xi);
        }
        const double2 ey = p[np + abs(im.x)], ez = p[2 * np + abs(im.y)];
        const double yi = im.x < 0 ? -ey.y : ey.y, zi = im.y < 0 ? -ez.y : ez.y;
        const double er = fma(ey.x, ez.x, -yi * zi), ei = fma(ey.x, zi, yi * ez.x);
        const double im_t = fma(er, ti, ei * tr);
        fx = fma(er, xi, fma(ei, xr, fx));
        fy = fma((double)im.x, im_t, fy);
        fz = fma((double)im.y, im_t, fz);
    }
    fx = warp_sum(fx);
    fy = warp_sum(fy);
    fz = warp_sum(fz);
    if (lane == 0) {
        const double q = coef * (i < a.nel ? a.q0 : a.q1);
        frec[i] = q * a.iL[0] * fx;
        frec[(size_t)a.n + i] = q * a.iL[1] * fy;
        frec[2 * (size_t)a.n + i] = q * a.iL[2] * fz;
    }
}

// ---------------------------------------------------------------------------
static double bspline_M(int n, double y) {
    if (y <= 0.0 || y >= (double)n) return 0.0;
    if (n == 2) return 1.0 - std::fabs(y - 1.0);
    return (y * bspline_M(n - 1, y) + ((double)n - y) * bspline_M(n - 1, y - 1.0)) / (double)(n - 1);
}

// |b(m)|^-2 per axis (36/(4+2cos)^2 for order 4, force.f90:834-839); odd
// orders vanish at the Nyquist index, where the mean of the neighbours is used.
std::vector<double> bspline_moduli(int order, int K) {
    std::vector<double> den(K), out(K);
    for (int m = 0; m < K; ++m) {
        if (order == 4) {
            const double z = 4.0 + 2.0 * std::cos(2.0 * kPi * m / K);
            den[m] = z * z / 36.0;
            continue;
        }
        double re = 0.0, im = 0.0;
        for (int k = 0; k <= order - 2; ++k) {
            const double mk = bspline_M(order, (double)(k + 1));
            re += mk * std::cos(2.0 * kPi * m * k / K);
            im += mk * std::sin(2.0 * kPi * m * k / K);
        }
        den[m] = re * re + im * im;
    }
    for (int m = 0; m < K; ++m)
        if (den[m] < 1e-7) den[m] = 0.5 * (den[(m - 1 + K) % K] + den[(m + 1) % K]);
    for (int m = 0; m < K; ++m) out[m] = 1.0 / den[m];
    return out;
}

int spme_free(tcp_ctx *c) {
    if (c->plans) {
        cufftDestroy(c->plan_f);
        cufftDestroy(c->plan_b);
        c->plans = false;
    }
    chain_free(c->bins);
    cudaFree(c->fft_tw32);
    cudaFree(c->fft_tw64);
    c->fft_tw32 = c->fft_tw64 = nullptr;
    cudaFree(c->Q);
    cudaFree(c->Qk);
    cudaFree(c->infl);
    cudaFree(c->Qf);
    cudaFree(c->Qkf);
    cudaFree(c->infl_f);
    c->Q = nullptr;
    c->Qk = nullptr;
    c->infl = nullptr;
    c->Qf = nullptr;
    c->Qkf = nullptr;
    c->infl_f = nullptr;
    return TCP_OK;
}

// blocks of 256 threads for the influence multiply: about four elements per
// thread, at most 4096 blocks (the size of the energy partial array)
static int spme_energy_blocks(const tcp_ctx *c) {
    const long total = (long)c->K3 * c->K2 * c->Kh;
    return (int)std::max<long>(1, std::min<long>((total + 1023) / 1024, 4096));
}

int spme_setup(tcp_ctx *c) {
    const tcp_params &p = c->p;
    c->K1 = p.K[0];
    c->K2 = p.K[1];
    c->K3 = p.K[2];
    c->Kh = c->K1 / 2 + 1;
    const size_t nreal = (size_t)c->K1 * c->K2 * c->K3;
    const size_t nhalf = (size_t)c->Kh * c->K2 * c->K3;
    c->spme_fp32 = c->p.precision == TCP_PREC_FP32C && !c->recip_fp64;
    if (!c->Q) {
        if (int rc = chain_alloc(c->bins, c->n, c->K2 * c->K3, p.order)) return rc;
        if (cudaMalloc(&c->Q, sizeof(double) * nreal) != cudaSuccess ||
            cudaMalloc(&c->Qk, sizeof(cufftDoubleComplex) * nhalf) != cudaSuccess ||
            cudaMalloc(&c->infl, sizeof(double) * nhalf) != cudaSuccess)
            return set_error(TCP_ERR_NOMEM, "SPME mesh allocation failed");
        if (c->spme_fp32 && (cudaMalloc(&c->Qf, sizeof(float) * nreal) != cudaSuccess ||
                             cudaMalloc(&c->Qkf, sizeof(cufftComplex) * nhalf) != cudaSuccess ||
                             cudaMalloc(&c->infl_f, sizeof(float) * nhalf) != cudaSuccess))
            return set_error(TCP_ERR_NOMEM, "SPME FP32 mesh allocation failed");
    }
    c->own_fft = fft_own(c->K1, c->K2, c->K3);
    if (c->own_fft) {
        for (const bool d : {false, true}) {
            if (!d && !c->spme_fp32) continue;
            if (int rc = fft_twiddles(c->K1, d, d ? &c->fft_tw64 : &c->fft_tw32)) return rc;
            if (int rc = fft_prepare(spme_chain_args(c), c->K1, d)) return rc;
        }
    } else if (!c->plans) {
        if (inject_fault("cufft_plan")) return set_error(TCP_ERR_CUFFT, "injected: cufftPlan3d failed");
        const cufftType tf = c->spme_fp32 ? CUFFT_R2C : CUFFT_D2Z;
        const cufftType tb = c->spme_fp32 ? CUFFT_C2R : CUFFT_Z2D;
        if (cufftPlan3d(&c->plan_f, c->K3, c->K2, c->K1, tf) != CUFFT_SUCCESS)
            return set_error(TCP_ERR_CUFFT, "cufftPlan3d forward failed");
        if (cufftPlan3d(&c->plan_b, c->K3, c->K2, c->K1, tb) != CUFFT_SUCCESS) {
            cufftDestroy(c->plan_f);
            return set_error(TCP_ERR_CUFFT, "cufftPlan3d inverse failed");
        }
        cufftSetStream(c->plan_f, c->stream);
        cufftSetStream(c->plan_b, c->stream);
        c->plans = true;
    }
    if (int rc = chain_prepare(spme_chain_args(c))) return rc;
    // theta(m) = exp(-pi^2 m^2/a^2)/m^2 (EWALD_SELF, force.f90:27-42) times
    // the B-spline moduli, on the half spectrum; theta(0) = 0.
    std::vector<double> bx = bspline_moduli(p.order, c->K1), by = bspline_moduli(p.order, c->K2),
                        bz = bspline_moduli(p.order, c->K3);
    std::vector<double> h(nhalf);
    const double a2 = c->alpha * c->alpha;
    for (int k = 0; k < c->K3; ++k) {
        const int iz = (k + c->K3 / 2) % c->K3 - c->K3 / 2;
        for (int j = 0; j < c->K2; ++j) {
            const int iy = (j + c->K2 / 2) % c->K2 - c->K2 / 2;
            for (int i = 0; i < c->Kh; ++i) {
                const int ix = (i + c->K1 / 2) % c->K1 - c->K1 / 2;
                const size_t idx = i + (size_t)c->Kh * (j + (size_t)c->K2 * k);
                if (ix == 0 && iy == 0 && iz == 0) {
                    h[idx] = 0.0;
                    continue;
                }
                const double m2 = (double)ix * ix / (p.box[0] * p.box[0]) + (double)iy * iy / (p.box[1] * p.box[1]) +
                                  (double)iz * iz / (p.box[2] * p.box[2]);
                h[idx] = std::exp(-m2 * kPi * kPi / a2) / m2 * bx[i] * by[j] * bz[k];
            }
        }
    }
    if (c->own_fft) {   // in the order of fft_convolve's transforms
        const std::vector<int> order = fft_order(c->K1);
        std::vector<double> t(nhalf);
        for (size_t i = 0; i < nhalf; ++i) t[i] = h[order[i]];
        h.swap(t);
    }
    TCP_CUDA(cudaMemcpyAsync(c->infl, h.data(), sizeof(double) * nhalf, cudaMemcpyHostToDevice, c->stream));
    if (c->spme_fp32) {
        std::vector<float> hf(h.begin(), h.end());
        TCP_CUDA(cudaMemcpyAsync(c->infl_f, hf.data(), sizeof(float) * nhalf, cudaMemcpyHostToDevice, c->stream));
        TCP_CUDA(cudaStreamSynchronize(c->stream));
    }
    TCP_CUDA(cudaStreamSynchronize(c->stream));
    return TCP_OK;
}

ChainArgs spme_chain_args(tcp_ctx *c) {
    ChainArgs a;
    a.n = c->n;
    a.nbins = c->K2 * c->K3;
    a.P = c->p.order;
    a.fp64 = !c->spme_fp32;
    a.k1max = c->K1;
    a.k2max = c->K2;
    a.planes = c->K3;
    a.nsys = 1;
    a.b = c->bins;
    const int K[3] = {c->K1, c->K2, c->K3};
    a.one.off = 0;
    a.one.nel = c->nel;
    a.one.bin_off = 0;
    a.one.plane_off = 0;
    a.one.mesh_off = 0;
    for (int d = 0; d < 3; ++d) {
        a.one.K[d] = K[d];
        a.one.hL[d] = c->p.box[d] * .5;
        a.one.KL[d] = (double)K[d] / c->p.box[d];
    }
    for (int t = 0; t < 2; ++t) a.one.q[t] = c->p.charge_scale * c->p.q[t];
    a.one.half_off = 0;
    a.one.own = c->own_fft;
    a.one.coef = kEps / (kPi * c->V);
    a.one.ecoef = kEps / (2.0 * kPi * c->V);
    a.many = nullptr;
    a.sys_of = nullptr;
    a.mesh = c->spme_fp32 ? (void *)c->Qf : (void *)c->Q;
    a.dipole = nullptr;
    a.ticket = c->tickets + kTickBin;
    return a;
}

// fft_convolve's arrays: the FP64 ones also serve the Hessian-vector products
// of FP32C contexts
static FftArgs spme_fft_args(tcp_ctx *c, bool fp64, bool energy) {
    FftArgs f;
    f.half = fp64 ? (void *)c->Qk : (void *)c->Qkf;
    f.infl = fp64 ? (const void *)c->infl : (const void *)c->infl_f;
    f.tw = fp64 ? c->fft_tw64 : c->fft_tw32;
    f.list = nullptr;
    f.epart = recip_epart(c);
    f.um = nullptr;
    f.energy = energy;
    return f;
}

// the red[] region after the force and kinetic partials holds the energy partials
double *recip_epart(tcp_ctx *c);

int launch_spme(tcp_ctx *c, bool energy) {
    const ChainArgs chain = spme_chain_args(c);
    if (!c->binned) c->launches += chain_bin(chain, c->x, c->rstream);
    c->binned = false;
    c->launches += chain_sort(chain, c->rstream);
    const long total = (long)c->K3 * c->K2 * c->Kh;
    const int eb = c->own_fft ? fft_energy_parts(c->K1) : spme_energy_blocks(c);
    double *epart = recip_epart(c);
    if (c->own_fft) {
        const FftArgs f = spme_fft_args(c, !c->spme_fp32, energy);
        c->launches += fft_convolve(chain, f, c->K1, 1, c->rstream);
        c->launches += chain_gather(chain, c->frec, epart, eb, kEps / (2.0 * kPi * c->V),
                                    energy ? c->scal + kScalUm : nullptr, c->rstream);
        TCP_CUDA(cudaGetLastError());
        return TCP_OK;
    }
    c->launches += chain_spread(chain, c->rstream);
    cufftSetStream(c->plan_f, c->rstream);
    cufftSetStream(c->plan_b, c->rstream);
    if (c->spme_fp32) {
        if (cufftExecR2C(c->plan_f, c->Qf, c->Qkf) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecR2C failed");
        spme_influence_f_kernel<<<eb, 256, 0, c->rstream>>>(c->Qkf, c->infl_f, (int)total, c->Kh, c->K1, epart, energy);
        c->launches++;
        if (cufftExecC2R(c->plan_b, c->Qkf, c->Qf) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecC2R failed");
    } else {
        if (cufftExecD2Z(c->plan_f, c->Q, c->Qk) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecD2Z failed");
        spme_influence_kernel<<<eb, 256, 0, c->rstream>>>(c->Qk, c->infl, total, c->Kh, c->K1, epart, energy);
        c->launches++;
        if (cufftExecZ2D(c->plan_b, c->Qk, c->Q) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecZ2D failed");
    }
    c->launches += chain_gather(chain, c->frec, epart, eb, kEps / (2.0 * kPi * c->V),
                                energy ? c->scal + kScalUm : nullptr, c->rstream);
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

void ewald_free(tcp_ctx *c) {
    void **bufs[] = {(void **)&c->kvec, (void **)&c->kS4, (void **)&c->ew_item, (void **)&c->ew_th,
                     (void **)&c->ew_part, (void **)&c->ew_z};
    for (void **b : bufs) {
        cudaFree(*b);
        *b = nullptr;
    }
}

int ewald_setup(tcp_ctx *c) {
    const tcp_params &p = c->p;
    const int nmax2 = p.ewald_nmax2;
    const int nm = (int)std::floor(std::sqrt((double)nmax2));
    std::vector<double> kv;
    for (int n3 = -nm; n3 <= nm; ++n3)
        for (int n2 = -nm; n2 <= nm; ++n2)
            for (int n1 = -nm; n1 <= nm; ++n1) {
                const int nn = n1 * n1 + n2 * n2 + n3 * n3;
                if (nn == 0 || nn > nmax2) continue;
                const double m[3] = {n1 / p.box[0], n2 / p.box[1], n3 / p.box[2]};
                const double m2 = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
                kv.push_back(m[0]);
                kv.push_back(m[1]);
                kv.push_back(m[2]);
                kv.push_back(std::exp(-m2 * kPi * kPi / (c->alpha * c->alpha)) / m2);
            }
    c->nk = (int)(kv.size() / 4);
    if (c->nk > c->red_cap - 7 * part_blocks(c->n))
        return set_error(TCP_ERR_BAD_PARAM, "ewald_nmax2 too large: more k-vectors than the energy buffer holds");
    ewald_free(c);
    if (c->nk == 0) return TCP_OK;
    TCP_CUDA(cudaMalloc(&c->kvec, sizeof(double) * kv.size()));
    TCP_CUDA(cudaMemcpyAsync(c->kvec, kv.data(), sizeof(double) * kv.size(), cudaMemcpyHostToDevice, c->stream));
    // items of the half space n1 >= 0, the longest columns first
    std::vector<int4> items;
    for (int base = 0; base <= nm; base += kEwN1)
        for (int n3 = -nm; n3 <= nm; ++n3)
            for (int n2 = -nm; n2 <= nm; ++n2) {
                const int rest = nmax2 - n2 * n2 - n3 * n3;
                int top = -1;
                while (top < nm && (top + 1) * (top + 1) <= rest) ++top;
                if (top >= base) items.push_back(make_int4(n2, n3, base, std::min(kEwN1, top - base + 1)));
            }
    std::stable_sort(items.begin(), items.end(), [](const int4 &p, const int4 &q) { return p.w > q.w; });
    const int ni = (int)items.size();
    std::vector<double> th((size_t)kEwN1 * ni, 0.0);
    for (int it = 0; it < ni; ++it)
        for (int k = 0; k < items[it].w; ++k) {
            const int n1 = items[it].z + k;
            if (n1 == 0 && items[it].x == 0 && items[it].y == 0) continue;
            const double m[3] = {n1 / p.box[0], items[it].x / p.box[1], items[it].y / p.box[2]};
            const double m2 = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
            th[(size_t)k * ni + it] = (n1 > 0 ? 2.0 : 1.0) * std::exp(-m2 * kPi * kPi / (c->alpha * c->alpha)) / m2;
        }
    // CTAs of the S kernel: one per SM and group of items, fewer where their
    // partial sums would take more than 64 MB
    const size_t per_cta = sizeof(double2) * kEwN1 * (size_t)ni;
    int blocks = std::min((c->n + kEwPart - 1) / kEwPart, c->num_sms);
    blocks = std::max(1, std::min<int>(blocks, (int)((64u << 20) / per_cta)));
    const int per = (((c->n + blocks - 1) / blocks) + kEwPart - 1) / kEwPart * kEwPart;
    c->ew_nblk = (c->n + per - 1) / per;
    c->ew_per = per;
    c->ew_nitem = ni;
    c->ew_nm = nm;
    if (cudaMalloc(&c->ew_item, sizeof(int4) * (size_t)ni) != cudaSuccess ||
        cudaMalloc(&c->ew_th, sizeof(double) * th.size()) != cudaSuccess ||
        cudaMalloc(&c->ew_part, per_cta * c->ew_nblk) != cudaSuccess || cudaMalloc(&c->ew_z, per_cta) != cudaSuccess)
        return set_error(TCP_ERR_NOMEM, "Ewald sum: device allocation failed");
    TCP_CUDA(cudaMemcpyAsync(c->ew_item, items.data(), sizeof(int4) * (size_t)ni, cudaMemcpyHostToDevice, c->stream));
    TCP_CUDA(cudaMemcpyAsync(c->ew_th, th.data(), sizeof(double) * th.size(), cudaMemcpyHostToDevice, c->stream));
    TCP_CUDA(cudaStreamSynchronize(c->stream));
    return TCP_OK;
}

int launch_ewald(tcp_ctx *c, bool energy) {
    if (c->nk == 0) {
        TCP_CUDA(cudaMemsetAsync(c->frec, 0, sizeof(double) * 3 * (size_t)c->n, c->rstream));
        TCP_CUDA(cudaMemsetAsync(c->scal + kScalUm, 0, sizeof(double), c->rstream));
        return TCP_OK;
    }
    EwArgs a;
    a.x = c->x;
    a.nel = c->nel;
    a.n = c->n;
    a.q0 = c->p.charge_scale * c->p.q[0];
    a.q1 = c->p.charge_scale * c->p.q[1];
    for (int d = 0; d < 3; ++d) a.iL[d] = 1.0 / c->p.box[d];
    a.nm = c->ew_nm;
    a.nitem = c->ew_nitem;
    a.item = c->ew_item;
    a.th = c->ew_th;
    a.part = c->ew_part;
    a.Z = c->ew_z;
    a.epart = recip_epart(c);
    a.nblk = c->ew_nblk;
    a.per = c->ew_per;
    // at most 10 KB: ewald_setup takes no more than 73,728 vectors, indexes up to 26
    const size_t phases = sizeof(double2) * 3 * (size_t)(a.nm + 1);
    const dim3 sgrid(a.nblk, (a.nitem + kEwThreads - 1) / kEwThreads);
    const int nsum = (kEwN1 * a.nitem + 31) / 32, wpb = kEwThreads / 32;
    ewald_sfac_kernel<<<sgrid, kEwThreads, phases * kEwPart, c->rstream>>>(a);
    ewald_sum_kernel<<<nsum, kEwThreads, 0, c->rstream>>>(a);
    ewald_force_kernel<<<(c->n + wpb - 1) / wpb + 1, kEwThreads, phases * wpb, c->rstream>>>(
        a, 2.0 * kEps / c->V, c->frec, nsum, kEps / (2.0 * kPi * c->V), energy ? c->scal + kScalUm : nullptr);
    c->launches += 3;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

// ---- reciprocal-space Hessian-vector products -------------------------------
// With Q(k) = sum_j q_j W_j(k), phi = A Q (the convolution of launch_spme) and
// E = c/2 Q.phi, c = eps/(pi V):
//   (H w)_i = c q_i [sum_k (hess W_i(k) w_i) phi(k) + sum_k grad W_i(k) dphi(k)],
//   dphi = A dQ, dQ(k) = sum_j q_j grad W_j(k) . w_j.
// Always FP64 (meshes hQ / hdQ, own D2Z / Z2D plans), whatever the precision
// of the force path.

void spme_hvp_free(tcp_ctx *c) {
    if (c->hplans) {
        cufftDestroy(c->hplan_f);
        cufftDestroy(c->hplan_b);
        c->hplans = false;
    }
    cudaFree(c->hQ);
    cudaFree(c->hdQ);
    cudaFree(c->hQk);
    cudaFree(c->kS4);
    c->hQ = c->hdQ = nullptr;
    c->hQk = nullptr;
    c->kS4 = nullptr;
}

int launch_spme_hvp(tcp_ctx *c, const double *w, double *hw, const std::function<int()> &real) {
    const size_t nreal = (size_t)c->K1 * c->K2 * c->K3;
    const size_t nhalf = (size_t)c->Kh * c->K2 * c->K3;
    if (!c->hQ) {
        if (cudaMalloc(&c->hQ, sizeof(double) * nreal) != cudaSuccess ||
            cudaMalloc(&c->hdQ, sizeof(double) * nreal) != cudaSuccess ||
            cudaMalloc(&c->hQk, sizeof(cufftDoubleComplex) * nhalf) != cudaSuccess)
            return set_error(TCP_ERR_NOMEM, "SPME Hessian mesh allocation failed");
    }
    if (!c->own_fft && !c->hplans) {
        if (cufftPlan3d(&c->hplan_f, c->K3, c->K2, c->K1, CUFFT_D2Z) != CUFFT_SUCCESS)
            return set_error(TCP_ERR_CUFFT, "cufftPlan3d D2Z failed");
        if (cufftPlan3d(&c->hplan_b, c->K3, c->K2, c->K1, CUFFT_Z2D) != CUFFT_SUCCESS) {
            cufftDestroy(c->hplan_f);
            return set_error(TCP_ERR_CUFFT, "cufftPlan3d Z2D failed");
        }
        cufftSetStream(c->hplan_f, c->stream);
        cufftSetStream(c->hplan_b, c->stream);
        c->hplans = true;
    }
    const long total = (long)nhalf;
    const int eb = spme_energy_blocks(c);
    double *mesh[2] = {c->hQ, c->hdQ};
    ChainArgs chain = spme_chain_args(c);
    chain.fp64 = 1;
    // The sort and phi = A Q run on stream2, beside the real-space part that
    // `real` queues on the main stream; dphi = A dQ follows that part there.
    // Each of these kernels leaves most of the GPU idle (N = 4,096, 32^3: 32
    // CTAs): one after the other H w took 267 us through the C call (FP32C), so 203 us.
    TCP_CUDA(cudaEventRecord(c->ev_fork, c->stream));
    TCP_CUDA(cudaStreamWaitEvent(c->stream2, c->ev_fork, 0));
    c->launches += chain_bin(chain, c->x, c->stream2);
    c->launches += chain_sort(chain, c->stream2);
    TCP_CUDA(cudaEventRecord(c->ev_pair_ready, c->stream2));
    if (int rc = real()) {
        TCP_CUDA(cudaStreamWaitEvent(c->stream, c->ev_pair_ready, 0));   // the sort: later calls sort into the same arrays
        return rc;
    }
    for (int pass = 0; pass < 2; ++pass) {
        chain.mesh = mesh[pass];
        chain.dipole = pass ? w : nullptr;
        if (c->own_fft) {
            FftArgs f = spme_fft_args(c, true, false);
            if (pass) {
                f.half = c->hQk;                       // beside the other convolution's
                TCP_CUDA(cudaStreamWaitEvent(c->stream, c->ev_pair_ready, 0));
            }
            c->launches += fft_convolve(chain, f, c->K1, 1, pass ? c->stream : c->stream2);
            if (!pass) TCP_CUDA(cudaEventRecord(c->ev_join, c->stream2));
            continue;
        }
        if (!pass) {                                   // cuFFT meshes: one plan, one after the other
            TCP_CUDA(cudaEventRecord(c->ev_join, c->stream2));
            TCP_CUDA(cudaStreamWaitEvent(c->stream, c->ev_join, 0));
        }
        c->launches += chain_spread(chain, c->stream);
        if (cufftExecD2Z(c->hplan_f, mesh[pass], c->hQk) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecD2Z failed");
        spme_influence_kernel<<<eb, 256, 0, c->stream>>>(c->hQk, c->infl, total, c->Kh, c->K1, nullptr, false);
        if (cufftExecZ2D(c->hplan_b, c->hQk, mesh[pass]) != CUFFT_SUCCESS) return set_error(TCP_ERR_CUFFT, "cufftExecZ2D failed");
        c->launches++;
    }
    TCP_CUDA(cudaStreamWaitEvent(c->stream, c->ev_join, 0));
    c->launches += chain_gather_hvp(chain, c->hQ, c->hdQ, w, hw, c->stream);
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

// plain Ewald: S(m) and dS(m) = sum_j q_j (2 pi i m.w_j) e^{i ph_j} per k-vector
__global__ void ewald_dsfac_kernel(const double *__restrict__ x, const double *__restrict__ w, int nel, int n,
                                   double q0, double q1, const double *__restrict__ kvec, double *__restrict__ kS4) {
    __shared__ double red[32];
    const double mx = kvec[4 * blockIdx.x], my = kvec[4 * blockIdx.x + 1], mz = kvec[4 * blockIdx.x + 2];
    double sr = 0.0, si = 0.0, dr = 0.0, di = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const double q = j < nel ? q0 : q1;
        const double ph = 2.0 * kPi * (mx * x[j] + my * x[(size_t)n + j] + mz * x[2 * (size_t)n + j]);
        const double mw = 2.0 * kPi * (mx * w[j] + my * w[(size_t)n + j] + mz * w[2 * (size_t)n + j]);
        double s, c;
        sincos(ph, &s, &c);
        sr += q * c;
        si += q * s;
        dr -= q * mw * s;
        di += q * mw * c;
    }
    sr = block_sum(sr, red);
    si = block_sum(si, red);
    dr = block_sum(dr, red);
    di = block_sum(di, red);
    if (threadIdx.x == 0) {
        kS4[4 * blockIdx.x] = sr;
        kS4[4 * blockIdx.x + 1] = si;
        kS4[4 * blockIdx.x + 2] = dr;
        kS4[4 * blockIdx.x + 3] = di;
    }
}

// (H w)_i = -(2 eps/V) q_i sum_m theta m [Im(conj(dS) e^{i ph_i}) + 2 pi (m.w_i) Re(conj(S) e^{i ph_i})]
__global__ void ewald_hvp_kernel(const double *__restrict__ x, const double *__restrict__ w, int nel, int n,
                                 double q0, double q1, const double *__restrict__ kvec,
                                 const double *__restrict__ kS4, int nk, double coef, double *__restrict__ hw) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double q = i < nel ? q0 : q1;
    const double xi = x[i], yi = x[(size_t)n + i], zi = x[2 * (size_t)n + i];
    const double wx = w[i], wy = w[(size_t)n + i], wz = w[2 * (size_t)n + i];
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;
    for (int k = 0; k < nk; ++k) {
        const double mx = kvec[4 * k], my = kvec[4 * k + 1], mz = kvec[4 * k + 2], th = kvec[4 * k + 3];
        double s, c;
        sincos(2.0 * kPi * (mx * xi + my * yi + mz * zi), &s, &c);
        const double mw = 2.0 * kPi * (mx * wx + my * wy + mz * wz);
        const double im_d = kS4[4 * k + 2] * s - kS4[4 * k + 3] * c;
        const double re_s = kS4[4 * k] * c + kS4[4 * k + 1] * s;
        const double t = th * (im_d + mw * re_s);
        h0 += t * mx;
        h1 += t * my;
        h2 += t * mz;
    }
    hw[i] += coef * q * h0;
    hw[(size_t)n + i] += coef * q * h1;
    hw[2 * (size_t)n + i] += coef * q * h2;
}

int launch_ewald_hvp(tcp_ctx *c, const double *w, double *hw) {
    if (c->nk == 0) return TCP_OK;
    if (!c->kS4 && cudaMalloc(&c->kS4, sizeof(double) * 4 * (size_t)c->nk) != cudaSuccess)
        return set_error(TCP_ERR_NOMEM, "Ewald Hessian buffer allocation failed");
    const double q0 = c->p.charge_scale * c->p.q[0], q1 = c->p.charge_scale * c->p.q[1];
    ewald_dsfac_kernel<<<c->nk, 256, 0, c->stream>>>(c->x, w, c->nel, c->n, q0, q1, c->kvec, c->kS4);
    ewald_hvp_kernel<<<(c->n + 127) / 128, 128, 0, c->stream>>>(c->x, w, c->nel, c->n, q0, q1, c->kvec, c->kS4,
                                                                c->nk, -2.0 * kEps / c->V, hw);
    c->launches += 2;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

}  // namespace tcp
