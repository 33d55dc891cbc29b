// pair_n3_f64.cu -- the FP64 real-space sum with Newton's third law: every
// unique pair (i < j) is evaluated once in FP64 and its force is added to both
// particles (Force_direct_self / _ext / _sum of force.f90:52-372, whose
// triangular loops also evaluate each pair once).
//
// Bound: the FP64 pipe.  GB300 starts one FP64 warp instruction per 64 cycles
// and SM quarter (596e9 FMA/s measured; conversions to or from FP64 cost the
// same slot), while the other pipes have 64 issue slots in that time, and one
// warp's dependent chain already reaches 94 % of the rate.  So everything that
// can leave the FP64 pipe without a loss in the result does:
//  * the radial functions of force.f90:104-106, 135-139 are Taylor
//    polynomials in x = a^2 r^2 around the centre of the segment that the
//    leading bits of x select (128 segments per octave, 256 above x = 8; tables
//    in shared memory): F(x) = (erfc(ar) + 2ar/sqrt(pi) e^{-x}) / (ar)^3 and
//    U(x) = erfc(ar)/(ar).  The terms from h^4 on are below 2^-24 of the sum
//    and are evaluated in FP32, whose rounding then weighs less than that of x
//    (the errors stand in pair_f64.cuh); the
//    others are four FMAs.  No square root, reciprocal, exponential or
//    erfc per pair.  The e-i terms (Kelbg: e^{-y} y^{-3/2} and
//    sqrt(pi) erfc(sqrt y) - e^{-y} y^{-1/2}, y = r^2/lambda^2; Deutsch:
//    e^{-s}(1+s)/s^3 and e^{-s}/s, s = r/rs) have tables of their own;
//  * the minimum image (force.f90:92) is the wrapped difference of 64-bit
//    fixed-point coordinates, and its conversion to FP64 is done with integer
//    instructions (box_diff);
//  * the segment index, the terms in FP32 and the cut-off test use the bits of
//    r^2; the RDF bin comes from FP32 and takes the FP64 square root only next
//    to a bin edge.
// That leaves 20 FP64 operations per Coulomb pair (r^2 3, h 1, the two
// polynomials 8, energy 1, forces 7), 59 with the table-driven exp, rsqrt and
// erfcx of pair_math.cuh, which stay for the pairs outside the tables (ar < 1/8
// or > 5.6, r < 0.7 lambda or rs) and for the ordered-pair kernel.
//
// And only the pairs inside rc, 52 % of all at rc = L/2, are evaluated: a warp
// finds them with FP32 arithmetic as a bit mask per lane (pair_f64.cuh), each
// lane then takes the next pair of its own i-particle, and when the first lane
// has none left the rest are dealt out over the warp.  A reaction goes to the
// global FP64 force with an atomic per component (91 G/s at the FP64 rate; L2
// takes 200 and more), without an operation on the FP64 pipe.
// Force sums, Kelbg, in us: with exp, rsqrt and erfcx per pair; all pairs from
// the tables; the near pairs alone:
//   N = 65,536   217,900  70,500  41,400 (38,700 at the FP64 rate)
//   N =  3,001     1,495     202     136 (    81)
//
// Work: a warp takes items from an atomic counter: 32 i-particles (a chunk,
// one per lane) against up to `group` j-chunks of 32, in the ring order of
// f64_ring; small systems, whose items would leave SM quarters idle, split the
// j-particles of a tile over `split` items.  The order of the atomics varies
// from run to run, so results vary in the last bits; TCP_FLAG_DETERMINISTIC
// selects the ordered-pair kernel with its fixed-order reduction instead.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "pair_f64.cuh"

namespace tcp {

// Taylor coefficients of function `func` at xc, k = 0..8, in long double (64
// bits or more).  The families obey upward recursions of positive terms for
// the derivatives with respect to -x/2:
//  Ewald    B_{n+1} = ((2n+1) B_n + 2^{n+1}/sqrt(pi) e^{-x})/x
//  Deutsch  A_{n+1} = (A_{n-1} + (2n+1) A_n)/z
//  Kelbg    e^{-y} y^{-p} as the product of two series; the energy's derivative is F/2.
constexpr int kTaylor = 9;
static void gauss_power(long double xc, long double p, long double *out) {   // e^{-x} x^{-p}
    long double e[kTaylor], s[kTaylor];              // e^{-h}, (1 + h/xc)^{-p}
    e[0] = s[0] = 1.0L;
    for (int k = 1; k < kTaylor; ++k) {
        e[k] = -e[k - 1] / k;
        s[k] = s[k - 1] * (-p - (k - 1)) / (k * xc);
    }
    const long double f0 = expl(-xc) * powl(xc, -p);
    for (int k = 0; k < kTaylor; ++k) {
        long double t = 0.0L;
        for (int q = 0; q <= k; ++q) t += e[q] * s[k - q];
        out[k] = f0 * t;
    }
}

// c0 and the series of the derivative -> the series
static void integrate_series(long double c0, long double scale, const long double *d, long double *out) {
    out[0] = c0;
    for (int k = 1; k < kTaylor; ++k) out[k] = scale * d[k - 1] / k;
}

static void taylor_of(int model, int func, long double xc, long double *out) {
    const long double rt = sqrtl(xc), spi = sqrtl(acosl(-1.0L));
    if (model == TCP_EI_KELBG) {
        long double g[kTaylor], f[kTaylor];
        gauss_power(xc, 0.5L, g);
        gauss_power(xc, 1.5L, f);
        if (func == kFuncU) {
            integrate_series(spi * erfcl(rt) - expl(-xc) / rt, 0.5L, f, out);
        } else if (func == kFuncDl) {
            integrate_series(erfcl(rt), -1.0L / spi, g, out);
        } else if (func == kFuncG2) {                // -2 F' = 2 F + 3 e^{-y} y^{-5/2}
            gauss_power(xc, 2.5L, g);
            for (int k = 0; k < kTaylor; ++k) out[k] = 2.0L * f[k] + 3.0L * g[k];
        } else {
            std::copy(func == kFuncGl ? g : f, (func == kFuncGl ? g : f) + kTaylor, out);
        }
        return;
    }
    constexpr int ND = kTaylor + 2;
    long double d[ND];                               // (-2 d/dx)^n of U
    if (model == TCP_EI_DEUTSCH) {
        d[0] = expl(-rt) / rt;
        d[1] = d[0] * (1.0L + rt) / xc;
        for (int n = 1; n + 1 < ND; ++n) d[n + 1] = (d[n - 1] + (2 * n + 1) * d[n]) / xc;
    } else {
        long double g = 2.0L / spi * expl(-xc);
        d[0] = erfcl(rt) / rt;
        for (int n = 0; n + 1 < ND; ++n) {
            d[n + 1] = ((2 * n + 1) * d[n] + g) / xc;
            g *= 2.0L;
        }
    }
    const int n0 = func == kFuncF ? 1 : (func == kFuncG2 ? 2 : 0);
    long double c = 1.0L;                            // (-1/2)^k / k!
    for (int k = 0; k < kTaylor; ++k) {
        out[k] = d[k + n0] * c;
        c *= -0.5L / (k + 1);
    }
    if (func == kFuncDl) {                           // e^{-s}: derivative -A_0/2
        const std::vector<long double> a(out, out + kTaylor);
        integrate_series(expl(-rt), -0.5L, a.data(), out);
    }
}

// Octaves of the tables: the lowest, and how many bits select the segments of each.
struct F64Octaves {
    int low, n, bits[kEiOct];
};
static const F64Octaves &octaves_of(int model) {
    static const F64Octaves ew = {kEwLow, kEwTop - kEwLow, {7, 7, 7, 7, 7, 7, 7, 7, 7, 8, 8}};
    static const F64Octaves kelbg = {kEiLow, 7, {5, 5, 5, 6, 6, 7, 7}};
    static const F64Octaves deutsch = {kEiLow, 12, {5, 5, 5, 5, 5, 5, 5, 6, 6, 6, 5, 5}};
    return model == TCP_EI_COULOMB ? ew : (model == TCP_EI_KELBG ? kelbg : deutsch);
}

static int segments_of(int model) {
    const F64Octaves &o = octaves_of(model);
    int n = 0;
    for (int k = 0; k < o.n; ++k) n += 1 << o.bits[k];
    return n;
}

// the point at fraction f of segment k
static double segment_at(int model, int k, double f) {
    const F64Octaves &o = octaves_of(model);
    int q = 0;
    while (q + 1 < o.n && k >= 1 << o.bits[q]) k -= 1 << o.bits[q++];
    return std::ldexp(1.0 + (k + f) / (1 << o.bits[q]), o.low + q);
}

double f64_segment_end(int model, int k) { return segment_at(model, k, 1.0); }

// One function over all its octaves, [vector][segment]: three vectors, and for
// the e-i families a fourth with t7, t8.  Written once per process.
static std::vector<F64Vec> build_function(int model, int func) {
    const bool ew = model == TCP_EI_COULOMB;
    const int n = segments_of(model);
    std::vector<F64Vec> t((size_t)4 * n);
    for (int s = 0; s < n; ++s) {
        long double c[kTaylor];
        taylor_of(model, func, segment_at(model, s, 0.5), c);
        t[s].d[0] = (double)c[0];
        t[s].d[1] = (double)c[1];
        t[n + s].d[0] = (double)c[2];
        t[n + s].d[1] = (double)c[3];
        F64Vec &v = t[2 * n + s];
        if (ew) {
            for (int k = 0; k < 4; ++k) v.f[k] = (float)c[4 + k];
        } else {
            v.d[0] = (double)c[4];
            v.f[2] = (float)c[5];
            v.f[3] = (float)c[6];
            t[3 * n + s].f[0] = (float)c[7];
            t[3 * n + s].f[1] = (float)c[8];
        }
    }
    return t;
}

static const std::vector<F64Vec> &function_of(int model, int func) {
    static std::once_flag once[3][5];
    static std::vector<F64Vec> tab[3][5];
    const int m = model == TCP_EI_COULOMB ? 0 : (model == TCP_EI_KELBG ? 1 : 2);
    std::call_once(once[m][func], [&] { tab[m][func] = build_function(model, func); });
    return tab[m][func];
}

std::vector<F64Vec> f64_table(int model, const int *funcs, int nf, int segments, int *nseg) {
    const bool ew = model == TCP_EI_COULOMB;
    const int full = (int)function_of(model, funcs[0]).size() / 4;
    const int n = segments > 0 ? std::min(full, segments) : full;
    std::vector<F64Vec> t((size_t)(ew ? ew_vec(nf) : ei_vec(nf)) * n);
    for (int f = 0; f < nf; ++f) {
        const std::vector<F64Vec> &q = function_of(model, funcs[f]);
        for (int v = 0; v < 3; ++v)
            std::copy(q.begin() + (size_t)v * full, q.begin() + (size_t)v * full + n, t.begin() + (size_t)(3 * f + v) * n);
        if (!ew)
            for (int s = 0; s < n; ++s)
                for (int k = 0; k < 2; ++k)
                    t[(size_t)(3 * nf + f / 2) * n + s].f[2 * (f & 1) + k] = q[(size_t)3 * full + s].f[k];
    }
    *nseg = n;
    return t;
}

// The general form of one pair at squared distance r2 (> 0, A^2): the weight w
// (force on i = eps qq w d) and the energy term pe, by rsqrt, exp and erfcx.
template <int KIND>
__device__ __noinline__ void n3_pair_general(const PairConsts &c, double r2, double &w, double &pe, const F64Tab &tb) {
    const double rinv = rsqrt_nr(r2);
    const double r = r2 * rinv;
    const double e = exp_neg_tab(c.alpha2 * r2, tb);
    double s = e * ewald_q(c.alpha * r, tb);              // erfc(ar) + 2ar/sqrt(pi) exp(-a^2 r^2), force.f90:104-106
    // the Ewald energy term erfc(ar)/r (force.f90:105, 1 - erf) = s/r - 2a/sqrt(pi) exp(-a^2 r^2)
    pe = fma(s, rinv, -c.c_gauss_d * e);
    if (KIND == 2) {                                      // Kelbg, e-i pairs
        if (r2 < c.kelbg_far2) {                          // r < 8.5 lambda
            const double g = exp_neg_tab(r2 * c.inv_lam2, tb);
            s -= g;
            pe += c.sqrtpi_lam_d * erfc_tab(r * c.inv_lam, g, tb) - g * rinv;
        }
    } else if (KIND == 1) {                               // Deutsch, force.f90:136-139
        const double y = exp_neg_tab(r * c.inv_rs_d, tb);
        s = s - y - y * r * c.inv_rs_d;
        pe = fma(-y, rinv, pe);
    }
    w = s * (rinv * rinv * rinv);
}

struct F64Shared {
    const uint4 *ew, *ei;
    const int *oct;          // F64Fast::ei_oct
    const F64Tab *tb;
    unsigned *hist;          // RDF: this pair type's bins
};

// One pair of the rotation step: weight (units of a^3) and energy (units of a)
// at r2, zero where !ok.  All lanes of the warp call it.
template <int KIND, bool ENERGY>
__device__ __forceinline__ double n3_pair_f64(const F64Fast &p, const PairConsts &c, double r2, bool ok, double &pe,
                                              const F64Shared &sh) {
    const float r2f = narrow(r2);
    const unsigned xb = __float_as_uint(r2f * p.kxf);
    bool need = ok && (xb < kEwLowBits || xb >= p.ew_hi);   // outside the Ewald table
    const F64At x = ew_at(sh.ew, xb, p.ew_hi, r2, p.kx);
    double w = ew_poly(x, p.ew_seg, 0), u = 0.0;
    w = ok ? w : 0.0;
    if (ENERGY) {
        u = ew_poly(x, p.ew_seg, 1);
        u = ok ? u : 0.0;
    }
    if (KIND != 0) {
        const unsigned yb = __float_as_uint(r2f * p.kyf);
        const bool near = ok && yb < p.ei_hi;
        if (__any_sync(0xffffffffu, near)) {
            need = need || (near && yb < kEiLowBits);
            const F64At y = ei_at(sh.ei, sh.oct, yb, p.ei_hi, r2, p.ky);
            w = fma(near ? p.cf : 0.0, ei_poly<true>(y, p.ei_seg, 0, 2), w);
            if (ENERGY) u = fma(near ? p.cu : 0.0, ei_poly<KIND == 1>(y, p.ei_seg, 1, 2), u);
        }
    }
    if (__any_sync(0xffffffffu, need)) {
        if (need) {
            double wg, ug;
            n3_pair_general<KIND>(c, r2 * p.to_a2, wg, ug, *sh.tb);
            w = wg * p.ia3;
            u = ug * p.ia;
        }
    }
    if (ENERGY) pe += u;
    return w;
}

// RDF: +2 per unique pair inside rc in bin INT(r/dx) of its type
// (force.f90:99-103), from the FP32 root; within 2^-12 of a bin edge from the
// FP64 one.
__device__ __forceinline__ void rdf_add_f64(const F64Fast &p, const PairConsts &c, double r2, bool ok, int pt,
                                            unsigned *hist) {
    const float r2f = narrow(r2);
    const float tb = sqrtf(r2f) * p.rinv_dx[pt];
    int bin = (int)fminf(tb, 1.0e6f);
    const float fr = tb - (float)bin;
    const bool edge = ok && tb < (float)kNbin + 1.0f && (fr < kRdfEdge || fr > 1.0f - kRdfEdge);
    if (__any_sync(0xffffffffu, edge)) {
        if (edge) bin = (int)(sqrt(r2 * p.to_a2) * c.inv_dxd[pt]);
    }
    if (ok && bin < kNbin) atomicAdd(&hist[bin], 2u);
}

// One pair: separation, weight (units of a^3, zero where !ok) and energy.  All
// lanes of the warp call it.
struct F64Pair {
    double w, u[3];
    bool ok;
};
template <int KIND, bool ENERGY, bool RDF, bool CUBIC>
__device__ __forceinline__ F64Pair f64_pair(const F64Fast &p, const N3Args &a, const F64Shared &sh, int pt,
                                            const F64Pos &xi, int j, bool live, double &pe) {
    F64Pair q;
    f64_separation<CUBIC>(a.c, xi, a.xl[j], q.u);
    const double r2 = fma(q.u[0], q.u[0], fma(q.u[1], q.u[1], q.u[2] * q.u[2]));
    // 0 < r2 < rc^2 on the bit patterns (r2 >= 0: they order as the values)
    const long long rb = __double_as_longlong(r2);
    q.ok = live && rb > 0 && rb < __double_as_longlong(p.rc2);
    if (RDF) rdf_add_f64(p, a.c, r2, q.ok, pt, sh.hist);
    q.w = n3_pair_f64<KIND, ENERGY>(p, a.c, r2, q.ok, pe, sh);
    return q;
}

// The near pairs of the warp's 32 i-particles (from i0 on, one per lane) with
// up to 128 j-particles of one species (from j0 on).  As long as every lane
// has one left, each takes its own next; the rest, a few per lane, are dealt
// out evenly.
template <int KIND, bool ENERGY, bool RDF, bool CUBIC>
__device__ __forceinline__ void f64_near(const F64Fast &p, const N3Args &a, const F64Shared &sh, int pt, int i0,
                                         const F64Pos &xi, int j0, F64Mask m, double (&fi)[3], double &pe) {
    const double qf = p.qf[pt];
    const size_t n = a.ntot;
#pragma unroll 1
    while (__all_sync(0xffffffffu, (m.lo | m.hi) != 0)) {
        const int j = j0 + mask_pop(m);
        const F64Pair q = f64_pair<KIND, ENERGY, RDF, CUBIC>(p, a, sh, pt, xi, j, true, pe);
        const double w = qf * q.w;
        fi[0] = fma(w, q.u[0], fi[0]);
        fi[1] = fma(w, q.u[1], fi[1]);
        fi[2] = fma(w, q.u[2], fi[2]);
        if (q.ok) add_force(a.facc + j, n, -w * q.u[0], -w * q.u[1], -w * q.u[2]);
    }
    const F64Deal deal = mask_deal(m);
#pragma unroll 1
    for (int t0 = 0; t0 < deal.total; t0 += 32) {
        const F64Dealt t = mask_dealt(m, deal, t0);
        F64Pos x;
        x.x = __shfl_sync(0xffffffffu, xi.x, t.lane);
        x.y = __shfl_sync(0xffffffffu, xi.y, t.lane);
        x.z = __shfl_sync(0xffffffffu, xi.z, t.lane);
        const int j = j0 + t.bit;
        const F64Pair q = f64_pair<KIND, ENERGY, RDF, CUBIC>(p, a, sh, pt, x, j, t.live, pe);
        if (q.ok) {
            const double w = qf * q.w, fx = w * q.u[0], fy = w * q.u[1], fz = w * q.u[2];
            add_force(a.facc + i0 + t.lane, n, fx, fy, fz);
            add_force(a.facc + j, n, -fx, -fy, -fz);
        }
    }
}

template <int EI, bool ENERGY, bool RDF, bool CUBIC>
__global__ void __launch_bounds__(kF64Threads, 1) pair_n3_f64_kernel(const N3Args a, const F64Fast p) {
    extern __shared__ __align__(128) uint4 tabs[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ double red[32];
    __shared__ unsigned hist[RDF ? 3 * kNbin : 1];
    __shared__ F64Tab tab;
    __shared__ int oct[kEiOct];
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < kEiOct) oct[tid] = p.ei_oct[tid];
    if (RDF)
        for (int k = tid; k < 3 * kNbin; k += kF64Threads) hist[k] = 0u;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        if (!(a.inject_skip && blockIdx.x == 0)) {        // test hook: the copy never comes
            const uint32_t b0 = (uint32_t)p.ew_seg * ew_vec(2) * 16u, b1 = (uint32_t)p.ei_seg * ei_vec(2) * 16u;
            mbar_arrive_expect_tx(&bar, b0 + b1);
            bulk_g2s(tabs, p.tab, b0, &bar);
            if (b1) bulk_g2s(tabs + p.ew_seg * ew_vec(2), p.tab + p.ew_seg * ew_vec(2), b1, &bar);
        }
    }
    load_f64_tab(tab);
    __syncthreads();
    const bool got = mbar_wait_bounded(&bar, 0u, kWaitLimitCycles);
    if (__syncthreads_or(!got)) {
        if (tid == 0) atomicOr(a.status, kStatusTmaTimeout);
        return;
    }
    F64Shared sh;
    sh.ew = tabs;
    sh.ei = tabs + p.ew_seg * ew_vec(2);
    sh.oct = oct;
    sh.tb = &tab;
    sh.hist = nullptr;
    double etot = 0.0;
    for (;;) {
        unsigned nx = 0;
        if (lane == 0) nx = atomicAdd(a.counter, 1u);
        const long long it = __shfl_sync(0xffffffffu, nx, 0);
        if (it >= p.items) break;
        int ca, d0, nd, part, istart, icnt, isp;
        f64_ring(p, it, ca, d0, nd, part);
        f64_chunk(p, a.g, ca, istart, icnt, isp);
        const longlong4_32a t = a.xl[istart + min(lane, icnt - 1)];
        const F64Pos xi{t.x, t.y, t.z};
        double fi[3] = {0.0, 0.0, 0.0};
        for (F64Run r{d0, d0 + nd}; f64_run(p, a.g, ca, isp, r);) {
            const F64Mask m = f64_mask(p, a.xl, xi, lane < icnt, r.j0, r.nj, r.diag, part);
            double pe = 0.0;
            if (RDF) sh.hist = hist + r.pt * kNbin;
            if (EI != 0 && r.pt == 1)
                f64_near<EI, ENERGY, RDF, CUBIC>(p, a, sh, r.pt, istart, xi, r.j0, m, fi, pe);
            else
                f64_near<0, ENERGY, RDF, CUBIC>(p, a, sh, r.pt, istart, xi, r.j0, m, fi, pe);
            if (ENERGY) etot = fma(p.qe[r.pt], pe, etot);
        }
        if (lane < icnt) add_force(a.facc + istart + lane, a.ntot, fi[0], fi[1], fi[2]);
    }
    if (ENERGY) {
        const double tot = block_sum(etot, red);
        if (tid == 0) a.upart[blockIdx.x] = tot;
    }
    if (RDF) {
        __syncthreads();
        for (int q = tid; q < 3 * kNbin; q += kF64Threads)
            if (hist[q]) atomicAdd(&a.rdf[q], (unsigned long long)hist[q]);
    }
}

// ---------------------------------------------------------------------------
typedef void (*F64Kernel)(const N3Args, const F64Fast);
template <int EI>
static F64Kernel f64_kernel_of(bool energy, bool rdf, bool cubic) {
    if (cubic) {
        if (energy) return rdf ? pair_n3_f64_kernel<EI, true, true, true> : pair_n3_f64_kernel<EI, true, false, true>;
        return rdf ? pair_n3_f64_kernel<EI, false, true, true> : pair_n3_f64_kernel<EI, false, false, true>;
    }
    if (energy) return rdf ? pair_n3_f64_kernel<EI, true, true, false> : pair_n3_f64_kernel<EI, true, false, false>;
    return rdf ? pair_n3_f64_kernel<EI, false, true, false> : pair_n3_f64_kernel<EI, false, false, false>;
}

static F64Kernel f64_kernel(const tcp_ctx *c, bool energy, bool rdf) {
    const bool cubic = c->pc.cubic != 0;
    if (c->p.ei_model == TCP_EI_DEUTSCH) return f64_kernel_of<1>(energy, rdf, cubic);
    if (c->p.ei_model == TCP_EI_KELBG) return f64_kernel_of<2>(energy, rdf, cubic);
    return f64_kernel_of<0>(energy, rdf, cubic);
}

bool n3_f64_applicable(const tcp_ctx *c) {
    return c->p.precision == TCP_PREC_FP64 && c->n >= 2 && !(c->flags & TCP_FLAG_DETERMINISTIC);
}

int n3_f64_grid(const tcp_ctx *c) { return std::max(1, c->num_sms); }   // the tables: one CTA per SM

// The table ends past the cut-off by more than the rounding of the FP32
// argument: pairs at its end would take the general form.
int ewald_segments(const tcp_ctx *c) {
    const F64Octaves &o = octaves_of(TCP_EI_COULOMB);
    const double x = c->pc.alpha2 * c->rc2 * (1.0 + 1e-6);
    int n = 0;
    for (int q = 0; q < o.n; ++q) {
        const double low = std::ldexp(1.0, o.low + q), part = std::min(std::max(x / low - 1.0, 0.0), 1.0);
        n += (int)std::ceil(part * (1 << o.bits[q]));
    }
    return std::max(n, 1 << kEwBits);
}

static const int kPairFuncs[] = {kFuncF, kFuncU};
static size_t f64_smem(int ew_seg, int ei_seg) { return 16 * ((size_t)ew_seg * ew_vec(2) + (size_t)ei_seg * ei_vec(2)); }

// Device tables of an FP64 context for its e-i model and cut-off (rebuilt with
// the pair constants, outside any stream capture).
int n3_f64_prepare(tcp_ctx *c) {
    int ew = 0, ei = 0;
    std::vector<F64Vec> t = f64_table(TCP_EI_COULOMB, kPairFuncs, 2, ewald_segments(c), &ew);
    if (c->p.ei_model != TCP_EI_COULOMB) {
        const std::vector<F64Vec> m = f64_table(c->p.ei_model, kPairFuncs, 2, 0, &ei);
        t.insert(t.end(), m.begin(), m.end());
    }
    adj_tables_free(c);                  // they follow the same parameters
    cudaFree(c->f64tab);
    c->f64tab = nullptr;
    TCP_CUDA(cudaMalloc(&c->f64tab, sizeof(F64Vec) * t.size()));
    TCP_CUDA(cudaMemcpy(c->f64tab, t.data(), sizeof(F64Vec) * t.size(), cudaMemcpyHostToDevice));
    c->f64_ew_seg = ew;
    c->f64_ei_seg = ei;
    for (int k = 0; k < 4; ++k)
        if (int rc = allow_shared(reinterpret_cast<const void *>(f64_kernel(c, k & 1, (k & 2) != 0)), f64_smem(ew, ei)))
            return rc;
    return TCP_OK;
}

// The upper words of two coordinates are less than a unit of 2^-32 of the box
// off, and the FP32 arithmetic of f64_mask 1e-6.
float f64_near2(const PairConsts &pc, double r) {
    const double box = pc.cubic ? 1.0 : std::max(pc.box[0], std::max(pc.box[1], pc.box[2]));
    const double b = r + 4.0 * box / 4294967296.0;
    return (float)(b * b * 1.00001);
}

// Constants and items for tables of ew_seg and ei_seg segments.
F64Fast f64_args(const tcp_ctx *c, int ew_seg, int ei_seg) {
    const PairConsts &pc = c->pc;
    const double L = pc.cubic ? pc.box[0] : 1.0, l = c->p.ei_model == TCP_EI_DEUTSCH ? pc.rs : pc.lambda;
    const double al = pc.alpha, a3 = al * al * al;
    F64Fast p;
    std::memset(&p, 0, sizeof p);
    p.ew_seg = ew_seg;
    p.ei_seg = ei_seg;
    auto end_bits = [](int model, int segments) {
        const float e = (float)f64_segment_end(model, segments - 1);
        unsigned b;
        std::memcpy(&b, &e, sizeof b);
        return b;
    };
    p.ew_hi = ew_seg ? end_bits(TCP_EI_COULOMB, ew_seg) : kEwLowBits + 1;
    if (ei_seg) {
        p.ei_hi = end_bits(c->p.ei_model, ei_seg);
        const F64Octaves &o = octaves_of(c->p.ei_model);
        for (int q = 0, n = 0; q < o.n; n += 1 << o.bits[q++]) {
            const int sh = 23 - o.bits[q];
            p.ei_oct[q] = sh + 32 * (n - (int)((unsigned)(127 + o.low + q) << o.bits[q]));
        }
    }
    p.kx = pc.alpha2 * (L * L);
    p.kxf = (float)p.kx;
    p.to_a2 = L * L;
    // the smallest r^2 whose rounded product with to_a2 reaches rc^2, so that
    // the cut-off test equals the one in A^2 to the last bit (rc = L/2 and
    // lattice positions put pairs exactly on it)
    p.rc2 = pc.rc2 / p.to_a2;
    while (p.rc2 * p.to_a2 < pc.rc2) p.rc2 = std::nextafter(p.rc2, HUGE_VAL);
    for (double t; (t = std::nextafter(p.rc2, 0.0)) * p.to_a2 >= pc.rc2;) p.rc2 = t;
    for (int d = 0; d < 3; ++d) p.boxf[d] = (float)((pc.cubic ? 1.0 : pc.box[d]) / 4294967296.0);
    p.near2 = f64_near2(pc, std::sqrt(p.rc2));
    p.ia3 = 1.0 / a3;
    p.ia = 1.0 / al;
    if (p.ei_seg) {
        p.ky = L * L / (l * l);
        p.kyf = (float)p.ky;
        p.cf = -1.0 / (l * l * l * a3);
        p.cu = (c->p.ei_model == TCP_EI_KELBG ? 1.0 : -1.0) / (l * al);
    }
    for (int t = 0; t < 3; ++t) {
        p.qf[t] = kEps * pc.qq[t] * a3 * L;
        p.qe[t] = pc.qq[t] * al;
        p.rinv_dx[t] = (float)(L * pc.inv_dxd[t]);
    }
    // Items of four tiles (their near pairs deal out to full warps, and the
    // last ones are a small part of the launch), smaller ones where fewer items
    // would leave SM quarters idle at the end, down to eighths of a tile where
    // there is not one for every warp.  Measured (us) at group/split 4/1, 2/1,
    // 1/1, 1/2, 1/4, 1/8: N = 24,000 5,768 5,817 5,946; 9,000 935 900 910;
    // 5,000 354 335 316 321 343; 3,001 230 183 145 136 142 157;
    // 1,500 230 125 75 60 53 56; 512 204 121 73 45 31 26.
    p.nce = (c->nel + 31) / 32;
    p.nc = p.nce + (c->nion + 31) / 32;
    const long long tiles = (long long)p.nc * (p.nc + 1) / 2, quarters = 4LL * c->num_sms;
    p.group = tiles >= 150 * quarters ? 4 : (tiles >= 50 * quarters ? 2 : 1);
    p.split = tiles >= 14 * quarters ? 1 : (tiles >= 5 * quarters ? 2 : (2 * tiles >= 3 * quarters ? 4 : 8));
    p.nd = p.nc / 2 + 1;
    auto items = [&p] { return (long long)p.nc * ((p.nd + p.group - 1) / p.group) * p.split; };
    while (items() > 0x7fffffff) p.group *= 2;   // the counter and f64_ring are 32-bit
    p.items = items();
    return p;
}

int launch_pair_n3_f64(tcp_ctx *c, bool energy, bool rdf, bool cleared) {
    if (!c->f64tab) return set_error(TCP_ERR_STATE, "no FP64 pair tables");
    N3Args a;
    std::memset(&a, 0, sizeof a);
    a.g.nel = c->nel;
    a.g.n = c->n;
    a.xl = c->xl;
    a.ntot = c->n;
    a.facc = c->fpart;
    a.upart = c->upart;
    a.status = c->status;
    a.counter = c->counter;
    a.c = c->pc;
    a.inject_skip = inject_fault("tile_wait") ? 1 : 0;
    a.rdf = c->rdf;
    F64Fast p = f64_args(c, c->f64_ew_seg, c->f64_ei_seg);
    p.tab = reinterpret_cast<const uint4 *>(c->f64tab);
    const int grid = (int)std::min<long long>(n3_f64_grid(c), (p.items + kF64Warps - 1) / kF64Warps);
    if (grid > c->n_upart) return set_error(TCP_ERR_STATE, "energy partial buffer smaller than the Newton-3 grid");
    c->n_upart_used = grid;
    if (!cleared) {
        TCP_CUDA(cudaMemsetAsync(c->fpart, 0, sizeof(double) * 3 * (size_t)c->n, c->stream));
        TCP_CUDA(cudaMemsetAsync(c->counter, 0, sizeof(unsigned), c->stream));
    }
    f64_kernel(c, energy, rdf)<<<grid, kF64Threads, f64_smem(p.ew_seg, p.ei_seg), c->stream>>>(a, p);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

}  // namespace tcp
