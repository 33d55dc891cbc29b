// pair_n3_f64.cu -- the FP64 real-space sum with Newton's third law: every
// unique pair (i < j) is evaluated once in FP64 and its force is added to both
// particles (Force_direct_self / _ext / _sum of force.f90:52-372, whose
// triangular loops also evaluate each pair once).
//
// Bound: the FP64 pipe.  GB300 starts one FP64 warp instruction per 64 cycles
// and SM quarter (596e9 FMA/s measured; conversions to or from FP64 cost the
// same slot), while the other pipes have 64 issue slots in that time, and one
// warp's dependent chain already reaches 94 % of the rate.  So everything that
// can leave the FP64 pipe without losing a bit of the result does:
//  * the radial functions of force.f90:104-106, 135-139 are Taylor
//    polynomials in x = a^2 r^2 around the centre of the segment that the
//    leading bits of x select (128 segments per octave, tables in shared
//    memory): F(x) = (erfc(ar) + 2ar/sqrt(pi) e^{-x}) / (ar)^3 and
//    U(x) = erfc(ar)/(ar).  With |h| <= 2^-8 x the terms from h^4 on are
//    below 2^-31 of the sum and are evaluated in FP32 without loss; the
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
// That leaves 19 FP64 operations per Coulomb pair (r^2 3, h 1, the two
// polynomials 8, energy 1, the six force components 6), 59 with the
// table-driven exp, rsqrt and erfcx of pair_math.cuh (N = 65,536, Kelbg: 217.9 ms a
// force call with those, 70.5 ms with the tables; N = 3,001: 1,495 against 202 us), which stay for the pairs
// below the tables (ar < 1/8, or r < lambda/8 or rs/8: about one in 10^5) and
// for the ordered-pair kernel.
//
// Work: a warp takes items from an atomic counter: 32 i-particles (a chunk,
// one per lane) against up to `group` j-chunks of 32; j's position and
// reaction rotate through the warp with shuffles.  Small systems, whose items
// would leave SM quarters idle, split the 32 rotation steps of a tile over
// `split` items.  Forces and energies are summed in FP64 per item and added to
// the global FP64 force with one atomic per particle and component.  The order
// of those atomics varies from run to run, so results vary in the last bits;
// TCP_FLAG_DETERMINISTIC selects the ordered-pair kernel with its fixed-order
// reduction instead.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "device_util.cuh"
#include "pair_n3.cuh"

namespace tcp {

// Three warps per SM quarter hide the latency of the FP32 and integer work and
// leave registers and shared memory for the reciprocal chain beside the launch.
constexpr int kF64Threads = 384;
constexpr int kF64Warps = kF64Threads / 32;

// ---- tables ---------------------------------------------------------------------
// Segments of an argument x in [2^-6, 2^top): the leading kEwBits (kEiBits)
// mantissa bits of x.  Per segment and function the coefficients c0..c3 (Ewald)
// or c0..c4 (e-i) in FP64 and the magnitudes of the four next ones in FP32,
// in 16-byte vectors [vector][segment] so that lanes on different segments
// use different banks.
constexpr int kEwBits = 7, kEwVec = 6;   // F: c0 c1 | c2 c3 | t4..t7, then U the same
constexpr int kEiBits = 5, kEiVec = 7;   // F: c0 c1 | c2 c3 | c4 t5 t6, U the same, then t7 t8 of F and U
constexpr int kTabLow = -6;              // the tables start at 2^-6
constexpr unsigned kTabLowBits = (127 + kTabLow) << 23;
constexpr int kEwTopMax = 6;             // Ewald: erfc(ar) is 0 beyond ar = 8 (1e-29 of the pair's 1/r)
constexpr int kKelbgTop = 6;             // Kelbg: e^{-64} = 1.6e-28
constexpr int kDeutschTop = 11;          // Deutsch: e^{-45} = 2.6e-20 of the pair's Coulomb term

// Taylor coefficients of F and U at xc, k = 0..8, in the working precision of
// long double (64 bits or more).  All three families obey upward recursions
// of positive terms for the derivatives with respect to -x/2:
//  Ewald    B_{n+1} = ((2n+1) B_n + 2^{n+1}/sqrt(pi) e^{-x})/x,  U = B_0, F = B_1
//  Deutsch  A_{n+1} = (A_{n-1} + (2n+1) A_n)/z,                  U = A_0, F = A_1
//  Kelbg    F = e^{-y} y^{-3/2} as the product of two series; U' = F/2.
constexpr int kTaylor = 9;
static void taylor_of(int model, long double xc, long double *F, long double *U) {
    const long double rt = sqrtl(xc);
    if (model == TCP_EI_KELBG) {
        const long double spi = sqrtl(acosl(-1.0L));
        long double e[kTaylor], s[kTaylor];          // e^{-h}, (1 + h/xc)^{-3/2}
        e[0] = s[0] = 1.0L;
        for (int k = 1; k < kTaylor; ++k) {
            e[k] = -e[k - 1] / k;
            s[k] = s[k - 1] * (-1.5L - (k - 1)) / (k * xc);
        }
        const long double f0 = expl(-xc) / (xc * rt);
        for (int k = 0; k < kTaylor; ++k) {
            long double t = 0.0L;
            for (int q = 0; q <= k; ++q) t += e[q] * s[k - q];
            F[k] = f0 * t;
        }
        U[0] = spi * erfcl(rt) - expl(-xc) / rt;
        for (int k = 1; k < kTaylor; ++k) U[k] = 0.5L * F[k - 1] / k;
        return;
    }
    long double d[kTaylor + 1];                      // (-2 d/dx)^n of U
    if (model == TCP_EI_DEUTSCH) {
        d[0] = expl(-rt) / rt;
        d[1] = d[0] * (1.0L + rt) / xc;
        for (int n = 1; n < kTaylor; ++n) d[n + 1] = (d[n - 1] + (2 * n + 1) * d[n]) / xc;
    } else {
        long double g = 2.0L / sqrtl(acosl(-1.0L)) * expl(-xc);
        d[0] = erfcl(rt) / rt;
        for (int n = 0; n < kTaylor; ++n) {
            d[n + 1] = ((2 * n + 1) * d[n] + g) / xc;
            g *= 2.0L;
        }
    }
    long double c = 1.0L;                            // (-1/2)^k / k!
    for (int k = 0; k < kTaylor; ++k) {
        U[k] = d[k] * c;
        F[k] = d[k + 1] * c;
        c *= -0.5L / (k + 1);
    }
}

static long double segment_centre(int k, int bits) {
    const int oct = kTabLow + (k >> bits), m = k & ((1 << bits) - 1);
    return ldexpl(1.0L + (m + 0.5L) / (1 << bits), oct);
}

struct F64Vec {
    union {
        double d[2];
        float f[4];
    };
};

// Full Ewald table (all octaves), or one e-i table; written once per process.
static std::vector<F64Vec> build_table(int model) {
    const bool ew = model == TCP_EI_COULOMB;
    const int bits = ew ? kEwBits : kEiBits, nvec = ew ? kEwVec : kEiVec;
    const int top = ew ? kEwTopMax : (model == TCP_EI_KELBG ? kKelbgTop : kDeutschTop);
    const int nseg = (top - kTabLow) << bits;
    std::vector<F64Vec> t((size_t)nvec * nseg);
    for (int s = 0; s < nseg; ++s) {
        long double c[2][kTaylor];
        taylor_of(model, segment_centre(s, bits), c[0], c[1]);
        for (int q = 0; q < 2; ++q) {
            double *lo = t[(size_t)(3 * q) * nseg + s].d, *mid = t[(size_t)(3 * q + 1) * nseg + s].d;
            lo[0] = (double)c[q][0];
            lo[1] = (double)c[q][1];
            mid[0] = (double)c[q][2];
            mid[1] = (double)c[q][3];
            F64Vec &v = t[(size_t)(3 * q + 2) * nseg + s];
            if (ew) {
                for (int k = 0; k < 4; ++k) v.f[k] = (float)c[q][4 + k];
            } else {   // T = t5 + t6 h + ...: of one sign within a family (F and U alternate)
                v.d[0] = (double)c[q][4];
                v.f[2] = (float)c[q][5];
                v.f[3] = (float)c[q][6];
                t[(size_t)6 * nseg + s].f[2 * q] = (float)c[q][7];
                t[(size_t)6 * nseg + s].f[2 * q + 1] = (float)c[q][8];
            }
        }
    }
    return t;
}

static const std::vector<F64Vec> &table_of(int model) {
    static const std::vector<F64Vec> ew = build_table(TCP_EI_COULOMB), ke = build_table(TCP_EI_KELBG),
                                     de = build_table(TCP_EI_DEUTSCH);
    return model == TCP_EI_KELBG ? ke : (model == TCP_EI_DEUTSCH ? de : ew);
}

// What the kernel needs besides PairConsts.  Lengths in units of the box where
// it is cubic (the fixed-point differences unscaled), in A otherwise.
struct F64Fast {
    const uint4 *tab;        // Ewald vectors, then e-i vectors
    int ew_seg, ei_seg;      // segments per vector
    unsigned ew_hi, ei_hi;   // float bits of the table ends
    double kx, ky;           // r^2 -> a^2 r^2, r^2/lambda^2 (or /rs^2)
    float kxf, kyf;
    double rc2;              // cut-off^2 (r^2 < rc2)
    double to_a2;            // r^2 -> A^2 (the general form)
    double cf, cu;           // weight and energy of the e-i term in units of the Ewald term's a^3 and a
    double ia3, ia;          // 1/a^3, 1/a
    double qf[3], qe[3];     // force factor (eV/A per unit weight and separation) and energy factor per pair type
    float rinv_dx[3];        // RDF: sqrt(r^2) -> r/dx
    int group, split;        // j-chunks per item; items per tile of rotation steps
    int nce, nc, ng;         // electron chunks, chunks, groups
    long long total;
};

// ---- pair arithmetic --------------------------------------------------------------
// (double)d 2^-64 for a 64-bit integer d without the FP64 pipe: the magnitude
// is normalised by its leading zeros, rounded to 53 bits and packed.  Valid
// for a nonzero upper word of the magnitude; small is set otherwise.
__device__ __forceinline__ double box_diff(long long d, bool &small) {
    const long long sg = d >> 63;
    const unsigned long long mag = (unsigned long long)((d ^ sg) - sg);
    const unsigned s = (unsigned)sg, ah = (unsigned)(mag >> 32), al = (unsigned)mag;
    const int z = __clz((int)ah);
    const unsigned nh = __funnelshift_l(al, ah, z), nl = al << (z & 31);
    const unsigned hi = (nh >> 11) + ((1021u - (unsigned)z) << 20), lo = __funnelshift_r(nl, nh, 11);
    const unsigned long long v = (((unsigned long long)hi << 32) | lo) + ((nl >> 10) & 1u);
    small = small || ah == 0u;
    return __hiloint2double((int)((unsigned)(v >> 32) | (s & 0x80000000u)), (int)(unsigned)v);
}

// positive normal float -> double without the FP64 pipe
__device__ __forceinline__ double widen(float t) {
    const unsigned b = __float_as_uint(t);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// the leading 24 bits of a double >= 0 as a float (0 below the normal floats;
// the separations stay far below their upper end)
__device__ __forceinline__ float narrow(double x) {
    const unsigned hi = (unsigned)__double2hiint(x);
    const unsigned b = __funnelshift_l((unsigned)__double2loint(x), hi, 3) + 0x40000000u;
    return __uint_as_float(hi < 0x38100000u ? 0u : b);
}

__device__ __forceinline__ double2 lds2(const uint4 *p) { return *reinterpret_cast<const double2 *>(p); }
__device__ __forceinline__ float4 lds4(const uint4 *p) { return *reinterpret_cast<const float4 *>(p); }

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
    bool need = ok && xb < kTabLowBits;                   // below the tables
    const unsigned xi = min(max(xb, kTabLowBits), p.ew_hi - 1u);
    const unsigned cb = (xi & ~((1u << (23 - kEwBits)) - 1u)) | (1u << (22 - kEwBits));   // segment centre
    const uint4 *t = sh.ew + ((xi - kTabLowBits) >> (23 - kEwBits));
    const double h = fma(r2, p.kx, -widen(__uint_as_float(cb)));
    const float hf = fmaf(r2f, p.kxf, -__uint_as_float(cb));
    const int n = p.ew_seg;
    const double2 f01 = lds2(t), f23 = lds2(t + n);
    const float4 f4 = lds4(t + 2 * n);
    double w = fma(h, widen(fmaf(fmaf(fmaf(f4.w, hf, f4.z), hf, f4.y), hf, f4.x)), f23.y);
    w = fma(h, fma(h, fma(h, w, f23.x), f01.y), f01.x);
    double u = 0.0;
    if (ENERGY) {
        const double2 u01 = lds2(t + 3 * n), u23 = lds2(t + 4 * n);
        const float4 u4 = lds4(t + 5 * n);
        u = fma(h, widen(fmaf(fmaf(fmaf(u4.w, hf, u4.z), hf, u4.y), hf, u4.x)), u23.y);
        u = fma(h, fma(h, fma(h, u, u23.x), u01.y), u01.x);
    }
    const bool in = ok && xb < p.ew_hi;
    w = in ? w : 0.0;
    u = in ? u : 0.0;
    if (KIND != 0) {
        const unsigned yb = __float_as_uint(r2f * p.kyf);
        const bool near = ok && yb < p.ei_hi;
        if (__any_sync(0xffffffffu, near)) {
            need = need || (near && yb < kTabLowBits);
            const unsigned yi = min(max(yb, kTabLowBits), p.ei_hi - 1u);
            const unsigned db = (yi & ~((1u << (23 - kEiBits)) - 1u)) | (1u << (22 - kEiBits));
            const uint4 *s = sh.ei + ((yi - kTabLowBits) >> (23 - kEiBits));
            const double g = fma(r2, p.ky, -widen(__uint_as_float(db)));
            const float gf = fmaf(r2f, p.kyf, -__uint_as_float(db));
            const int m = p.ei_seg;
            const float4 t78 = lds4(s + 6 * m);
            // the FP32 part T has the sign of its leading term: F negative
            // (k = 5), U negative for Deutsch, positive for Kelbg (U' = F/2)
            const double2 a01 = lds2(s), a23 = lds2(s + m), a4 = lds2(s + 2 * m);
            const float a5 = __int_as_float(__double2loint(a4.y)), a6 = __int_as_float(__double2hiint(a4.y));
            const float tf = fmaf(fmaf(fmaf(t78.y, gf, t78.x), gf, a6), gf, a5);
            double v = fma(-g, widen(-tf), a4.x);
            v = fma(g, fma(g, fma(g, fma(g, v, a23.y), a23.x), a01.y), a01.x);
            w = fma(near ? p.cf : 0.0, v, w);
            if (ENERGY) {
                const double2 b01 = lds2(s + 3 * m), b23 = lds2(s + 4 * m), b4 = lds2(s + 5 * m);
                const float b5 = __int_as_float(__double2loint(b4.y)), b6 = __int_as_float(__double2hiint(b4.y));
                const float tu = fmaf(fmaf(fmaf(t78.w, gf, t78.z), gf, b6), gf, b5);
                v = KIND == 2 ? fma(g, widen(tu), b4.x) : fma(-g, widen(-tu), b4.x);
                v = fma(g, fma(g, fma(g, fma(g, v, b23.y), b23.x), b01.y), b01.x);
                u = fma(near ? p.cu : 0.0, v, u);
            }
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

// ---- items ----------------------------------------------------------------------
// Chunks of 32 particles, electrons first (a chunk holds one species).
__device__ __forceinline__ void f64_chunk(const F64Fast &p, const N3Geom &g, int k, int &start, int &cnt, int &sp) {
    sp = k < p.nce ? 0 : 1;
    start = sp ? g.nel + (k - p.nce) * 32 : k * 32;
    cnt = min(32, (sp ? g.n : g.nel) - start);
}

// Item -> (chunk a, group of j-chunks, part of the rotation).  Rows come in
// blocks of `group` chunks: the rows of block A hold the groups A .. ng-1, so
// block A starts at group (A ng - A (A - 1)/2).
__device__ __forceinline__ void f64_item(const F64Fast &p, long long it, int &a, int &grp, int &part) {
    part = (int)(it % p.split);
    const long long t = it / p.split;
    auto start = [&](int A) { return (long long)p.group * ((long long)A * p.ng - (long long)A * (A - 1) / 2); };
    const float b = (float)p.ng + 0.5f;
    int A = (int)(b - sqrtf(fmaxf(b * b - 2.0f * (float)t / (float)p.group, 0.0f)));
    A = max(0, min(A, p.ng - 1));
    while (A > 0 && start(A) > t) --A;
    while (A + 1 < p.ng && start(A + 1) <= t) ++A;
    const int o = (int)(t - start(A)), w = p.ng - A;
    a = A * p.group + o / w;
    grp = A + o % w;
}

// One tile: the warp's 32 i-particles against chunk b, rotation steps [s0, s1).
template <int KIND, bool ENERGY, bool MASKED, bool RDF, bool CUBIC>
__device__ __forceinline__ void f64_tile(const F64Fast &p, const N3Args &a, const F64Shared &sh, int pt, bool diag,
                                         int icnt, long long xi0, long long xi1, long long xi2, int jstart, int jcnt,
                                         int s0, int s1, double (&fi)[3], double &pe) {
    const int lane = threadIdx.x & 31, src = (lane + 1) & 31;
    const int j0 = (lane + s0) & 31;
    const longlong4_32a t = a.xl[jstart + min(j0, jcnt - 1)];
    long long xj0 = t.x, xj1 = t.y, xj2 = t.z;
    double jx = 0.0, jy = 0.0, jz = 0.0;
#pragma unroll 1
    for (int s = s0; s < s1; ++s) {
        const long long d0 = (long long)((unsigned long long)xi0 - (unsigned long long)xj0);
        const long long d1 = (long long)((unsigned long long)xi1 - (unsigned long long)xj1);
        const long long d2 = (long long)((unsigned long long)xi2 - (unsigned long long)xj2);
        bool small = false;
        double dx = box_diff(d0, small), dy = box_diff(d1, small), dz = box_diff(d2, small);
        if (__any_sync(0xffffffffu, small)) {   // a component below 2^-32 of the box, zero among them
            constexpr double k = 5.421010862427522e-20;   // 2^-64
            dx = (double)d0 * k;
            dy = (double)d1 * k;
            dz = (double)d2 * k;
        }
        if (!CUBIC) {
            dx *= a.c.box[0];
            dy *= a.c.box[1];
            dz *= a.c.box[2];
        }
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        // 0 < r2 < rc^2 on the bit patterns (r2 >= 0: they order as the values)
        const long long rb = __double_as_longlong(r2);
        bool ok = rb > 0 && rb < __double_as_longlong(p.rc2);
        if (MASKED) {   // diagonal tiles: lane l with l + s, s = 1 .. 16, meets every pair once
            ok = ok && lane < icnt && ((lane + s) & 31) < jcnt;
            if (diag) ok = ok && s >= 1 && (s < 16 || (s == 16 && lane < 16));
        }
        if (RDF) rdf_add_f64(p, a.c, r2, ok, pt, sh.hist);
        const double w = n3_pair_f64<KIND, ENERGY>(p, a.c, r2, ok, pe, sh);
        fi[0] = fma(w, dx, fi[0]);
        fi[1] = fma(w, dy, fi[1]);
        fi[2] = fma(w, dz, fi[2]);
        jx = fma(w, dx, jx);
        jy = fma(w, dy, jy);
        jz = fma(w, dz, jz);
        xj0 = __shfl_sync(0xffffffffu, xj0, src);
        xj1 = __shfl_sync(0xffffffffu, xj1, src);
        xj2 = __shfl_sync(0xffffffffu, xj2, src);
        jx = __shfl_sync(0xffffffffu, jx, src);
        jy = __shfl_sync(0xffffffffu, jy, src);
        jz = __shfl_sync(0xffffffffu, jz, src);
    }
    const int jl = (lane + s1) & 31;   // the particle whose reaction this lane holds now
    if (jl < jcnt) {
        const double q = -p.qf[pt];
        double *f = a.facc + jstart + jl;
        atomicAdd(f, q * jx);
        atomicAdd(f + a.ntot, q * jy);
        atomicAdd(f + 2 * (size_t)a.ntot, q * jz);
    }
}

template <int EI, bool ENERGY, bool RDF, bool CUBIC>
__global__ void __launch_bounds__(kF64Threads, 1) pair_n3_f64_kernel(const N3Args a, const F64Fast p) {
    extern __shared__ __align__(128) uint4 tabs[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ double red[32];
    __shared__ unsigned hist[RDF ? 3 * kNbin : 1];
    __shared__ F64Tab tab;
    const int tid = threadIdx.x, lane = tid & 31;
    if (RDF)
        for (int k = tid; k < 3 * kNbin; k += kF64Threads) hist[k] = 0u;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        if (!(a.inject_skip && blockIdx.x == 0)) {        // test hook: the copy never comes
            const uint32_t b0 = (uint32_t)p.ew_seg * kEwVec * 16u, b1 = (uint32_t)p.ei_seg * kEiVec * 16u;
            mbar_arrive_expect_tx(&bar, b0 + b1);
            bulk_g2s(tabs, p.tab, b0, &bar);
            if (b1) bulk_g2s(tabs + p.ew_seg * kEwVec, p.tab + p.ew_seg * kEwVec, b1, &bar);
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
    sh.ei = tabs + p.ew_seg * kEwVec;
    sh.tb = &tab;
    sh.hist = nullptr;
    double etot = 0.0;
    for (;;) {
        unsigned nx = 0;
        if (lane == 0) nx = atomicAdd(a.counter, 1u);
        const long long it = __shfl_sync(0xffffffffu, nx, 0);
        if (it >= p.total) break;
        int ca, grp, part, istart, icnt, isp;
        f64_item(p, it, ca, grp, part);
        if (ca >= p.nc) continue;                         // the last block of rows may be short
        f64_chunk(p, a.g, ca, istart, icnt, isp);
        const int s0 = part * 32 / p.split, s1 = (part + 1) * 32 / p.split;
        const longlong4_32a t = a.xl[istart + min(lane, icnt - 1)];
        double fi[3] = {0.0, 0.0, 0.0};
        const int b1 = min(p.nc, (grp + 1) * p.group);
        for (int b = max(ca, grp * p.group); b < b1; ++b) {
            int jstart, jcnt, jsp;
            f64_chunk(p, a.g, b, jstart, jcnt, jsp);
            const int pt = isp + jsp;
            const bool diag = b == ca, masked = diag || icnt < 32 || jcnt < 32;
            double pe = 0.0, ft[3] = {0.0, 0.0, 0.0};
            if (RDF) sh.hist = hist + pt * kNbin;
#define TCP_F64_TILE(KIND, MASKED) \
    f64_tile<KIND, ENERGY, MASKED, RDF, CUBIC>(p, a, sh, pt, diag, icnt, t.x, t.y, t.z, jstart, jcnt, s0, s1, ft, pe)
            if (EI != 0 && pt == 1) {
                if (masked) TCP_F64_TILE(EI, true);
                else TCP_F64_TILE(EI, false);
            } else {
                if (masked) TCP_F64_TILE(0, true);
                else TCP_F64_TILE(0, false);
            }
#undef TCP_F64_TILE
            for (int k = 0; k < 3; ++k) fi[k] = fma(p.qf[pt], ft[k], fi[k]);
            if (ENERGY) etot = fma(p.qe[pt], pe, etot);
        }
        if (lane < icnt) {
            double *f = a.facc + istart + lane;
            atomicAdd(f, fi[0]);
            atomicAdd(f + a.ntot, fi[1]);
            atomicAdd(f + 2 * (size_t)a.ntot, fi[2]);
        }
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

// octaves of the Ewald table that the cut-off reaches
static int ewald_octaves(const tcp_ctx *c) {
    int top = kTabLow + 1;
    while (top < kEwTopMax && std::ldexp(1.0, top) < c->pc.alpha2 * c->rc2) ++top;
    return top - kTabLow;
}

static size_t f64_smem(int ew_seg, int ei_seg) { return 16 * ((size_t)ew_seg * kEwVec + (size_t)ei_seg * kEiVec); }

// Device tables of an FP64 context for its e-i model and cut-off (rebuilt with
// the pair constants, outside any stream capture).
int n3_f64_prepare(tcp_ctx *c) {
    const int oct = ewald_octaves(c), ew = oct << kEwBits;
    const std::vector<F64Vec> &full = table_of(TCP_EI_COULOMB);
    const int nfull = (int)(full.size() / kEwVec);
    std::vector<F64Vec> t;
    for (int v = 0; v < kEwVec; ++v) t.insert(t.end(), full.begin() + (size_t)v * nfull, full.begin() + (size_t)v * nfull + ew);
    int ei = 0;
    if (c->p.ei_model != TCP_EI_COULOMB) {
        const std::vector<F64Vec> &m = table_of(c->p.ei_model);
        ei = (int)(m.size() / kEiVec);
        t.insert(t.end(), m.begin(), m.end());
    }
    cudaFree(c->f64tab);
    c->f64tab = nullptr;
    TCP_CUDA(cudaMalloc(&c->f64tab, sizeof(F64Vec) * t.size()));
    TCP_CUDA(cudaMemcpy(c->f64tab, t.data(), sizeof(F64Vec) * t.size(), cudaMemcpyHostToDevice));
    c->f64_ew_seg = ew;
    c->f64_ei_seg = ei;
    for (int k = 0; k < 4; ++k)
        TCP_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void *>(f64_kernel(c, k & 1, (k & 2) != 0)),
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f64_smem(ew, ei)));
    return TCP_OK;
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
    const PairConsts &pc = c->pc;
    const double L = pc.cubic ? pc.box[0] : 1.0, l = c->p.ei_model == TCP_EI_DEUTSCH ? pc.rs : pc.lambda;
    const double al = pc.alpha, a3 = al * al * al;
    F64Fast p;
    std::memset(&p, 0, sizeof p);
    p.tab = reinterpret_cast<const uint4 *>(c->f64tab);
    p.ew_seg = c->f64_ew_seg;
    p.ei_seg = c->f64_ei_seg;
    p.ew_hi = kTabLowBits + ((unsigned)(p.ew_seg >> kEwBits) << 23);
    p.ei_hi = kTabLowBits + ((unsigned)(p.ei_seg >> kEiBits) << 23);
    p.kx = pc.alpha2 * (L * L);
    p.kxf = (float)p.kx;
    p.to_a2 = L * L;
    // the smallest r^2 whose rounded product with to_a2 reaches rc^2, so that
    // the cut-off test equals the one in A^2 to the last bit (rc = L/2 and
    // lattice positions put pairs exactly on it)
    p.rc2 = pc.rc2 / p.to_a2;
    while (p.rc2 * p.to_a2 < pc.rc2) p.rc2 = std::nextafter(p.rc2, HUGE_VAL);
    for (double t; (t = std::nextafter(p.rc2, 0.0)) * p.to_a2 >= pc.rc2;) p.rc2 = t;
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
    // Items of four tiles once there are enough of them that the last ones,
    // about 0.3 ms each, are a small part of the launch; single tiles below,
    // and halves or quarters of a tile's rotation where even those are too few
    // to fill the SM quarters evenly.
    p.nce = (c->nel + 31) / 32;
    p.nc = p.nce + (c->nion + 31) / 32;
    const long long tiles = (long long)p.nc * (p.nc + 1) / 2, quarters = 4LL * c->num_sms;
    p.group = tiles >= 512 * quarters ? 4 : 1;
    p.split = tiles >= 16 * quarters ? 1 : (tiles >= 8 * quarters ? 2 : 4);
    p.ng = (p.nc + p.group - 1) / p.group;
    p.total = (long long)p.group * p.ng * (p.ng + 1) / 2 * p.split;
    const int grid = (int)std::min<long long>(n3_f64_grid(c), (p.total + kF64Warps - 1) / kF64Warps);
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
