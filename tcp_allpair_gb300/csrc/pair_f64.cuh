// pair_f64.cuh -- what the FP64 tile kernels share (the real-space sum,
// pair_n3_f64.cu, and its derivatives, adjoint.cu): the radial tables and their
// evaluation, the conversions that stay off the FP64 pipe, and the items.  The
// reasons stand in pair_n3_f64.cu.
#pragma once

#include "device_util.cuh"
#include "pair_n3.cuh"

#include <vector>

namespace tcp {

// Three warps per SM quarter hide the latency of the FP32 and integer work.  The
// tables take 64 to 210 KB of shared memory: one CTA per SM, and no room for
// the plane kernels of a reciprocal chain beside it, which run before or after.
constexpr int kF64Threads = 384;
constexpr int kF64Warps = kF64Threads / 32;

// ---- tables ---------------------------------------------------------------------
// Segments of the argument, a power of two of them per octave (the leading
// mantissa bits select one).  Per segment and function the Taylor coefficients
// c0..c3 (Ewald) or c0..c4 (e-i) in FP64 and the four next ones in FP32, in
// 16-byte vectors [vector][segment] so that lanes on different segments use
// different banks.  A table holds several functions:
//   Ewald   c0 c1 | c2 c3 | t4 .. t7           per function
//   e-i     c0 c1 | c2 c3 | c4 t5 t6           per function, then t7 t8 of two functions per vector
//
// Where the functions fall as e^{-x} the terms do so with the segment's width,
// not with its width over x: the octaves from there on have more segments, so
// that the FP32 terms stay below 2^-24 of the sum.  Largest relative errors of
// all the functions (100 to 150 random arguments an octave, against 45 digits),
// and with the first octave's number of segments in every octave:
//   Ewald    x < 4 3e-16, < 8 5e-16, < 16 4e-16 (1.5e-14), < 32 5e-15 (3e-13)
//   Kelbg    y < 4 1.5e-15, < 16 1.1e-15 (2.7e-13), < 32 9e-16 (3e-11), < 64 6e-14 (1e-8)
//   Deutsch  s < 8 5e-15, < 23 1.1e-15 (4e-13), < 32 3e-12, < 45 3e-11
// An argument rounded to FP64 alone makes them uncertain by x 2^-53.  The last
// octaves are coarser than that, for shared memory: there the functions are
// below e^{-32} (Kelbg) and e^{-22} (Deutsch), so that a pair's force and
// energy do not feel it; the derivatives with respect to lambda of a system
// with no nearer e-i pair do.
constexpr int kEwLow = -6, kEwMid = 3, kEwTop = 5;   // 2^kEwBits segments an octave, twice that from 2^kEwMid on
constexpr int kEwBits = 7;
constexpr unsigned kEwLowBits = (127 + kEwLow) << 23, kEwMidBits = (127 + kEwMid) << 23;
constexpr int kEiLow = -1, kEiOct = 12;              // octaves of the longer one; F64Fast::ei_oct
constexpr unsigned kEiLowBits = (127 + kEiLow) << 23;
__host__ __device__ constexpr int ew_vec(int nf) { return 3 * nf; }
__host__ __device__ constexpr int ei_vec(int nf) { return 3 * nf + (nf + 1) / 2; }
// Below the tables, and past the end of the Ewald one (a^2 r^2 = 32), the
// general form takes the pair.  The e-i functions are 0 from the end of theirs
// on: e^{-64} = 1.6e-28 (Kelbg), e^{-45} = 2.6e-20 (Deutsch) of the Coulomb term.

// The functions.  Ewald (x = a^2 r^2): the Taylor families of B_n, B_0 =
// erfc(sqrt x)/sqrt x; Deutsch (z = r^2/rs^2): A_n, A_0 = e^{-s}/s, s = sqrt z;
// Kelbg (y = r^2/lambda^2).
enum F64Func {
    kFuncU,      // energy: B_0, A_0, sqrt(pi) erfc(sqrt y) - e^{-y} y^{-1/2}
    kFuncF,      // force weight: B_1, A_1, e^{-y} y^{-3/2}
    kFuncG2,     // -2 dF/d(argument): B_2, A_2
    kFuncGl,     // lambda derivative of the force weight: A_0, e^{-y} y^{-1/2}
    kFuncDl      // lambda derivative of the energy: e^{-s}, erfc(sqrt y)
};

// Host side (pair_n3_f64.cu): the vectors of one table for the functions
// given, the first `segments` of it (0: all); *nseg: its segments.
struct F64Vec {
    union {
        double d[2];
        float f[4];
    };
};
std::vector<F64Vec> f64_table(int model, const int *funcs, int nf, int segments, int *nseg);
double f64_segment_end(int model, int k);   // upper end of segment k
int ewald_segments(const tcp_ctx *c);       // segments of the Ewald table that the cut-off reaches

// What the kernel needs besides PairConsts.  Lengths in units of the box where
// it is cubic (the fixed-point differences unscaled), in A otherwise.
struct F64Fast {
    const uint4 *tab;        // Ewald vectors, then e-i vectors
    int ew_seg, ei_seg;      // segments per vector
    unsigned ew_hi, ei_hi;   // float bits of the table ends
    int ei_oct[kEiOct];      // per octave of the e-i table: shift of the segment's bits | 32 x offset
    double kx, ky;           // r^2 -> a^2 r^2, r^2/lambda^2 (or /rs^2)
    float kxf, kyf;
    double rc2;              // cut-off^2 (r^2 < rc2)
    float boxf[3], near2;    // 2^-32 of the box; a bound of rc2 for the FP32 test of f64_mask
    double to_a2;            // r^2 -> A^2 (the general form)
    double cf, cu;           // weight and energy of the e-i term in units of the Ewald term's a^3 and a
    double ia3, ia;          // 1/a^3, 1/a
    double qf[3], qe[3];     // force factor (eV/A per unit weight and separation) and energy factor per pair type
    float rinv_dx[3];        // RDF: sqrt(r^2) -> r/dx
    int group, split;        // j-chunks per item; items per tile
    int nce, nc, nd;         // electron chunks, chunks, distances in their ring (f64_ring)
    long long items;
};

F64Fast f64_args(const tcp_ctx *c, int ew_seg, int ei_seg);   // tab: the caller's
float f64_near2(const PairConsts &pc, double r);   // F64Fast::near2 for a distance r (units of F64Fast)

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

// the same for either sign
__device__ __forceinline__ float narrow_signed(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), mag = hi & 0x7fffffffu;
    const unsigned b = __funnelshift_l((unsigned)__double2loint(x), mag, 3) + 0x40000000u;
    return __uint_as_float((mag < 0x38100000u ? 0u : b) | (hi & 0x80000000u));
}

// Where an argument lies in a table: vector offset of its segment, distance h
// to the centre in FP64, and in FP32 from that (a difference in FP32 would be
// off by 2^-23 x).  xb: the bits of the FP32 argument; sh, base: the segment is
// (xb >> sh) + base.
struct F64At {
    const uint4 *t;
    double h;
    float hf;
};
__device__ __forceinline__ F64At f64_at(const uint4 *tab, unsigned xi, int sh, int base, double r2, double k) {
    const unsigned q = xi >> sh;
    F64At a;
    a.t = tab + ((int)q + base);
    a.h = fma(r2, k, -widen(__uint_as_float((2u * q + 1u) << (sh - 1))));
    a.hf = narrow_signed(a.h);
    return a;
}
__device__ __forceinline__ F64At ew_at(const uint4 *tab, unsigned xb, unsigned hi, double r2, double k) {
    constexpr int SH = 23 - kEwBits, MID = (kEwMid - kEwLow) << kEwBits;
    const unsigned xi = min(max(xb, kEwLowBits), hi - 1u);
    const bool low = xi < kEwMidBits;
    return f64_at(tab, xi, low ? SH : SH - 1, low ? -(int)(kEwLowBits >> SH) : MID - (int)(kEwMidBits >> (SH - 1)), r2, k);
}
__device__ __forceinline__ F64At ei_at(const uint4 *tab, const int *oct, unsigned yb, unsigned hi, double r2, double k) {
    const unsigned yi = min(max(yb, kEiLowBits), hi - 1u);
    const int o = oct[(yi - kEiLowBits) >> 23];
    return f64_at(tab, yi, o & 31, o >> 5, r2, k);
}

// function f of an Ewald table of n segments
__device__ __forceinline__ double ew_poly(const F64At &a, int n, int f) {
    const double2 c01 = lds2(a.t + 3 * f * n), c23 = lds2(a.t + (3 * f + 1) * n);
    const float4 t4 = lds4(a.t + (3 * f + 2) * n);
    const double w = fma(a.h, widen(fmaf(fmaf(fmaf(t4.w, a.hf, t4.z), a.hf, t4.y), a.hf, t4.x)), c23.y);
    return fma(a.h, fma(a.h, fma(a.h, w, c23.x), c01.y), c01.x);
}

// function f of nf of an e-i table of n segments; NEG: its FP32 part T is
// negative (k = 5 of a completely monotone function; the Kelbg energy's is
// positive, U' = F/2)
template <bool NEG>
__device__ __forceinline__ double ei_poly(const F64At &a, int n, int f, int nf) {
    const double2 c01 = lds2(a.t + 3 * f * n), c23 = lds2(a.t + (3 * f + 1) * n), c4 = lds2(a.t + (3 * f + 2) * n);
    const float2 t78 = reinterpret_cast<const float2 *>(a.t + (3 * nf + f / 2) * n)[f & 1];
    const float t5 = __int_as_float(__double2loint(c4.y)), t6 = __int_as_float(__double2hiint(c4.y));
    const float t = fmaf(fmaf(fmaf(t78.y, a.hf, t78.x), a.hf, t6), a.hf, t5);
    const double v = NEG ? fma(-a.h, widen(-t), c4.x) : fma(a.h, widen(t), c4.x);
    return fma(a.h, fma(a.h, fma(a.h, fma(a.h, v, c23.y), c23.x), c01.y), c01.x);
}

// ---- items ----------------------------------------------------------------------
// Chunks of 32 particles, electrons first (a chunk holds one species).
__device__ __forceinline__ void f64_chunk(const F64Fast &p, const N3Geom &g, int k, int &start, int &cnt, int &sp) {
    sp = k < p.nce ? 0 : 1;
    start = sp ? g.nel + (k - p.nce) * 32 : k * 32;
    cnt = min(32, (sp ? g.n : g.nel) - start);
}

// The chunks form a ring: chunk a meets the chunks a, a + 1, .., a + nc/2
// behind it, at the distance nc/2 of an even ring in its first half only, so
// that every pair of chunks meets once.  Item -> (a, first distance d0 of up to
// `group`, their number nd, part).  Items that run at the same time lie on
// different i- and j-chunks: in rows of the triangle they added to the same 32
// particles, whose atomics (0.8 ns each on one address) then set the time
// (N = 24,000: 10.3 ms against the 5.7 of the FP64 operations).
__device__ __forceinline__ void f64_ring(const F64Fast &p, long long it, int &a, int &d0, int &nd, int &part) {
    const unsigned u = (unsigned)it, r = (unsigned)(p.nc * p.split), k = u / r, q = u - k * r;
    part = (int)(q / (unsigned)p.nc);
    a = (int)(q - (unsigned)part * (unsigned)p.nc);
    d0 = (int)k * p.group;
    nd = min(p.group, p.nd - d0);
    if (2 * (d0 + nd - 1) == p.nc && 2 * a >= p.nc) --nd;
}

// The next run of an item: up to kMaskChunks chunks of one species among its
// distances [d, end); false after the last.
constexpr int kMaskChunks = 4;
struct F64Run {
    int d, end;
    int pt, j0, nj;          // pair type, particles
    bool diag;               // starts with the i-particles' own chunk
};
__device__ __forceinline__ bool f64_run(const F64Fast &p, const N3Geom &g, int a, int isp, F64Run &r) {
    if (r.d >= r.end) return false;
    const int b = a + r.d < p.nc ? a + r.d : a + r.d - p.nc, jsp = b < p.nce ? 0 : 1;
    const int run = min(min(r.end - r.d, (jsp ? p.nc : p.nce) - b), kMaskChunks);
    r.pt = isp + jsp;
    r.j0 = jsp ? g.nel + (b - p.nce) * 32 : b * 32;
    r.nj = min(run * 32, (jsp ? g.n : g.nel) - r.j0);
    r.diag = r.d == 0;
    r.d += run;
    return true;
}

// ---- near pairs ---------------------------------------------------------------------
// Half of all pairs lie past rc = L/2, and a warp instruction on the FP64 pipe
// takes as long whether its lanes need it or not.  So a warp first finds the
// pairs inside rc with FP32 arithmetic (12 issue slots a step of the 64 that
// one FP64 operation takes) as a bit mask per lane, and evaluates those alone.
struct F64Pos {
    long long x, y, z;       // 64-bit fixed point
};
struct F64Mask {
    unsigned long long lo, hi;   // j-particles 0 .. 127 of a lane's i-particle
};

__device__ __forceinline__ long long f64_sub(long long a, long long b) {
    return (long long)((unsigned long long)a - (unsigned long long)b);
}

// minimum-image separation of two particles in units of the box (A where it is not cubic)
template <bool CUBIC>
__device__ __forceinline__ void f64_separation(const PairConsts &c, const F64Pos &xi, const longlong4_32a &xj,
                                               double (&u)[3]) {
    const long long d[3] = {f64_sub(xi.x, xj.x), f64_sub(xi.y, xj.y), f64_sub(xi.z, xj.z)};
    bool small = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = box_diff(d[k], small);
    if (__any_sync(0xffffffffu, small))   // a component below 2^-32 of the box, zero among them
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = (double)d[k] * 5.421010862427522e-20;   // 2^-64
    if (!CUBIC)
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] *= c.box[k];
}

// The pairs of the lane's i-particle with the nj (up to 128) j-particles from
// j0 on that may lie inside rc, those of part `part` of every chunk; diag: the
// first chunk is the i-particles' own (each pair once).
__device__ __forceinline__ F64Mask f64_mask(const F64Fast &p, const longlong4_32a *xl, const F64Pos &xi, bool live,
                                            int j0, int nj, bool diag, int part) {
    const int lane = threadIdx.x & 31;
    const int s0 = part * 32 / p.split, s1 = (part + 1) * 32 / p.split;
    const int xh = (int)(xi.x >> 32), yh = (int)(xi.y >> 32), zh = (int)(xi.z >> 32);
    F64Mask m{0ull, 0ull};
    for (int c = 0; c * 32 < nj; ++c) {
        const longlong4_32a t = xl[j0 + min(c * 32 + lane, nj - 1)];
        const int jx = (int)(t.x >> 32), jy = (int)(t.y >> 32), jz = (int)(t.z >> 32);
        unsigned w = 0u;
#pragma unroll 4
        for (int s = s0; s < s1; ++s) {
            const float dx = (float)(int)((unsigned)xh - (unsigned)__shfl_sync(0xffffffffu, jx, s)) * p.boxf[0];
            const float dy = (float)(int)((unsigned)yh - (unsigned)__shfl_sync(0xffffffffu, jy, s)) * p.boxf[1];
            const float dz = (float)(int)((unsigned)zh - (unsigned)__shfl_sync(0xffffffffu, jz, s)) * p.boxf[2];
            if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < p.near2) w |= 1u << s;
        }
        if (nj - c * 32 < 32) w &= (1u << (nj - c * 32)) - 1u;
        if (diag && c == 0) w &= 0xfffffffeu << lane;
        if (!live) w = 0u;
        if (c < 2)
            m.lo |= (unsigned long long)w << (32 * c);
        else
            m.hi |= (unsigned long long)w << (32 * c - 64);
    }
    return m;
}

// the first j-particle of a mask that is not empty, taken out of it
__device__ __forceinline__ int mask_pop(F64Mask &m) {
    if (m.lo) {
        const int j = __ffsll((long long)m.lo) - 1;
        m.lo &= m.lo - 1;
        return j;
    }
    const int j = __ffsll((long long)m.hi) + 63;
    m.hi &= m.hi - 1;
    return j;
}

// The pairs left in the warp's masks, numbered lane by lane: total, and per
// lane those up to and including its own.
struct F64Deal {
    int total, upto, own;
};
__device__ __forceinline__ F64Deal mask_deal(const F64Mask &m) {
    F64Deal d;
    d.own = __popcll(m.lo) + __popcll(m.hi);
    d.upto = d.own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, d.upto, o);
        if ((int)(threadIdx.x & 31) >= o) d.upto += v;
    }
    d.total = __shfl_sync(0xffffffffu, d.upto, 31);
    return d;
}

// pair t0 + lane of them: the lane whose it is and its bit there; pair 0 where
// there is none
struct F64Dealt {
    int lane, bit;
    bool live;
};
__device__ __forceinline__ F64Dealt mask_dealt(const F64Mask &m, const F64Deal &d, int t0) {
    F64Dealt r;
    int t = t0 + (int)(threadIdx.x & 31);
    r.live = t < d.total;
    t = r.live ? t : 0;
    r.lane = 0;
#pragma unroll
    for (int b = 16; b; b >>= 1)
        if (__shfl_sync(0xffffffffu, d.upto, r.lane + b - 1) <= t) r.lane += b;
    t -= __shfl_sync(0xffffffffu, d.upto - d.own, r.lane);
    const unsigned long long lo = __shfl_sync(0xffffffffu, m.lo, r.lane), hi = __shfl_sync(0xffffffffu, m.hi, r.lane);
    // bit t of the 128: the half, the word and then the place in it
    const int nl = __popcll(lo);
    unsigned long long v = t < nl ? lo : hi;
    r.bit = t < nl ? 0 : 64;
    t -= t < nl ? 0 : nl;
#pragma unroll
    for (int b = 32; b; b >>= 1) {
        const int c = __popcll(v & ((1ull << b) - 1ull));
        if (t >= c) {
            t -= c;
            v >>= b;
            r.bit += b;
        }
    }
    return r;
}

__device__ __forceinline__ void add_force(double *f, size_t n, double x, double y, double z) {
    atomicAdd(f, x);
    atomicAdd(f + n, y);
    atomicAdd(f + 2 * n, z);
}

}  // namespace tcp
