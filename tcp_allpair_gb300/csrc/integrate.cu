// integrate.cu -- velocity Verlet halves and thermostats (vverlet.f90),
// net-force removal (REMOVE_RIGIDMTN, force.f90:974-1007), the SPME_SUM add,
// deterministic FP64 reductions, and the host-record gather/scatter kernels.
//
// All state is FP64 SoA [3][n].  Every kernel that moves positions also
// refreshes the two pair-kernel copies: 32-bit fixed point (int4) and
// double4_32a.  Reductions write one partial per CTA; the last CTA of the same
// launch sums them in a fixed order, so results do not depend on scheduling.
#include <cmath>

#include "device_util.cuh"
#include "spme_chain.cuh"
#include "tcp_internal.h"

namespace tcp {

constexpr int kIntThreads = 256;

// GB300's FP64 pipe runs at 1/64 of the FP32 rate and an FP64 division is a
// chain of about ten FP64 operations, so the per-particle kernels divide by
// the box length through its reciprocal (iL = 1/L, set on the host) and by
// the mass through dt/(2m) computed once per thread.

struct IntArgs {
    double *x, *v, *f;
    int4 *xq;
    double4_32a *xd;
    longlong4_32a *xl;
    int copies;              // pair-kernel copies to refresh: kCopyXq | kCopyXd | kCopyXl
    int nel, n;
    double xm0, xm1;
    double L0, L1, L2;
    double iL0, iL1, iL2;    // 1/L
};

// The copies a context's kernels read: the FP32C kernels the 32-bit fixed
// point, the FP64 kernels the doubles (ordered-pair and derivative kernels) and
// the 64-bit fixed point (Newton-3 kernels).
enum { kCopyXq = 1, kCopyXd = 2, kCopyXl = 4 };

__device__ __forceinline__ void store_pos(const IntArgs &a, int i, double x0, double x1, double x2) {
    a.x[i] = x0;
    a.x[(size_t)a.n + i] = x1;
    a.x[2 * (size_t)a.n + i] = x2;
    if (a.copies & kCopyXq)
        a.xq[i] = make_int4(fixed_coord(x0, a.iL0), fixed_coord(x1, a.iL1), fixed_coord(x2, a.iL2), 0);
    if (a.copies & kCopyXd) a.xd[i] = make_double4_32a(x0, x1, x2, 0.0);
    if (a.copies & kCopyXl) {
        longlong4_32a q;
        q.x = fixed_coord64(x0, a.iL0);
        q.y = fixed_coord64(x1, a.iL1);
        q.z = fixed_coord64(x2, a.iL2);
        q.w = 0;
        a.xl[i] = q;
    }
}

__device__ __forceinline__ double wrap(double x, double L, double iL) { return wrap_box(x, L, iL); }


// Finit's step back / forward, init.f90:171-185 and 223-237
__global__ void shift_kernel(const IntArgs a, double sdt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double y[3];
    const double L[3] = {a.L0, a.L1, a.L2}, iL[3] = {a.iL0, a.iL1, a.iL2};
    for (int k = 0; k < 3; ++k) y[k] = wrap(a.x[(size_t)k * a.n + i] + sdt * a.v[(size_t)k * a.n + i], L[k], iL[k]);
    store_pos(a, i, y[0], y[1], y[2]);
}

// component d of particle i
__device__ __forceinline__ void store_comp(const IntArgs &a, int d, int i, double x, double iL) {
    a.x[(size_t)d * a.n + i] = x;
    if (a.copies & kCopyXq) reinterpret_cast<int *>(a.xq + i)[d] = fixed_coord(x, iL);
    if (a.copies & kCopyXd) reinterpret_cast<double *>(a.xd + i)[d] = x;
    if (a.copies & kCopyXl) reinterpret_cast<long long *>(a.xl + i)[d] = fixed_coord64(x, iL);
}

__global__ void refresh_kernel(const IntArgs a, const double *__restrict__ x) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * a.n) return;
    const int d = t / a.n;
    store_comp(a, d, t - d * a.n, x[t], d == 0 ? a.iL0 : (d == 1 ? a.iL1 : a.iL2));
}

// What the half kick of a step does besides: the accumulators of the pair
// launch and the bins of the SPME chain (their own launches otherwise).
struct StepPrep {
    double *fpart;           // [3][n], cleared; null: not this kernel's job
    double *upart;
    int nupart;
    unsigned *counter;
    int bin;                 // bin the positions for the chain
    ChainArgs chain;
};

// VVerletNotemp1 (vverlet.f90:148-167) / VVerletStoch1 (vverlet.f90:34-55).
// A thread per component: the FP64 chain of a particle (its three components
// one after the other took 45 dependent operations of 34 ns) is a third as
// long and a small system spreads over three times the warps.
// Without KICK the preparation alone (the autotuner's replays).
template <bool BIN, bool KICK>
__global__ void __launch_bounds__(kPartThreads) vverlet1_kernel(const IntArgs a, double dt, double hdm0, double hdm1,
                                                                double alpha_lgv, int stoch, const StepPrep s) {
    __shared__ int sb[BIN ? 3 : 1][kPartBlock];
    __shared__ double sa[BIN ? 3 : 1][kPartBlock];
    const int k = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, i = blockIdx.x * kPartBlock + k;
    const bool live = i < a.n;
    if (live) {
        const double L = d == 0 ? a.L0 : (d == 1 ? a.L1 : a.L2), iL = d == 0 ? a.iL0 : (d == 1 ? a.iL1 : a.iL2);
        const size_t o = (size_t)d * a.n + i;
        double y = a.x[o];
        if (KICK) {
            const double hdm = i < a.nel ? hdm0 : hdm1;    // dt/(2m), divided on the host
            double v = a.v[o];
            if (stoch)
                v = v * (1.0 - alpha_lgv * hdm) + hdm * a.f[o];   // vverlet.f90:37-38
            else
                v = v + hdm * a.f[o];                      // vverlet.f90:151
            a.v[o] = v;
            y = wrap_fast(y + dt * v, L, iL);              // vverlet.f90:152-153
            store_comp(a, d, i, y, iL);
        }
        if (s.fpart) s.fpart[o] = 0.0;
        if (BIN) {
            const SpmeGeom &g = s.chain.one;
            sb[d][k] = bin_axis(y, g.hL[d], g.KL[d], g.K[d], s.chain.P, sa[d][k]);
        }
    }
    const int t = blockIdx.x * kPartThreads + threadIdx.x;
    if (s.fpart) {
        for (int u = t; u < s.nupart; u += gridDim.x * kPartThreads) s.upart[u] = 0.0;
        if (t == 0) *s.counter = 0u;
    }
    if (BIN) {
        __syncthreads();
        if (live && d == 0) {
            const ChainArgs &c = s.chain;
            const double arg[3] = {sa[0][k], sa[1][k], sa[2][k]}, q = i < a.nel ? c.one.q[0] : c.one.q[1];
            if (c.fp64)
                bin_store<double>(c.b, i, a.n, arg, q, sb[0][k], sb[1][k], sb[2][k], c.one.K[1], 0);
            else
                bin_store<float>(c.b, i, a.n, arg, q, sb[0][k], sb[1][k], sb[2][k], c.one.K[1], 0);
        }
        if (s.chain.nbins <= kScanTail && last_block(s.chain.ticket)) scan_bins(s.chain.b, s.chain.nbins);
    }
}

// ---- Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) ---------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
        const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
        ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
        key.x += W0;
        key.y += W1;
    }
    return ctr;
}

// Three standard normals for (particle, step): Box-Muller on the words of
// two Philox blocks (counter = {particle, step lo, step hi, 0|1}).
__device__ __forceinline__ void gauss3(uint64_t seed, long long step, int i, double g[3]) {
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    const uint4 r0 = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)step, (uint32_t)((uint64_t)step >> 32), 0u), key);
    const uint4 r1 = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)step, (uint32_t)((uint64_t)step >> 32), 1u), key);
    const double s = 2.3283064365386963e-10;  // 2^-32
    const double u1 = ((double)r0.x + 0.5) * s, u2 = ((double)r0.y + 0.5) * s;
    const double u3 = ((double)r1.x + 0.5) * s, u4 = ((double)r1.y + 0.5) * s;
    const double ra = sqrt(-2.0 * log(u1)), rb = sqrt(-2.0 * log(u3));
    g[0] = ra * cos(2.0 * kPi * u2);
    g[1] = ra * sin(2.0 * kPi * u2);
    g[2] = rb * cos(2.0 * kPi * u4);
}

struct KickArgs {
    IntArgs a;
    double dt;
    double hdm0, hdm1;       // dt/(2m) per species (host-divided: the same correctly rounded value)
    int thermo;              // TCP_THERMO_*
    int remove_net;          // subtract sum(f)/n first (REMOVE_RIGIDMTN fused)
    double *mv_part;         // [2][nb] output partials (species)
    int vdf;
    unsigned long long *vdf_counts;
    double dv0, dv1;
    double T0, T1, tau, alpha_lgv;
    uint64_t seed;
    double *scal;            // kScal*: mean force in, sums of m v^2 in (rescale) and out, the step counter
    int last_pass;           // this pass ends the step's second half
    unsigned *ticket;
};

__device__ __forceinline__ void vdf_add(const KickArgs &k, int s, double mv2) {
    const double t = mv2 / 3.0 / (s == 0 ? k.dv0 : k.dv1);   // vverlet.f90:201
    if (t < (double)kNbin) atomicAdd(&k.vdf_counts[s * kNbin + (int)t], 1ull);
}

// Sum over a CTA of kPartThreads threads; valid in thread 0.
__device__ __forceinline__ double part_sum(double v, double *sh) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kPartThreads / 32; ++w) r += sh[w];
    __syncthreads();
    return r;
}

// The end of a kinetic pass: the CTA's sums of m v^2 per species, and in the
// last CTA the totals (in a fixed order) and the VDF of the final velocities.
__device__ __forceinline__ void kick_end(const KickArgs &k, double mv2, bool live, int s) {
    __shared__ double red[8];
    __shared__ double smv[3][kPartBlock];
    if (k.vdf) {
        const int p = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock;
        smv[d][p] = mv2;
        __syncthreads();
        if (d == 0 && live) vdf_add(k, s, smv[0][p] + smv[1][p] + smv[2][p]);
    }
    // one species per CTA but for the one where the ions begin
    const int nb = gridDim.x, i0 = blockIdx.x * kPartBlock;
    const bool mixed = i0 < k.a.nel && i0 + kPartBlock > k.a.nel;
    double te, ti;
    if (mixed) {
        te = part_sum(s == 0 ? mv2 : 0.0, red);
        ti = part_sum(s == 0 ? 0.0 : mv2, red);
    } else {
        te = part_sum(mv2, red);
        ti = 0.0;
        if (i0 >= k.a.nel) {
            ti = te;
            te = 0.0;
        }
    }
    if (threadIdx.x == 0) {
        k.mv_part[blockIdx.x] = te;
        k.mv_part[nb + blockIdx.x] = ti;
    }
    if (last_block(k.ticket)) {
        double e = 0.0, n = 0.0;
        for (int b = threadIdx.x; b < nb; b += kPartThreads) {
            e += __ldcg(k.mv_part + b);
            n += __ldcg(k.mv_part + nb + b);
        }
        e = part_sum(e, red);
        n = part_sum(n, red);
        if (threadIdx.x == 0) {
            k.scal[kScalMv2e] = e;
            k.scal[kScalMv2i] = n;
            if (k.last_pass) k.scal[kScalStep] += 1.0;   // one second half-kick per MD step
        }
    }
}

// Second half kick (vverlet.f90:194-219 NOTEMP, :250-255 BEREND/ISOKIN first
// loop, :91-123 STOCH), a thread per component; per-species sums of m v^2 and
// the VDF when no rescale follows.  The sums of the CTAs are added by the last
// one to finish (a launch of their own took 10 us, and 3 threads adding the
// force partials in every CTA as much again).
__global__ void __launch_bounds__(kPartThreads) kick2_kernel(const KickArgs k) {
    const IntArgs &a = k.a;
    const int p = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, i = blockIdx.x * kPartBlock + p;
    const bool live = i < a.n, stoch = k.thermo == TCP_THERMO_STOCH;
    const int s = i < a.nel ? 0 : 1;
    __shared__ double eta[3][kPartBlock];
    if (stoch) {
        if (live && d == 0) {
            double g[3];
            gauss3(k.seed, (long long)k.scal[kScalStep], i, g);
            for (int q = 0; q < 3; ++q) eta[q][p] = g[q];
        }
        __syncthreads();
    }
    double mv2 = 0.0;
    if (live) {
        const double xm = s == 0 ? a.xm0 : a.xm1;
        const double hdm = s == 0 ? k.hdm0 : k.hdm1;      // dt/(2m)
        const size_t o = (size_t)d * a.n + i;
        double fd = a.f[o], vv;
        if (k.remove_net) fd -= k.scal[kScalFx + d];                         // force.f90:999-1004
        if (stoch) {
            const double beta = sqrt(2.0 * k.alpha_lgv * (s == 0 ? k.T0 : k.T1) / k.dt);
            fd = fd + eta[d][p] * beta;                                      // vverlet.f90:95
            vv = (a.v[o] + hdm * fd) * (1.0 / (1.0 + k.alpha_lgv * hdm));    // vverlet.f90:96-97
        } else {
            vv = a.v[o] + hdm * fd;                                          // vverlet.f90:197
        }
        if (k.remove_net || stoch) a.f[o] = fd;
        a.v[o] = vv;
        mv2 = vv * vv * xm;                                                  // vverlet.f90:199
    }
    kick_end(k, mv2, live, s);
}

// Rescale pass of VVerletIsokin2 / VVerletBerend2 (vverlet.f90:331-344,
// 257-270): lambda per species from the first-pass sums, v *= lambda,
// sum m v^2 and VDF.
__global__ void __launch_bounds__(kPartThreads) rescale_kernel(const KickArgs k) {
    const IntArgs &a = k.a;
    const int p = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, i = blockIdx.x * kPartBlock + p;
    const bool live = i < a.n;
    const int s = i < a.nel ? 0 : 1;
    double mv2 = 0.0;
    if (live) {
        const int cnt = s == 0 ? a.nel : a.n - a.nel;
        const double T0 = k.scal[s == 0 ? kScalMv2e : kScalMv2i] / (double)(3 * cnt);
        const double T = s == 0 ? k.T0 : k.T1;
        const double lam = k.thermo == TCP_THERMO_ISOKIN ? sqrt(T / T0) : sqrt(1.0 + k.dt * (T / T0 - 1.0) / k.tau);
        const size_t o = (size_t)d * a.n + i;
        const double vv = a.v[o] * lam;
        a.v[o] = vv;
        mv2 = vv * vv * (s == 0 ? a.xm0 : a.xm1);
    }
    kick_end(k, mv2, live, s);
}

// The end of a pass over the forces: sum(f)/n into fbar by the last CTA, with
// the pair energy when upart is given.
__device__ __forceinline__ void force_end(double f, double *part, int n, double *scal, const double *upart, int nu,
                                          unsigned *ticket) {
    __shared__ double red[8];
    const int d = threadIdx.x / kPartBlock, w = threadIdx.x >> 5, nb = gridDim.x;
    f = warp_sum(f);
    if ((threadIdx.x & 31) == 0) red[w] = f;
    __syncthreads();
    if (threadIdx.x < 3) part[threadIdx.x * nb + blockIdx.x] = red[2 * threadIdx.x] + red[2 * threadIdx.x + 1];
    if (!last_block(ticket)) return;
    double s = 0.0;
    for (int b = threadIdx.x % kPartBlock; b < nb; b += kPartBlock) s += __ldcg(part + d * nb + b);
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[w] = s;
    __syncthreads();
    if (threadIdx.x < 3) scal[kScalFx + threadIdx.x] = (red[2 * threadIdx.x] + red[2 * threadIdx.x + 1]) / (double)n;
    if (upart) {
        __syncthreads();
        double u = 0.0;
        for (int k = threadIdx.x; k < nu; k += kPartThreads) u += upart[k];
        u = part_sum(u, red);
        if (threadIdx.x == 0) scal[kScalUr] = u;
    }
}

// f = sum over splits of fpart (+ frec: the SPME_SUM add of force.f90:953-964
// fused), the mean force for REMOVE_RIGIDMTN (force.f90:986-993) and the pair
// energy.  When a tile wait of the pair kernel ran out (status), some partials
// were never written: f is then left as it was and the caller reports the error.
__global__ void __launch_bounds__(kPartThreads) force_finalize_kernel(const double *__restrict__ fpart, int nsplit,
                                                                      const double *__restrict__ frec,
                                                                      double *__restrict__ f, int n,
                                                                      double *__restrict__ fsum_part,
                                                                      const unsigned *__restrict__ status,
                                                                      double *__restrict__ scal,
                                                                      const double *__restrict__ upart, int nu,
                                                                      unsigned *ticket) {
    const int k = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, i = blockIdx.x * kPartBlock + k;
    const bool write = !(*status & kStatusTmaTimeout);
    double acc = 0.0;
    if (i < n) {
        for (int sp = 0; sp < nsplit; ++sp) acc += fpart[((size_t)sp * 3 + d) * n + i];
        if (frec) acc += frec[(size_t)d * n + i];
        if (write) f[(size_t)d * n + i] = acc;
    }
    force_end(acc, fsum_part, n, scal, upart, nu, ticket);
}

// f += frec (SPME_SUM, force.f90:953-964; null: f as it is) and the mean force
__global__ void __launch_bounds__(kPartThreads) add_rec_kernel(double *__restrict__ f, const double *__restrict__ frec,
                                                               int n, double *__restrict__ fsum_part,
                                                               double *__restrict__ scal, unsigned *ticket) {
    const int k = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, i = blockIdx.x * kPartBlock + k;
    double v = 0.0;
    if (i < n) {
        const size_t o = (size_t)d * n + i;
        v = f[o];
        if (frec) {
            v += frec[o];
            f[o] = v;
        }
    }
    force_end(v, fsum_part, n, scal, nullptr, 0, ticket);
}

// f -= sum(f)/n (REMOVE_RIGIDMTN, force.f90:996-1004)
__global__ void remove_net_kernel(double *__restrict__ f, int n, const double *__restrict__ scal) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 3 * n) f[t] -= scal[kScalFx + t / n];
}

// ---- host records <-> SoA ------------------------------------------------
// The fields a transfer moves: up to three 3-double fields of a record (x, v,
// f), listed by increasing byte offset so that consecutive words of a record
// are consecutive in memory.
struct RecFields {
    long off[3];   // byte offset of each field in the record
    int id[3];     // 0 = x, 1 = v, 2 = f
    int nf;
};

static RecFields rec_fields(long off_x, long off_v, long off_f) {
    RecFields fl;
    fl.nf = 0;
    const long offs[3] = {off_x, off_v, off_f};
    for (int k = 0; k < 3; ++k)
        if (offs[k] >= 0) {
            int at = fl.nf++;
            while (at > 0 && fl.off[at - 1] > offs[k]) {
                fl.off[at] = fl.off[at - 1];
                fl.id[at] = fl.id[at - 1];
                --at;
            }
            fl.off[at] = offs[k];
            fl.id[at] = k;
        }
    for (int k = fl.nf; k < 3; ++k) {
        fl.off[k] = 0;
        fl.id[k] = -1;
    }
    return fl;
}

// stage holds `count` records of `stride` bytes (device memory, or host
// memory the device can address).  Records -> SoA; new positions also refresh
// the two pair-kernel copies.  A CTA takes kIntThreads records: its threads
// first read the records' words in order (consecutive threads, consecutive
// words: a warp's loads fall on a few contiguous runs instead of 32 records)
// into shared memory, then one thread per record stores its fields.
__global__ void __launch_bounds__(kIntThreads) extract_kernel(const unsigned char *__restrict__ stage, long stride,
                                                              const RecFields fl, int count, int first,
                                                              const IntArgs a) {
    __shared__ double buf[kIntThreads * 9];
    const int r0 = blockIdx.x * kIntThreads;
    const int nr = min(kIntThreads, count - r0);
    const int nw = 3 * fl.nf;
    // all of a thread's (at most 9) loads are issued before the first is
    // used: over the host link each round trip takes microseconds
    double word[9];
#pragma unroll
    for (int u = 0; u < 9; ++u) {
        const int w = threadIdx.x + u * kIntThreads;
        if (w < nr * nw) {
            const int r = w / nw, q = w - r * nw, k = q / 3;
            const long off = k == 0 ? fl.off[0] : (k == 1 ? fl.off[1] : fl.off[2]);
            word[u] = reinterpret_cast<const double *>(stage + (size_t)(r0 + r) * stride + off)[q - 3 * k];
        }
    }
#pragma unroll
    for (int u = 0; u < 9; ++u) {
        const int w = threadIdx.x + u * kIntThreads;
        if (w < nr * nw) buf[w] = word[u];
    }
    __syncthreads();
    const int r = threadIdx.x;
    if (r >= nr) return;
    const int i = first + r0 + r, n = a.n;
    const double *rec = buf + r * nw;
    for (int k = 0; k < fl.nf; ++k) {
        const int id = k == 0 ? fl.id[0] : (k == 1 ? fl.id[1] : fl.id[2]);
        const double *w = rec + 3 * k;
        if (id == 0) {
            store_pos(a, i, w[0], w[1], w[2]);
        } else {
            double *dst = id == 1 ? a.v : a.f;
            for (int d = 0; d < 3; ++d) dst[(size_t)d * n + i] = w[d];
        }
    }
}

// SoA -> host records: the inverse of extract_kernel, writing the fields of
// record r at dst + r*stride + off (dst in host memory the device can
// address).  One thread per 8-byte word, consecutive threads on consecutive
// words of the record span, so that a warp's stores fall on a few contiguous
// runs of host memory.
__global__ void scatter_kernel(unsigned char *__restrict__ dst, long stride, const RecFields fl, int count,
                               int first, int n, const double *x, const double *v, const double *f) {
    const int nw = 3 * fl.nf;
    const long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= (long long)count * nw) return;
    const int r = (int)(w / nw), q = (int)(w - (long long)r * nw), k = q / 3, d = q - 3 * k;
    const long off = k == 0 ? fl.off[0] : (k == 1 ? fl.off[1] : fl.off[2]);
    const int id = k == 0 ? fl.id[0] : (k == 1 ? fl.id[1] : fl.id[2]);
    const double *src = id == 0 ? x : (id == 1 ? v : f);
    reinterpret_cast<double *>(dst + (size_t)r * stride + off)[d] = src[(size_t)d * n + first + r];
}

// SoA -> [count][fields][3] packed doubles
__global__ void pack_kernel(double *__restrict__ out, int count, int first, int n, const double *x,
                            const double *v, const double *f, const double *f2, int nf) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= count) return;
    const int i = first + r;
    const double *src[4] = {x, v, f, f2};
    int slot = 0;
    for (int q = 0; q < 4; ++q) {
        if (!src[q]) continue;
        for (int d = 0; d < 3; ++d) out[((size_t)r * nf + slot) * 3 + d] = src[q][(size_t)d * n + i];
        ++slot;
    }
}

// FP32 peak: 8 independent FFMA chains per thread
__global__ void ffma_peak_kernel(float *out, int iters, float a, float b) {
    float r0 = threadIdx.x, r1 = r0 + 1, r2 = r0 + 2, r3 = r0 + 3, r4 = r0 + 4, r5 = r0 + 5, r6 = r0 + 6,
          r7 = r0 + 7;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            r0 = fmaf(r0, a, b);
            r1 = fmaf(r1, a, b);
            r2 = fmaf(r2, a, b);
            r3 = fmaf(r3, a, b);
            r4 = fmaf(r4, a, b);
            r5 = fmaf(r5, a, b);
            r6 = fmaf(r6, a, b);
            r7 = fmaf(r7, a, b);
        }
    }
    const float s = r0 + r1 + r2 + r3 + r4 + r5 + r6 + r7;
    if (s == 1234.5f) out[0] = s;   // keeps the chains live
}

// ---------------------------------------------------------------------------
static IntArgs int_args(tcp_ctx *c) {
    IntArgs a;
    a.x = c->x;
    a.v = c->v;
    a.f = c->f;
    a.xq = c->xq;
    a.xd = c->xd;
    a.xl = c->xl;
    a.copies = c->p.precision == TCP_PREC_FP32C ? kCopyXq : (kCopyXd | kCopyXl);
    a.nel = c->nel;
    a.n = c->n;
    a.xm0 = c->p.xm[0];
    a.xm1 = c->p.xm[1];
    a.L0 = c->p.box[0];
    a.L1 = c->p.box[1];
    a.L2 = c->p.box[2];
    a.iL0 = 1.0 / a.L0;
    a.iL1 = 1.0 / a.L1;
    a.iL2 = 1.0 / a.L2;
    return a;
}

static int nblocks(int n) { return (n + kIntThreads - 1) / kIntThreads; }

// red[] layout: [3][nb] force sums | [2][nb] kinetic pass 0 | [2][nb] pass 1 | recip energy
int part_blocks(int n) { return (n + kPartBlock - 1) / kPartBlock; }
double *fsum_part(tcp_ctx *c) { return c->red; }
double *mv_part(tcp_ctx *c, int pass) { return c->red + 3 * (size_t)part_blocks(c->n) + (size_t)pass * 2 * part_blocks(c->n); }
double *recip_epart(tcp_ctx *c) { return c->red + 7 * (size_t)part_blocks(c->n); }
int red_capacity(int n, int extra) { return 7 * part_blocks(n) + extra; }

int launch_refresh_positions(tcp_ctx *c, const double *x) {
    refresh_kernel<<<nblocks(3 * c->n), kIntThreads, 0, c->stream>>>(int_args(c), x ? x : c->x);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_shift(tcp_ctx *c, double sdt) {
    shift_kernel<<<nblocks(c->n), kIntThreads, 0, c->stream>>>(int_args(c), sdt);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

static StepPrep step_prep(tcp_ctx *c) {
    StepPrep s;
    s.fpart = c->fpart;
    s.upart = c->upart;
    s.nupart = c->n_upart;
    s.counter = c->counter;
    s.bin = c->p.reciprocal == TCP_RECIP_SPME;
    if (s.bin) {
        s.chain = spme_chain_args(c);
        s.chain.ticket = c->tickets + kTickStep;
    }
    return s;
}

int launch_vverlet1(tcp_ctx *c, double dt, bool prepare) {
    StepPrep s;
    s.fpart = nullptr;
    s.bin = 0;
    if (prepare) s = step_prep(c);
    const double h0 = 0.5 * dt / c->p.xm[0], h1 = 0.5 * dt / c->p.xm[1];
    const int stoch = c->p.thermo == TCP_THERMO_STOCH, nb = part_blocks(c->n);
    if (s.bin)
        vverlet1_kernel<true, true><<<nb, kPartThreads, 0, c->stream>>>(int_args(c), dt, h0, h1, c->p.alpha_lgv, stoch, s);
    else
        vverlet1_kernel<false, true><<<nb, kPartThreads, 0, c->stream>>>(int_args(c), dt, h0, h1, c->p.alpha_lgv, stoch, s);
    c->cleared = prepare;
    c->binned = s.bin != 0;
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_prepare(tcp_ctx *c) {
    const StepPrep s = step_prep(c);
    if (s.bin)
        vverlet1_kernel<true, false><<<part_blocks(c->n), kPartThreads, 0, c->stream>>>(int_args(c), 0.0, 0.0, 0.0, 0.0, 0, s);
    else
        vverlet1_kernel<false, false><<<part_blocks(c->n), kPartThreads, 0, c->stream>>>(int_args(c), 0.0, 0.0, 0.0, 0.0, 0, s);
    c->cleared = true;
    c->binned = s.bin != 0;
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_force_finalize(tcp_ctx *c, bool add_rec, bool energy) {
    force_finalize_kernel<<<part_blocks(c->n), kPartThreads, 0, c->stream>>>(
        c->fpart, c->fpart_splits, add_rec ? c->frec : nullptr, c->f, c->n, fsum_part(c), c->status, c->scal,
        energy ? c->upart : nullptr, c->n_upart_used, c->tickets + kTickForce);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_spme_sum(tcp_ctx *c) {
    add_rec_kernel<<<part_blocks(c->n), kPartThreads, 0, c->stream>>>(c->f, c->frec, c->n, fsum_part(c), c->scal,
                                                                      c->tickets + kTickAdd);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_fsum(tcp_ctx *c) {
    add_rec_kernel<<<part_blocks(c->n), kPartThreads, 0, c->stream>>>(c->f, nullptr, c->n, fsum_part(c), c->scal,
                                                                      c->tickets + kTickAdd);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_remove_rigid(tcp_ctx *c) {
    remove_net_kernel<<<nblocks(3 * c->n), kIntThreads, 0, c->stream>>>(c->f, c->n, c->scal);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_kick2(tcp_ctx *c, double dt, bool remove_net, bool apply_thermo, bool vdf) {
    KickArgs k;
    k.a = int_args(c);
    k.dt = dt;
    k.hdm0 = 0.5 * dt / c->p.xm[0];
    k.hdm1 = 0.5 * dt / c->p.xm[1];
    k.thermo = c->p.thermo;
    const bool rescale = apply_thermo && (c->p.thermo == TCP_THERMO_ISOKIN || c->p.thermo == TCP_THERMO_BEREND);
    if (!apply_thermo && k.thermo != TCP_THERMO_STOCH) k.thermo = TCP_THERMO_NOTEMP;
    k.remove_net = remove_net;
    k.mv_part = mv_part(c, 0);
    k.vdf = vdf && !rescale;
    k.vdf_counts = c->vdf;
    k.dv0 = c->p.dv_e;
    k.dv1 = c->p.dv_i;
    k.T0 = c->p.Te;
    k.T1 = c->p.Ti;
    k.tau = c->p.tau;
    k.alpha_lgv = c->p.alpha_lgv;
    k.seed = c->p.seed;
    k.scal = c->scal;
    k.last_pass = !rescale;
    k.ticket = c->tickets + kTickKick;
    const int nb = part_blocks(c->n);
    kick2_kernel<<<nb, kPartThreads, 0, c->stream>>>(k);
    c->launches++;
    if (rescale) {
        k.thermo = c->p.thermo;
        k.remove_net = 0;
        k.mv_part = mv_part(c, 1);
        k.vdf = vdf;
        k.last_pass = 1;
        k.ticket = c->tickets + kTickScale;
        rescale_kernel<<<nb, kPartThreads, 0, c->stream>>>(k);
        c->launches++;
    }
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_extract(tcp_ctx *c, const unsigned char *src, int first, int count, long stride, long off_x, long off_v,
                   long off_f, cudaStream_t st) {
    const RecFields fl = rec_fields(off_x, off_v, off_f);
    if (fl.nf == 0 || count <= 0) return TCP_OK;
    extract_kernel<<<nblocks(count), kIntThreads, 0, st ? st : c->stream>>>(src, stride, fl, count, first,
                                                                             int_args(c));
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_scatter(tcp_ctx *c, unsigned char *dst, int first, int count, long stride, long off_x, long off_v,
                   long off_f, const double *fsrc, cudaStream_t st) {
    const RecFields fl = rec_fields(off_x, off_v, off_f);
    if (fl.nf == 0 || count <= 0) return TCP_OK;
    const long long words = (long long)count * 3 * fl.nf;
    scatter_kernel<<<(unsigned)((words + kIntThreads - 1) / kIntThreads), kIntThreads, 0, st ? st : c->stream>>>(
        dst, stride, fl, count, first, c->n, c->x, c->v, fsrc);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_pack(tcp_ctx *c, int first, int count, bool x, bool v, bool f, bool frec, int *nf) {
    *nf = (int)x + (int)v + (int)f + (int)frec;
    pack_kernel<<<nblocks(count), kIntThreads, 0, c->stream>>>(reinterpret_cast<double *>(c->d_stage), count, first,
                                                               c->n, x ? c->x : nullptr, v ? c->v : nullptr,
                                                               f ? c->f : nullptr, frec ? c->frec : nullptr, *nf);
    c->launches++;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

int launch_fp32_peak(int device, double *tffma) {
    cudaDeviceProp prop;
    TCP_CUDA(cudaGetDeviceProperties(&prop, device));
    float *out;
    TCP_CUDA(cudaMalloc(&out, sizeof(float)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = prop.multiProcessorCount * 8, threads = 256, iters = 4096;
    ffma_peak_kernel<<<blocks, threads>>>(out, 16, 1.0000001f, 1e-7f);   // warm-up
    cudaEventRecord(e0);
    ffma_peak_kernel<<<blocks, threads>>>(out, iters, 1.0000001f, 1e-7f);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    const double ffma = (double)blocks * threads * iters * 16.0 * 8.0;
    *tffma = ffma / (ms * 1e-3) / 1e12;
    TCP_CUDA(cudaGetLastError());
    return TCP_OK;
}

}  // namespace tcp
