// spme_chain.cu -- charge spreading and force gather of the SPME chain
// (Force_SPME4, force.f90:697-755 and 868-919), for one system or a batch.
//
// The spread is atomic-free and every mesh point is summed in the same order
// on every call: particles are counting-sorted by the (y, z) mesh column of
// their support's base point (bin = by + K2 bz), each bin in particle order,
// and a mesh row is then gathered from the P^2 bins that reach it.
//
//   bin      per particle: base indexes, spline arguments, bin and slot
//            (integer atomics; fused into the half kick of a step); its last
//            CTA scans the bin counts
//   place    list by bin
//   weights  particles in bin order (a particle's place inside its bin is the
//            number of smaller indexes there) and their 6P spline values
//   spread   rows of the mesh gather their particles, P lanes per row
//   gather   8 lanes per particle over its P^2 rows
//
// These kernels are short (microseconds) and latency-bound on small systems,
// so the launches in sequence were cut (the memset, scan and in-bin sort have
// no launch of their own) and each is spread over as many SMs as there are
// particles for: a thread per component, 64 particles per CTA.
#include <algorithm>

#include "spme_chain.cuh"

namespace tcp {

// one system's binning when no half kick did it (a force call on its own, the
// Hessian-vector products)
template <typename T>
__global__ void __launch_bounds__(kPartThreads) chain_bin_kernel(const ChainArgs c, const double *__restrict__ x) {
    __shared__ int sb[3][kPartBlock];
    __shared__ double sa[3][kPartBlock];
    const int k = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, m = blockIdx.x * kPartBlock + k;
    const SpmeGeom &g = c.one;
    if (m < c.n) sb[d][k] = bin_axis(x[(size_t)d * c.n + m], g.hL[d], g.KL[d], g.K[d], c.P, sa[d][k]);
    __syncthreads();
    if (d == 0 && m < c.n) {
        const double a[3] = {sa[0][k], sa[1][k], sa[2][k]};
        bin_store<T>(c.b, m, c.n, a, m < g.nel ? g.q[0] : g.q[1], sb[0][k], sb[1][k], sb[2][k], g.K[1], 0);
    }
    if (c.nbins <= kScanTail && last_block(c.ticket)) scan_bins(c.b, c.nbins);
}

// prefix sums of many bins in three launches (the first also zeroes the counts)
constexpr int kScanBlock = 1024;
__global__ void scan_block_kernel(const SpreadBins b, int nbins) {
    __shared__ int ws[32];
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    const int v = i < nbins ? b.count[i] : 0;
    if (i < nbins) b.count[i] = 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        int t = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        ws[lane] = t;
    }
    __syncthreads();
    const int incl = x + (w > 0 ? ws[w - 1] : 0);
    if (i < nbins) b.start[i] = incl - v;
    if (threadIdx.x == kScanBlock - 1) b.bsum[blockIdx.x] = incl;
}

// every CTA adds the block sums before its own (a few hundred at most)
__global__ void __launch_bounds__(kScanBlock) scan_add_kernel(const SpreadBins b, int nbins, int total) {
    __shared__ int ws[32];
    __shared__ int base;
    int v = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kScanBlock) v += b.bsum[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        v = ws[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) base = v;
    }
    __syncthreads();
    const int i = blockIdx.x * kScanBlock + threadIdx.x;
    if (i < nbins) b.start[i] += base;
    if (i == 0) b.start[nbins] = total;
}

__global__ void chain_place_kernel(int n, SpreadBins b) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) b.list[b.start[b.bin[m]] + b.rank[m]] = m;
}

template <int P, typename T>
__global__ void __launch_bounds__(kPartThreads) chain_weights_kernel(int n, SpreadBins b) {
    __shared__ int spos[kPartBlock], sm[kPartBlock];
    const int k = threadIdx.x % kPartBlock, d = threadIdx.x / kPartBlock, t = blockIdx.x * kPartBlock + k;
    if (d == 0 && t < n) {
        const int m = b.list[t], bin = b.bin[m], s = b.start[bin], e = b.start[bin + 1];
        int pos = s;
        for (int q = s; q < e; ++q) pos += b.list[q] < m;
        spos[k] = pos;
        sm[k] = m;
        b.order[pos] = m;
        b.base[pos] = b.base_m[m];
        static_cast<T *>(b.q)[pos] = static_cast<const T *>(b.q_m)[m];
    }
    __syncthreads();
    if (t >= n) return;
    T W[P], dW[P];
    spline_at<P, T>(static_cast<const T *>(b.arg)[(size_t)d * n + sm[k]], W, dW);
    T *w = static_cast<T *>(b.ew) + ((size_t)spos[k] * 3 + d) * 2 * P;
#pragma unroll
    for (int j = 0; j < P; ++j) {
        w[j] = W[j];
        w[P + j] = dW[j];
    }
}

// The spread on its own (meshes that cuFFT transforms, and the Hessian-vector
// products): a CTA owns a few rows of one plane, P lanes per row (chain_rows).
// A warp that owned 8, 4 or 2 rows and laid the P x P points of a plane over
// its lanes executed 3-5 times the instructions, most lanes past the owned
// rows (whole chain at N = 9,000, 48^3, order 6, FP64: 240 us then, 163 us now).
constexpr int kSpreadThreads = 128;
template <int P, typename T, bool BATCH, bool DIP = false>
__global__ void __launch_bounds__(kSpreadThreads) chain_spread_kernel(const ChainArgs c, int rows, int per_plane) {
    constexpr bool F32 = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char smem[];
    // CTA -> (system, plane, first row): the planes are numbered like the bins
    int s = 0;
    if (BATCH) {
        int lo = 0, hi = c.nsys - 1;
        const int b = blockIdx.x / per_plane;    // plane among all systems' (plane_off ascending)
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (c.many[mid].plane_off <= b) lo = mid; else hi = mid - 1;
        }
        s = lo;
    }
    const SpmeGeom &g = BATCH ? c.many[s] : c.one;
    const int z = blockIdx.x / per_plane - (BATCH ? g.plane_off : 0), y0 = (blockIdx.x % per_plane) * rows;
    const int nrow = min(rows, g.K[1] - y0), K1 = g.K[0];
    if (nrow <= 0 || (BATCH && g.own)) return;   // batch: a smaller mesh than the largest, or fft_convolve's
    T *h = reinterpret_cast<T *>(smem);
    float *lo = reinterpret_cast<float *>(h + (size_t)rows * c.k1max);
    const StageBuf<T> st = stage_at<T>(smem + (size_t)rows * c.k1max * 8, P);
    for (int k = threadIdx.x; k < nrow * K1; k += kSpreadThreads) {
        h[k] = (T)0;
        if (F32) lo[k] = 0.f;
    }
    chain_rows<P, T, kSpreadThreads, DIP>(c, g, z, y0, nrow, h, lo, K1, st, threadIdx.x, 1, 0, 1);
    __syncthreads();
    T *mesh = static_cast<T *>(c.mesh) + g.mesh_off + (size_t)K1 * (y0 + (size_t)g.K[1] * z);
    for (int k = threadIdx.x; k < nrow * K1; k += kSpreadThreads) mesh[k] = F32 ? h[k] + (T)lo[k] : h[k];
}

// force gather, force.f90:868-919: 8 lanes per particle, each over every
// eighth of its P^2 mesh rows, in T; the sums over lanes in T, the force in
// FP64.  Particles in bin order, so that a warp's rows are read together.
// Bound: L2 latency (a thread per particle ran the P^2 rows one after the
// other: 12.1 us at N = 4,096, order 4, now 5.9 us).  The last CTA adds up the energy partials of the
// influence multiply (single systems).
constexpr int kGatherThreads = 128;
template <int P, typename T, bool BATCH>
__global__ void __launch_bounds__(kGatherThreads) chain_gather_kernel(const ChainArgs c, double *__restrict__ frec,
                                                                      const double *__restrict__ epart, int nepart,
                                                                      double escale, double *__restrict__ um) {
    constexpr int NP = kGatherThreads / 8;
    __shared__ T sw[NP * 6 * P];
    __shared__ double red[32];
    if (um && blockIdx.x == gridDim.x - 1) {
        double e = 0.0;
        for (int k = threadIdx.x; k < nepart; k += kGatherThreads) e += epart[k];
        e = block_sum(e, red);
        if (threadIdx.x == 0) *um = e * escale;
        return;
    }
    const int t0 = blockIdx.x * NP, np = min(NP, c.n - t0);
    const T *ew = static_cast<const T *>(c.b.ew) + (size_t)t0 * 6 * P;
    for (int k = threadIdx.x; k < np * 6 * P; k += kGatherThreads) sw[k] = ew[k];
    __syncthreads();
    const int p = threadIdx.x >> 3, sub = threadIdx.x & 7;
    const int t = t0 + min(p, np - 1);           // idle groups repeat the last particle
    const int m = c.b.order[t];
    const SpmeGeom &g = BATCH ? c.many[c.sys_of[m]] : c.one;
    const int4 base = c.b.base[t];
    const int K1 = g.K[0], K2 = g.K[1], K3 = g.K[2], bx = base.x, by = base.y, bz = base.z;
    const T *w = sw + (size_t)min(p, np - 1) * 6 * P;
    const T *mesh = static_cast<const T *>(c.mesh) + g.mesh_off;
    int xs[P];
    T W[P], dW[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
        W[i] = w[i];
        dW[i] = w[P + i];
        const int x = bx + i;
        xs[i] = x >= K1 ? x - K1 : x;
    }
    T gx = 0, gy = 0, gz = 0;
#pragma unroll
    for (int r0 = 0; r0 < P * P; r0 += 8) {
        const int r = r0 + sub;
        if (r < P * P) {
            const int k = r / P, j = r - k * P;
            int iy = by + j, iz = bz + k;
            iy -= iy >= K2 ? K2 : 0;
            iz -= iz >= K3 ? K3 : 0;
            const T *row = mesh + (size_t)K1 * (iy + (size_t)K2 * iz);
            T sx = 0, sd = 0;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const T ph = row[xs[i]];
                sx += dW[i] * ph;
                sd += W[i] * ph;
            }
            const T wy = w[2 * P + j], dy = w[3 * P + j], wz = w[4 * P + k], dz = w[5 * P + k];
            gx += sx * (wy * wz);
            gy += sd * (dy * wz);
            gz += sd * (wy * dz);
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
        gx += __shfl_xor_sync(0xffffffffu, gx, o);
        gy += __shfl_xor_sync(0xffffffffu, gy, o);
        gz += __shfl_xor_sync(0xffffffffu, gz, o);
    }
    if (sub < 3 && p < np) {
        // F = -eps/(pi V) q (K_d/L_d) sum dW W W phi
        const double q = m - g.off < g.nel ? g.q[0] : g.q[1];
        const double s = sub == 0 ? (double)gx : (sub == 1 ? (double)gy : (double)gz);
        frec[(size_t)sub * c.n + m] = -g.coef * q * s * g.KL[sub];
    }
}

// The reciprocal Hessian-vector product's gather, 8 lanes per particle as
// above, always FP64: (H w)_i = c q_i [sum_k (hess W_i(k) w_i) phi(k) + sum_k
// grad W_i(k) dphi(k)].  Bound: the FP64 pipe (about 45 operations a mesh row)
// and L2 latency; a thread per particle took 45 us at N = 4,096, order 4.
template <int P>
__global__ void __launch_bounds__(kGatherThreads) chain_gather_hvp_kernel(const ChainArgs c, const double *__restrict__ phi,
                                                                          const double *__restrict__ dphi,
                                                                          const double *__restrict__ w,
                                                                          double *__restrict__ hw) {
    constexpr int NP = kGatherThreads / 8;
    __shared__ double sw[NP][3][3 * P];          // W, W', W'' per axis
    const int t0 = blockIdx.x * NP, np = min(NP, c.n - t0);
    const int p = min((int)threadIdx.x >> 3, np - 1), sub = threadIdx.x & 7;   // idle groups repeat the last particle
    const bool live = (int)threadIdx.x >> 3 < np;
    const int m = c.b.order[t0 + p];
    const SpmeGeom &g = c.one;
    if (live && sub < 3) {
        double W[P], dW[P], d2W[P];
        const double arg = static_cast<const double *>(c.b.arg)[(size_t)sub * c.n + m], kl = g.KL[sub];
        spline_w2<P>(P == 4 ? 1.0 - arg : arg, W, dW, d2W);
#pragma unroll
        for (int j = 0; j < P; ++j) {
            sw[p][sub][j] = W[j];
            sw[p][sub][P + j] = dW[j] * kl;
            sw[p][sub][2 * P + j] = d2W[j] * (kl * kl);
        }
    }
    __syncthreads();
    const int4 base = c.b.base[t0 + p];
    const int K1 = g.K[0], K2 = g.K[1], K3 = g.K[2];
    const int bx = base.x, by = base.y, bz = base.z;
    const double *sx = sw[p][0], *sy = sw[p][1], *sz = sw[p][2];
    const double w0 = w[m], w1 = w[(size_t)c.n + m], w2 = w[2 * (size_t)c.n + m];
    double h[3] = {0.0, 0.0, 0.0};
    for (int r = sub; r < P * P; r += 8) {
        const int k = r / P, j = r - k * P;
        int iy = by + j, iz = bz + k;
        iy -= iy >= K2 ? K2 : 0;
        iz -= iz >= K3 ? K3 : 0;
        const size_t ro = (size_t)K1 * (iy + (size_t)K2 * iz);
        double sp = 0, sdp = 0, sd2p = 0, sq = 0, sdq = 0;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int x = bx + i >= K1 ? bx + i - K1 : bx + i;
            const double ph = phi[ro + x], dph = dphi[ro + x];
            sp = fma(sx[i], ph, sp);
            sdp = fma(sx[P + i], ph, sdp);
            sd2p = fma(sx[2 * P + i], ph, sd2p);
            sq = fma(sx[i], dph, sq);
            sdq = fma(sx[P + i], dph, sdq);
        }
        const double Wy = sy[j], dWy = sy[P + j], d2Wy = sy[2 * P + j], Wz = sz[k], dWz = sz[P + k], d2Wz = sz[2 * P + k];
        // Hessian of W x gradient rows, times w, times phi; gradient times dphi
        const double yz = Wy * Wz, dyz = dWy * Wz, ydz = Wy * dWz;
        const double hxy = sdp * dyz, hxz = sdp * ydz, hyz = sp * (dWy * dWz);
        h[0] += fma(fma(sd2p, w0, sdq), yz, fma(hxy, w1, hxz * w2));
        h[1] += fma(hxy, w0, fma(fma(sp, d2Wy * w1, sq * dWy), Wz, hyz * w2));
        h[2] += fma(hxz, w0, fma(hyz, w1, Wy * fma(sp, d2Wz * w2, sq * dWz)));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int d = 0; d < 3; ++d) h[d] += __shfl_xor_sync(0xffffffffu, h[d], o);
    if (live && sub < 3) {
        const double q = m < g.nel ? g.q[0] : g.q[1];
        hw[(size_t)sub * c.n + m] += g.coef * q * (sub == 0 ? h[0] : (sub == 1 ? h[1] : h[2]));
    }
}

// ---------------------------------------------------------------------------
int chain_bin(const ChainArgs &c, const double *x, cudaStream_t st) {
    const int blocks = (c.n + kPartBlock - 1) / kPartBlock;
    if (c.fp64)
        chain_bin_kernel<double><<<blocks, kPartThreads, 0, st>>>(c, x);
    else
        chain_bin_kernel<float><<<blocks, kPartThreads, 0, st>>>(c, x);
    return 1;
}

// Rows of a CTA of the spread: one pass of its warps, or what fits
static int chain_spread_rows(int P, int k1max) {
    const int rows = kSpreadThreads / 32 * (32 / P);
    return std::max(1, std::min(rows, (int)((150u << 10) / ((size_t)k1max * 8))));
}
static size_t chain_spread_bytes(int P, int k1max) {   // two-float FP32 or FP64: 8 bytes a point
    return (size_t)chain_spread_rows(P, k1max) * k1max * 8 + std::max(stage_bytes<double>(P), stage_bytes<double>(P, true));
}

template <int P, typename T>
static int sort_p(const ChainArgs &c, cudaStream_t st) {
    const int nb = (c.n + kPartBlock - 1) / kPartBlock;
    int launches = 2;
    if (c.nbins > kScanTail) {
        const int sb = (c.nbins + kScanBlock - 1) / kScanBlock;
        scan_block_kernel<<<sb, kScanBlock, 0, st>>>(c.b, c.nbins);
        scan_add_kernel<<<sb, kScanBlock, 0, st>>>(c.b, c.nbins, c.n);
        launches += 2;
    }
    chain_place_kernel<<<(c.n + 127) / 128, 128, 0, st>>>(c.n, c.b);
    chain_weights_kernel<P, T><<<nb, kPartThreads, 0, st>>>(c.n, c.b);
    return launches;
}

template <int P, typename T, bool BATCH>
static int spread_p(const ChainArgs &c, cudaStream_t st) {
    const int rows = chain_spread_rows(P, c.k1max), per_plane = (c.k2max + rows - 1) / rows;
    const size_t sm = chain_spread_bytes(P, c.k1max);
    if (!BATCH && sizeof(T) == 8 && c.dipole)
        chain_spread_kernel<P, double, false, true><<<c.planes * per_plane, kSpreadThreads, sm, st>>>(c, rows, per_plane);
    else
        chain_spread_kernel<P, T, BATCH><<<c.planes * per_plane, kSpreadThreads, sm, st>>>(c, rows, per_plane);
    return 1;
}

#define TCP_CHAIN_ORDER(CALL)           \
    switch (c.P) {                      \
        case 4: CALL(4); break;         \
        case 5: CALL(5); break;         \
        case 6: CALL(6); break;         \
        case 7: CALL(7); break;         \
        default: CALL(8); break;        \
    }

int chain_sort(const ChainArgs &c, cudaStream_t st) {
    int n = 0;
#define TCP_CALL(P) n = c.fp64 ? sort_p<P, double>(c, st) : sort_p<P, float>(c, st)
    TCP_CHAIN_ORDER(TCP_CALL)
#undef TCP_CALL
    return n;
}

int chain_spread(const ChainArgs &c, cudaStream_t st) {   // c.dipole: FP64 single systems
    int n = 0;
#define TCP_CALL(P) \
    n = c.many ? spread_p<P, float, true>(c, st) : (c.fp64 ? spread_p<P, double, false>(c, st) : spread_p<P, float, false>(c, st))
    TCP_CHAIN_ORDER(TCP_CALL)
#undef TCP_CALL
    return n;
}

template <int P, typename T, bool BATCH>
static void gather_p(const ChainArgs &c, double *frec, const double *epart, int nepart, double escale, double *um,
                     cudaStream_t st) {
    constexpr int NP = kGatherThreads / 8;
    chain_gather_kernel<P, T, BATCH><<<(c.n + NP - 1) / NP + (um ? 1 : 0), kGatherThreads, 0, st>>>(c, frec, epart, nepart,
                                                                                                   escale, um);
}

int chain_gather(const ChainArgs &c, double *frec, const double *epart, int nepart, double escale, double *um,
                 cudaStream_t st) {
#define TCP_CALL(P)                                                                            \
    if (c.many) gather_p<P, float, true>(c, frec, epart, nepart, escale, um, st);              \
    else if (c.fp64) gather_p<P, double, false>(c, frec, epart, nepart, escale, um, st);       \
    else gather_p<P, float, false>(c, frec, epart, nepart, escale, um, st)
    TCP_CHAIN_ORDER(TCP_CALL)
#undef TCP_CALL
    return 1;
}

int chain_gather_hvp(const ChainArgs &c, const double *phi, const double *dphi, const double *w, double *hw,
                     cudaStream_t st) {
    constexpr int NP = kGatherThreads / 8;
#define TCP_CALL(P) chain_gather_hvp_kernel<P><<<(c.n + NP - 1) / NP, kGatherThreads, 0, st>>>(c, phi, dphi, w, hw)
    TCP_CHAIN_ORDER(TCP_CALL)
#undef TCP_CALL
    return 1;
}

// shared-memory limit of the spread for this mesh (once, outside any capture)
int chain_prepare(const ChainArgs &c) {
    const size_t bytes = chain_spread_bytes(c.P, c.k1max);
    int rc = TCP_OK;
#define TCP_LIMIT(K) \
    if (!rc) rc = allow_shared(reinterpret_cast<const void *>(K), bytes)
#define TCP_CALL(P)                                    \
    do {                                               \
        TCP_LIMIT((chain_spread_kernel<P, float, true>));    \
        TCP_LIMIT((chain_spread_kernel<P, float, false>));   \
        TCP_LIMIT((chain_spread_kernel<P, double, false>));  \
        TCP_LIMIT((chain_spread_kernel<P, double, false, true>)); \
    } while (0)
    TCP_CHAIN_ORDER(TCP_CALL)
#undef TCP_CALL
#undef TCP_LIMIT
    return rc;
}

// bins of a system of n particles and nbins mesh columns (T at most double)
int chain_alloc(SpreadBins &b, int n, int nbins, int order) {
    const size_t rounds = (size_t)nbins + 16 * kPartThreads;   // whole rounds of scan_bins
    struct { void **p; size_t bytes; } want[] = {
        {(void **)&b.count, sizeof(int) * rounds}, {(void **)&b.start, sizeof(int) * ((size_t)nbins + 1)},
        {(void **)&b.bsum, sizeof(int) * ((size_t)nbins / kScanBlock + 1)}, {(void **)&b.rank, sizeof(int) * (size_t)n},
        {(void **)&b.list, sizeof(int) * (size_t)n}, {(void **)&b.order, sizeof(int) * (size_t)n},
        {(void **)&b.bin, sizeof(int) * (size_t)n}, {(void **)&b.base_m, sizeof(int4) * (size_t)n},
        {(void **)&b.base, sizeof(int4) * (size_t)n}, {&b.arg, sizeof(double) * 3 * (size_t)n},
        {&b.q_m, sizeof(double) * (size_t)n}, {&b.q, sizeof(double) * (size_t)n},
        {&b.ew, sizeof(double) * 6 * (size_t)order * (size_t)n}};
    for (auto &w : want)
        if (cudaMalloc(w.p, w.bytes) != cudaSuccess) return set_error(TCP_ERR_NOMEM, "SPME bin allocation failed");
    TCP_CUDA(cudaMemset(b.count, 0, sizeof(int) * rounds));
    return TCP_OK;
}

void chain_free(SpreadBins &b) {
    void **p[] = {(void **)&b.count, (void **)&b.start, (void **)&b.bsum, (void **)&b.rank, (void **)&b.list,
                  (void **)&b.order, (void **)&b.bin, (void **)&b.base_m, (void **)&b.base, &b.arg, &b.q_m, &b.q, &b.ew};
    for (void **q : p) {
        cudaFree(*q);
        *q = nullptr;
    }
}

}  // namespace tcp
