// spme_fft.cu -- the convolution of the SPME chain on cubic meshes of 32, 48,
// 64, 96 or 128 points a side: charge spreading, forward transform, influence
// multiply with the energy, and inverse transform in three kernels, for one
// system or a batch (other meshes: cuFFT, spme.cu).
//
//   forward   a CTA owns one (x, y) plane: it gathers the plane's charges
//             (chain_rows) in shared memory and transforms it along x and y
//             there
//   z         a CTA owns 16 columns: transform along z, multiply by the
//             influence function (theta(m) |b(m)|^-2, force.f90:833-842), sum
//             the energy, transform back
//   inverse   a CTA owns one plane again: back along y and x, writes phi
//
// cuFFT takes three launches each way for these sizes, and spread and
// influence multiply one each; on small meshes every launch is a few
// microseconds of latency.  The whole chain in us, cuFFT and here:
//   N = 4,096, 32^3, order 4     FP32C 80  45   FP64 125  73
//   N = 9,000, 48^3, order 6          112  76        166 135
//   N = 16,384, 64^3, order 4          93  68        179 141
//   N = 40,000, 96^3, order 5         145 125        381 339
//   N = 65,536, 128^3, order 5        182 161        710 538
//
// A line of N = R1 R2 points is transformed in place in two passes of small
// DFTs held in registers: over the R1 points R2 a + b of each b, times the
// twiddle, then over the R2 points R2 c + d of each c.  Position R2 c + d then
// holds frequency c + R1 d; nothing is reordered: the influence function is
// stored in the same order and the inverse passes run backwards.  Two real
// rows share one complex transform, and the half spectrum of a row replaces
// its N reals: the real part of frequency k at the position of k, the
// imaginary part at that of N - k.
#include <cmath>
#include <vector>

#include "spme_chain.cuh"

namespace tcp {

template <typename T>
struct C2 {
    T x, y;
};
template <typename T>
__device__ __forceinline__ C2<T> cmul(C2<T> a, C2<T> b) {
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}

// cos(2 pi k / 48), k = 0 .. 12
__device__ constexpr double kCos48[13] = {1.0, 0.99144486137381041114, 0.96592582628906828675, 0.92387953251128675613, 0.86602540378443864676, 0.79335334029123516458, 0.7071067811865475244, 0.60876142900872063942, 0.5, 0.38268343236508977173, 0.25881904510252076235, 0.13052619222005159155, 0.0};
__device__ constexpr double cos48(int k) {
    k = k % 48;
    if (k > 24) k = 48 - k;
    return k <= 12 ? kCos48[k] : -kCos48[24 - k];
}
__device__ constexpr double sin48(int k) { return cos48(k + 36); }

// In-register DFT of R points, frequencies in order: exp(-2 pi i) forward,
// exp(+2 pi i) inverse, unnormalised.
template <int R>
struct Split;
template <> struct Split<4> { static constexpr int a = 2; };
template <> struct Split<6> { static constexpr int a = 3; };
template <> struct Split<8> { static constexpr int a = 4; };
template <> struct Split<12> { static constexpr int a = 4; };
template <> struct Split<16> { static constexpr int a = 4; };

template <int R, bool INV, typename T>
__device__ __forceinline__ void dft(C2<T> *v) {
    if constexpr (R == 2) {
        const C2<T> a = v[0], b = v[1];
        v[0] = {a.x + b.x, a.y + b.y};
        v[1] = {a.x - b.x, a.y - b.y};
    } else if constexpr (R == 3) {
        constexpr T h = (T)0.86602540378443864676;
        const C2<T> a = v[0], s = {v[1].x + v[2].x, v[1].y + v[2].y}, d = {v[1].x - v[2].x, v[1].y - v[2].y};
        const C2<T> m = {a.x - (T)0.5 * s.x, a.y - (T)0.5 * s.y};
        const T k = INV ? -h : h;
        v[0] = {a.x + s.x, a.y + s.y};
        v[1] = {m.x + k * d.y, m.y - k * d.x};
        v[2] = {m.x - k * d.y, m.y + k * d.x};
    } else if constexpr (R == 4) {
        const C2<T> s0 = {v[0].x + v[2].x, v[0].y + v[2].y}, d0 = {v[0].x - v[2].x, v[0].y - v[2].y};
        const C2<T> s1 = {v[1].x + v[3].x, v[1].y + v[3].y}, d1 = {v[1].x - v[3].x, v[1].y - v[3].y};
        v[0] = {s0.x + s1.x, s0.y + s1.y};
        v[2] = {s0.x - s1.x, s0.y - s1.y};
        if (INV) {
            v[1] = {d0.x - d1.y, d0.y + d1.x};
            v[3] = {d0.x + d1.y, d0.y - d1.x};
        } else {
            v[1] = {d0.x + d1.y, d0.y - d1.x};
            v[3] = {d0.x - d1.y, d0.y + d1.x};
        }
    } else {
        constexpr int A = Split<R>::a, B = R / A;
        C2<T> y[R];                              // [c][b]
#pragma unroll
        for (int b = 0; b < B; ++b) {
            C2<T> u[A];
#pragma unroll
            for (int a = 0; a < A; ++a) u[a] = v[B * a + b];
            dft<A, INV>(u);
#pragma unroll
            for (int c = 0; c < A; ++c) {
                const int k = (48 / R) * b * c;
                const C2<T> w = {(T)cos48(k), (T)(INV ? sin48(k) : -sin48(k))};
                y[c * B + b] = b * c == 0 ? u[c] : cmul(u[c], w);
            }
        }
#pragma unroll
        for (int c = 0; c < A; ++c) {
            dft<B, INV>(y + c * B);
#pragma unroll
            for (int d = 0; d < B; ++d) v[c + A * d] = y[c * B + d];
        }
    }
}

// N = R1 R2
template <int N>
struct Line;
template <> struct Line<32> { static constexpr int R1 = 4, R2 = 8; };
template <> struct Line<48> { static constexpr int R1 = 6, R2 = 8; };
template <> struct Line<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct Line<96> { static constexpr int R1 = 8, R2 = 12; };
template <> struct Line<128> { static constexpr int R1 = 8, R2 = 16; };

template <int N>
__host__ __device__ constexpr int pos_of(int k) { return Line<N>::R2 * (k % Line<N>::R1) + k / Line<N>::R1; }
// Column u of a plane in the packed half spectrum, u < N/2: the positions of
// its real and imaginary parts and its frequency; column 0 holds the real
// columns 0 and N/2.
template <int N>
__device__ __forceinline__ void column_of(int u, int &p, int &pi) {
    constexpr int R1 = Line<N>::R1, R2 = Line<N>::R2;
    const int c = u / (R2 / 2), d = u - c * (R2 / 2);
    p = R2 * c + d;
    pi = u == 0 ? R2 / 2 : (c == 0 ? R2 - d : R2 * (R1 - c) + (R2 - 1 - d));
}
template <int N>
__host__ __device__ constexpr int column_freq(int u) {
    return u / (Line<N>::R2 / 2) + Line<N>::R1 * (u % (Line<N>::R2 / 2));
}

// Threads of the plane kernels: enough warps for the P-lane rows of the
// spread, few enough registers for the radix-12 and -16 DFTs.  Small planes
// spread with several groups of threads, each taking its share of the P planes
// of particles into rows of its own, because a row's particles follow one
// another (32^3, N = 4,096: 64 a row).
template <int N, typename T>
__host__ __device__ constexpr int plane_threads() { return N <= 64 ? 512 : (sizeof(T) == 8 ? 384 : (N == 96 ? 512 : 704)); }
template <int N>
__host__ __device__ constexpr int spread_groups() { return N == 32 ? 4 : (N <= 64 ? 2 : 1); }
template <int N>
__host__ __device__ constexpr int plane_stride() { return N + 1; }
template <int N, typename T>
__host__ __device__ constexpr size_t plane_bytes(int P, bool dipole = false) {   // P = 0: the inverse kernel
    const size_t plane = (size_t)N * plane_stride<N>();
    return 2 * N * sizeof(T) + (P ? spread_groups<N>() * (plane * 8 + stage_bytes<T>(P, dipole)) : plane * sizeof(T));
}

// The two passes over a line whose points are re[n * step], im[n * step]; the
// inverse runs pass two first.
template <int N, bool INV, typename T>
__device__ __forceinline__ void pass_one(T *re, T *im, int step, int b, const C2<T> *tw) {
    constexpr int R1 = Line<N>::R1, R2 = Line<N>::R2;
    C2<T> v[R1];
#pragma unroll
    for (int a = 0; a < R1; ++a) {
        v[a] = {re[(R2 * a + b) * step], im[(R2 * a + b) * step]};
        if (INV) {
            const C2<T> w = tw[a * b];
            v[a] = cmul(v[a], {w.x, -w.y});
        }
    }
    dft<R1, INV>(v);
#pragma unroll
    for (int c = 0; c < R1; ++c) {
        if (!INV) v[c] = cmul(v[c], tw[c * b]);
        re[(R2 * c + b) * step] = v[c].x;
        im[(R2 * c + b) * step] = v[c].y;
    }
}
template <int N, bool INV, typename T>
__device__ __forceinline__ void pass_two(T *re, T *im, int step, int c) {
    constexpr int R2 = Line<N>::R2;
    C2<T> v[R2];
#pragma unroll
    for (int d = 0; d < R2; ++d) v[d] = {re[(R2 * c + d) * step], im[(R2 * c + d) * step]};
    dft<R2, INV>(v);
#pragma unroll
    for (int d = 0; d < R2; ++d) {
        re[(R2 * c + d) * step] = v[d].x;
        im[(R2 * c + d) * step] = v[d].y;
    }
}

template <int N, typename T, bool BATCH>
__device__ __forceinline__ const SpmeGeom &geom_of_block(const ChainArgs &c, const FftArgs &f, int per, int &local, int &sys) {
    sys = BATCH ? f.list[blockIdx.x / per] : 0;
    local = BATCH ? blockIdx.x % per : blockIdx.x;
    return BATCH ? c.many[sys] : c.one;
}

// DIP: the mesh dipoles of c.dipole instead of the charges.
template <int N, typename T, bool BATCH, bool DIP>
__global__ void __launch_bounds__(plane_threads<N, T>()) fft_forward_kernel(const ChainArgs c, const FftArgs f) {
    constexpr int NT = plane_threads<N, T>(), S = plane_stride<N>(), R1 = Line<N>::R1, R2 = Line<N>::R2;
    constexpr bool F32 = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char smem[];
    C2<T> *tw = reinterpret_cast<C2<T> *>(smem);
    T *hi = reinterpret_cast<T *>(tw + N);
    const int tid = threadIdx.x;
    int z, sys;
    const SpmeGeom &g = geom_of_block<N, T, BATCH>(c, f, N, z, sys);
    for (int k = tid; k < N; k += NT) tw[k] = static_cast<const C2<T> *>(f.tw)[k];
    {
        constexpr int G = spread_groups<N>(), NG = NT / G;
        const int q = tid / NG, t = tid - q * NG;
        // group q: its rows (two-float FP32 or FP64, 8 bytes a point) and its stage
        T *h = hi + (size_t)q * N * S;
        float *lo0 = reinterpret_cast<float *>(hi + (size_t)G * N * S), *lo = lo0 + (size_t)q * N * S;   // FP32C
        unsigned char *stages = reinterpret_cast<unsigned char *>(hi) + (size_t)G * N * S * 8;
        for (int k = t; k < N * S; k += NG) {
            h[k] = (T)0;
            if (F32) lo[k] = 0.f;
        }
#define TCP_ROWS(P)                                                                                                    \
    case P:                                                                                                            \
        chain_rows<P, T, NG, DIP>(c, g, z, 0, N, h, lo, S, stage_at<T>(stages + q * stage_bytes<T>(P, DIP), P), t, 1 + q, q, G); \
        break
        switch (c.P) {
            TCP_ROWS(4);
            TCP_ROWS(5);
            TCP_ROWS(6);
            TCP_ROWS(7);
            TCP_ROWS(8);
        }
#undef TCP_ROWS
        __syncthreads();
        for (int k = tid; k < N * S; k += NT) {
            T v = hi[k];
            float e = F32 ? lo0[k] : 0.f;
            for (int u = 1; u < G; ++u) {
                const T w = hi[(size_t)u * N * S + k];
                if (F32) {
                    const T sum = v + w, bp = sum - v;
                    e += lo0[(size_t)u * N * S + k] + (float)((v - (sum - bp)) + (w - bp));
                    v = sum;
                } else {
                    v += w;
                }
            }
            hi[k] = F32 ? v + (T)e : v;
        }
        __syncthreads();
    }
    // x: rows 2j and 2j + 1 as real and imaginary part
    for (int t = tid; t < N / 2 * R2; t += NT) {
        const int j = t / R2, b = t - j * R2;
        pass_one<N, false>(hi + 2 * j * S, hi + (2 * j + 1) * S, 1, b, tw);
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R1; t += NT) {
        const int j = t / R1, q = t - j * R1;
        pass_two<N, false>(hi + 2 * j * S, hi + (2 * j + 1) * S, 1, q);
    }
    __syncthreads();
    // the two rows' half spectra
    for (int t = tid; t < N / 2 * (N / 2); t += NT) {
        const int j = t / (N / 2), u = t - j * (N / 2);
        if (u == 0) continue;                    // frequencies 0 and N/2 are in place
        int p, q;
        column_of<N>(u, p, q);
        T *r0 = hi + 2 * j * S, *r1 = r0 + S;
        const C2<T> a = {r0[p], r1[p]}, b = {r0[q], r1[q]};
        r0[p] = (T)0.5 * (a.x + b.x);
        r0[q] = (T)0.5 * (a.y - b.y);
        r1[p] = (T)0.5 * (a.y + b.y);
        r1[q] = (T)0.5 * (b.x - a.x);
    }
    __syncthreads();
    // y
    for (int t = tid; t < N / 2 * R2; t += NT) {
        const int b = t / (N / 2), u = t - b * (N / 2);
        int p, q;
        column_of<N>(u, p, q);
        pass_one<N, false>(hi + p, hi + q, S, b, tw);
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R1; t += NT) {
        const int d = t / (N / 2), u = t - d * (N / 2);
        int p, q;
        column_of<N>(u, p, q);
        pass_two<N, false>(hi + p, hi + q, S, d);
    }
    __syncthreads();
    C2<T> *out = static_cast<C2<T> *>(f.half) + g.half_off + (size_t)z * (N / 2 + 1) * N;
    for (int t = tid; t < (N / 2 + 1) * N; t += NT) {
        const int u = t / N, y = t - u * N;
        int p, q;
        column_of<N>(u == N / 2 ? 0 : u, p, q);
        C2<T> v = {hi[y * S + p], hi[y * S + q]};
        if (u == 0 || u == N / 2) {              // the real columns 0 and N/2 share column 0
            const int k = y / R2 + R1 * (y % R2), ym = pos_of<N>((N - k) % N);
            const C2<T> w = {hi[ym * S + p], hi[ym * S + q]};
            v = u == 0 ? C2<T>{(T)0.5 * (v.x + w.x), (T)0.5 * (v.y - w.y)}
                       : C2<T>{(T)0.5 * (v.y + w.y), (T)0.5 * (w.x - v.x)};
        }
        out[t] = v;
    }
}

constexpr int kZCols = 16;
template <int N>
__host__ __device__ constexpr int z_threads() { return kZCols * Line<N>::R2; }

template <int N, typename T, bool BATCH>
__global__ void __launch_bounds__(z_threads<N>()) fft_z_kernel(const ChainArgs c, const FftArgs f) {
    constexpr int R1 = Line<N>::R1, R2 = Line<N>::R2, C = kZCols, ROW = (N / 2 + 1) * N, PER = ROW / C;
    static_assert(ROW % C == 0, "whole tiles of columns");
    __shared__ C2<T> s[N][C + 1];
    __shared__ C2<T> tw[N];
    __shared__ double red[32];
    int tile, sys;
    const SpmeGeom &g = geom_of_block<N, T, BATCH>(c, f, PER, tile, sys);
    const int tid = threadIdx.x, col = tid % C, q = tid / C, i = tile * C + col;
    for (int k = tid; k < N; k += z_threads<N>()) tw[k] = static_cast<const C2<T> *>(f.tw)[k];
    C2<T> *half = static_cast<C2<T> *>(f.half) + g.half_off + i;
    C2<T> v[R1];
#pragma unroll
    for (int a = 0; a < R1; ++a) v[a] = half[(size_t)(R2 * a + q) * ROW];
    dft<R1, false>(v);
    __syncthreads();                             // tw
#pragma unroll
    for (int k = 0; k < R1; ++k) s[R2 * k + q][col] = cmul(v[k], tw[k * q]);
    __syncthreads();
    double e = 0.0;
    if (q < R1) {
        C2<T> w[R2];
#pragma unroll
        for (int d = 0; d < R2; ++d) w[d] = s[R2 * q + d][col];
        dft<R2, false>(w);
        const T *infl = static_cast<const T *>(f.infl) + g.half_off + i;
        T et = 0;
#pragma unroll
        for (int d = 0; d < R2; ++d) {
            const T th = infl[(size_t)(R2 * q + d) * ROW];
            et += th * (w[d].x * w[d].x + w[d].y * w[d].y);
            w[d].x *= th;
            w[d].y *= th;
        }
        // columns 1 .. N/2 - 1 stand for a conjugate pair
        const int u = i / N;
        e = (double)et * (u == 0 || u == N / 2 ? 1.0 : 2.0);
        dft<R2, true>(w);
#pragma unroll
        for (int d = 0; d < R2; ++d) {
            const C2<T> t = tw[q * d];
            s[R2 * q + d][col] = cmul(w[d], {t.x, -t.y});
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < R1; ++a) v[a] = s[R2 * a + q][col];
    dft<R1, true>(v);
#pragma unroll
    for (int a = 0; a < R1; ++a) half[(size_t)(R2 * a + q) * ROW] = v[a];
    if (f.energy) {
        e = block_sum(e, red);
        if (tid == 0) {
            if (BATCH) atomicAdd(f.um + sys, e * g.ecoef);
            else f.epart[blockIdx.x] = e;
        }
    }
}

template <int N, typename T, bool BATCH>
__global__ void __launch_bounds__(plane_threads<N, T>()) fft_inverse_kernel(const ChainArgs c, const FftArgs f) {
    constexpr int NT = plane_threads<N, T>(), S = plane_stride<N>(), R1 = Line<N>::R1, R2 = Line<N>::R2;
    extern __shared__ __align__(16) unsigned char smem[];
    C2<T> *tw = reinterpret_cast<C2<T> *>(smem);
    T *r = reinterpret_cast<T *>(tw + N);
    const int tid = threadIdx.x;
    int z, sys;
    const SpmeGeom &g = geom_of_block<N, T, BATCH>(c, f, N, z, sys);
    for (int k = tid; k < N; k += NT) tw[k] = static_cast<const C2<T> *>(f.tw)[k];
    const C2<T> *in = static_cast<const C2<T> *>(f.half) + g.half_off + (size_t)z * (N / 2 + 1) * N;
    for (int t = tid; t < N / 2 * N; t += NT) {
        const int u = t / N, y = t - u * N;
        int p, q;
        column_of<N>(u, p, q);
        C2<T> v = in[t];
        if (u == 0) {                            // columns 0 and N/2: A + i B
            const C2<T> b = in[N / 2 * N + y];
            v = {v.x - b.y, v.y + b.x};
        }
        r[y * S + p] = v.x;
        r[y * S + q] = v.y;
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R1; t += NT) {
        const int d = t / (N / 2), u = t - d * (N / 2);
        int p, q;
        column_of<N>(u, p, q);
        pass_two<N, true>(r + p, r + q, S, d);
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R2; t += NT) {
        const int b = t / (N / 2), u = t - b * (N / 2);
        int p, q;
        column_of<N>(u, p, q);
        pass_one<N, true>(r + p, r + q, S, b, tw);
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * (N / 2); t += NT) {
        const int j = t / (N / 2), u = t - j * (N / 2);
        if (u == 0) continue;
        int p, q;
        column_of<N>(u, p, q);
        T *r0 = r + 2 * j * S, *r1 = r0 + S;
        const C2<T> a = {r0[p], r0[q]}, b = {r1[p], r1[q]};   // the rows' frequency k
        r0[p] = a.x - b.y;                       // Z(k) = A + i B, Z(N - k) = conj(A) + i conj(B)
        r1[p] = a.y + b.x;
        r0[q] = a.x + b.y;
        r1[q] = b.x - a.y;
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R1; t += NT) {
        const int j = t / R1, q = t - j * R1;
        pass_two<N, true>(r + 2 * j * S, r + (2 * j + 1) * S, 1, q);
    }
    __syncthreads();
    for (int t = tid; t < N / 2 * R2; t += NT) {
        const int j = t / R2, b = t - j * R2;
        pass_one<N, true>(r + 2 * j * S, r + (2 * j + 1) * S, 1, b, tw);
    }
    __syncthreads();
    T *mesh = static_cast<T *>(c.mesh) + g.mesh_off + (size_t)z * N * N;
    for (int t = tid; t < N * N; t += NT) mesh[t] = r[(t / N) * S + t % N];
}

// ---------------------------------------------------------------------------
// The lengths of the workloads in system.py, and 96 between the last two.  Others
// are not built, each being a set of kernels: 72 or 144 would take the radices
// that are there, 40, 56, 80 or 100 one of 5 or 7, and beyond about 150 points
// a plane of 8-byte points (FP64, or two-float FP32) and its stage do not fit
// in the shared memory of an SM.  With cuFFT the FP32C chain takes 78 us at N =
// 4,096, 40^3, order 4, 126 at 24,000, 80^3, order 5, 137 at 40,000, 100^3,
// order 5, where 32^3, 64^3 and 96^3 take 45, 105 and 125 here.
bool fft_own(int K1, int K2, int K3) {
    return K1 == K2 && K2 == K3 && (K1 == 32 || K1 == 48 || K1 == 64 || K1 == 96 || K1 == 128);
}

// frequency at position p of a transformed line
static int freq_at(int N, int p) {
    const int R1 = N == 32 ? 4 : (N == 48 ? 6 : 8), R2 = N / R1;
    return p / R2 + R1 * (p % R2);
}

// Index into a natural half spectrum [kz][ky][kx <= N/2] of element i of the
// transform order [z][column][y].
std::vector<int> fft_order(int N) {
    const int R1 = N == 32 ? 4 : (N == 48 ? 6 : 8), R2 = N / R1, Kh = N / 2 + 1;
    std::vector<int> o((size_t)N * Kh * N);
    size_t i = 0;
    for (int z = 0; z < N; ++z)
        for (int u = 0; u < Kh; ++u) {
            const int kx = u == N / 2 ? N / 2 : u / (R2 / 2) + R1 * (u % (R2 / 2));
            for (int y = 0; y < N; ++y) o[i++] = kx + Kh * (freq_at(N, y) + N * freq_at(N, z));
        }
    return o;
}

// exp(-2 pi i k/N) as N complex values of the precision
int fft_twiddles(int N, bool fp64, void **tw) {
    std::vector<double> d(2 * N);
    for (int k = 0; k < N; ++k) {
        d[2 * k] = std::cos(2.0 * kPi * k / N);
        d[2 * k + 1] = -std::sin(2.0 * kPi * k / N);
    }
    std::vector<float> f(d.begin(), d.end());
    const size_t bytes = 2 * (size_t)N * (fp64 ? sizeof(double) : sizeof(float));
    cudaFree(*tw);
    *tw = nullptr;
    TCP_CUDA(cudaMalloc(tw, bytes));
    TCP_CUDA(cudaMemcpy(*tw, fp64 ? (const void *)d.data() : (const void *)f.data(), bytes, cudaMemcpyHostToDevice));
    return TCP_OK;
}

template <int N, typename T, bool BATCH>
static int convolve_n(const ChainArgs &c, const FftArgs &f, int systems, cudaStream_t st) {
    constexpr int NT = plane_threads<N, T>();
    constexpr bool D = !BATCH && sizeof(T) == 8;
    if (D && c.dipole)
        fft_forward_kernel<N, T, BATCH, D><<<N * systems, NT, plane_bytes<N, T>(c.P, true), st>>>(c, f);
    else
        fft_forward_kernel<N, T, BATCH, false><<<N * systems, NT, plane_bytes<N, T>(c.P), st>>>(c, f);
    fft_z_kernel<N, T, BATCH><<<(N / 2 + 1) * N / kZCols * systems, z_threads<N>(), 0, st>>>(c, f);
    fft_inverse_kernel<N, T, BATCH><<<N * systems, NT, plane_bytes<N, T>(0), st>>>(c, f);
    return 3;
}

template <int N, typename T, bool BATCH>
static int prepare_n(int P) {
    constexpr bool D = !BATCH && sizeof(T) == 8;
    int rc = allow_shared(reinterpret_cast<const void *>(fft_forward_kernel<N, T, BATCH, false>), plane_bytes<N, T>(P));
    if (!rc && D) rc = allow_shared(reinterpret_cast<const void *>(fft_forward_kernel<N, T, BATCH, D>), plane_bytes<N, T>(P, true));
    if (!rc) rc = allow_shared(reinterpret_cast<const void *>(fft_inverse_kernel<N, T, BATCH>), plane_bytes<N, T>(0));
    return rc;
}

#define TCP_FFT_SIZE(N, CALL)          \
    switch (N) {                       \
        case 32: CALL(32); break;      \
        case 48: CALL(48); break;      \
        case 64: CALL(64); break;      \
        case 96: CALL(96); break;      \
        default: CALL(128); break;     \
    }

int fft_energy_parts(int N) { return (N / 2 + 1) * N / kZCols; }

// Spread, transform, influence multiply and inverse transform of `systems`
// meshes of N points a side (a batch's in f.list), phi left in c.mesh.
int fft_convolve(const ChainArgs &c, const FftArgs &f, int N, int systems, cudaStream_t st) {
    int n = 0;
#define TCP_CALL(N)                                                               \
    n = c.many ? convolve_n<N, float, true>(c, f, systems, st)            \
               : (c.fp64 ? convolve_n<N, double, false>(c, f, 1, st) : convolve_n<N, float, false>(c, f, 1, st))
    TCP_FFT_SIZE(N, TCP_CALL)
#undef TCP_CALL
    return n;
}

// shared-memory limits (once, outside any capture)
int fft_prepare(const ChainArgs &c, int N, bool fp64) {
    int rc = TCP_OK;
#define TCP_CALL(N) rc = c.many ? prepare_n<N, float, true>(c.P) : (fp64 ? prepare_n<N, double, false>(c.P) : prepare_n<N, float, false>(c.P))
    TCP_FFT_SIZE(N, TCP_CALL)
#undef TCP_CALL
    return rc;
}

}  // namespace tcp
