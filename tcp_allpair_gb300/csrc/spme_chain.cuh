// spme_chain.cuh -- binning of the SPME chain: the part that runs where the
// positions are written (the half-kick kernels of integrate.cu and batch.cu)
// and the types its other kernels (spme_chain.cu) share.
#pragma once

#include "device_util.cuh"
#include "spme_math.cuh"
#include "tcp_internal.h"

namespace tcp {

constexpr int kPartBlock = 64;                   // particles per CTA of the kernels with a thread per component
constexpr int kPartThreads = 3 * kPartBlock;     // thread d kPartBlock + k: component d of particle k
constexpr int kScanTail = 3072;                  // bins that the last CTA of the binning kernel scans itself (one round)

// True in the last CTA of the grid to get here, after every other CTA's
// earlier writes; the ticket is left at zero for the next launch.
__device__ __forceinline__ bool last_block(unsigned *ticket) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        if (last) *ticket = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Mesh coordinate of component d of a particle (force.f90:700-702): the first
// mesh index of its support, wrapped, and the argument of its spline weights
// (z = INT(u) - u + 1 for order 4, whose cubics the reference writes in z;
// u - INT(u) otherwise).
__device__ __forceinline__ int bin_axis(double x, double hL, double KL, int K, int P, double &arg) {
    const double u = (x + hL) * KL;
    const int iu = (int)u;
    arg = P == 4 ? ((double)iu - u) + 1.0 : u - (double)iu;
    return wrapi(iu - (P - 3), K);
}

// Exclusive prefix sum of count[0..nbins) into start[0..nbins] by one CTA;
// the counts are left at zero for the next binning.  Sixteen bins per thread
// and round (count is padded to whole rounds).
__device__ __forceinline__ void scan_bins(const SpreadBins &b, int nbins) {
    __shared__ int ws[32];
    __shared__ int carry;
    const int nt = blockDim.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    for (int c0 = 0; c0 < nbins; c0 += 16 * nt) {
        int4 *c = reinterpret_cast<int4 *>(b.count + c0 + 16 * threadIdx.x);
        int n[16];
#pragma unroll
        for (int k = 0; k < 4; ++k) *reinterpret_cast<int4 *>(n + 4 * k) = __ldcg(c + k);
        int v = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) v += n[k];
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = make_int4(0, 0, 0, 0);
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        __syncthreads();                         // ws and carry of the round before are read
        if (lane == 31) ws[w] = x;
        __syncthreads();
        int at = carry + x - v;
        for (int k = 0; k < w; ++k) at += ws[k];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int bin = c0 + 16 * threadIdx.x + k;
            if (bin < nbins) b.start[bin] = at;
            at += n[k];
        }
        __syncthreads();
        if (threadIdx.x == nt - 1) carry = at;
    }
    __syncthreads();
    if (threadIdx.x == 0) b.start[nbins] = carry;
}

// Bin and spline arguments of one particle from its three base indexes.
template <typename T>
__device__ __forceinline__ void bin_store(const SpreadBins &b, int m, int n, const double *arg, double q, int bx, int by,
                                          int bz, int K2, int bin_off) {
    const int bin = bin_off + by + K2 * bz;
    b.rank[m] = atomicAdd(&b.count[bin], 1);
    b.bin[m] = bin;
    b.base_m[m] = make_int4(bx, by, bz, 0);
    T *a = static_cast<T *>(b.arg);
    for (int d = 0; d < 3; ++d) a[(size_t)d * n + m] = (T)arg[d];
    static_cast<T *>(b.q_m)[m] = (T)q;
}

// Spread into the mesh rows y0 .. y0 + nrow - 1 of plane z, held in shared
// memory by the threads of one group (warps `warp0` .. of the CTA, NG threads,
// named barrier `bar`; the whole CTA where there is one group).  For each jz =
// jz0, jz0 + jzs, .. the particles of plane z - jz whose support reaches the
// rows -- at most two runs of the sorted list -- are staged in shared memory,
// kStage (or half that) at a time, with their factors q W_z W_y; then P lanes own one row and
// walk its particles, lane l adding the point bx + l: no two lanes ever add to
// one point, and every point is summed in the same order (jz, bin, particle)
// on every call.  hi, and lo in FP32, hold the rows (cleared by the caller;
// row r at r * stride): FP32C mode sums in two-float FP32 (TwoSum hi/lo, about
// 48 bits), FP64 mode in FP64.
//
// Bound: the latency of a visit (a particle's turn in a row, about 80 cycles
// from shared memory, P^2 of them per particle) and instruction issue, about
// 20 instructions a visit of 32/P rows.
constexpr int kStage = 256;
constexpr int kStageBins = 136;          // bins that reach one CTA's rows: at most 128 (a plane) or rows + P - 1
template <typename T>
struct StageBuf {
    T *w;                // [kStage][2 P]: W_x, then q W_z W_y (dipoles: [kStage][4 P], W_x, W_x', then their factors)
    int *bx;             // [kStage] base x, and base y as the number of its bin among those of run (bits 24 and up)
    int2 *run;           // [kStageBins] list range of each bin
};
template <typename T>
__host__ __device__ constexpr size_t stage_bytes(int P, bool dipole = false) {
    return (dipole ? kStage / 2 : kStage) * ((dipole ? 4 : 2) * (size_t)P * sizeof(T) + sizeof(int)) + kStageBins * sizeof(int2);
}
template <typename T>
__device__ __forceinline__ StageBuf<T> stage_at(void *p, int P) {
    StageBuf<T> s;
    s.run = static_cast<int2 *>(p);
    s.w = reinterpret_cast<T *>(s.run + kStageBins);
    s.bx = reinterpret_cast<int *>(s.w + kStage * 2 * P);   // half as many dipoles, twice the factors
    return s;
}

__device__ __forceinline__ void group_sync(int bar, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory");
}

// DIP: the mesh dipole grad W . c.dipole of every particle (K/L times the index
// derivatives) instead of its charge.
template <int P, typename T, int NG, bool DIP = false>
__device__ __forceinline__ void chain_rows(const ChainArgs &c, const SpmeGeom &g, int z, int y0, int nrow, T *hi,
                                           float *lo, int stride, const StageBuf<T> &st, int tid, int bar, int jz0,
                                           int jzs) {
    constexpr bool F32 = sizeof(T) == 4;
    constexpr int RG = 32 / P, ST = DIP ? kStage / 2 : kStage;
    const int K1 = g.K[0], K2 = g.K[1], K3 = g.K[2];
    const int lane = tid & 31, grp = lane / P, l = lane - grp * P;
    const unsigned mask = ((1u << P) - 1u) << (grp * P);
    const T *ew = static_cast<const T *>(c.b.ew), *eq = static_cast<const T *>(c.b.q);
    const int nb = min(nrow + P - 1, K2), blo = nb == K2 ? 0 : y0 - P + 1;   // bins blo .. blo + nb - 1
    for (int jz = jz0; jz < P; jz += jzs) {
        const int bz = z - jz < 0 ? z - jz + K3 : z - jz;
        const int *start = c.b.start + g.bin_off + K2 * bz;
        group_sync(bar, NG);                     // the rows are cleared, the last stage is read
        for (int k = tid; k < nb; k += NG) {
            const int b = blo + k < 0 ? blo + k + K2 : blo + k;
            st.run[k] = make_int2(start[b], start[b + 1]);
        }
        for (int piece = blo < 0 ? 0 : 1; piece < 2; ++piece) {
            const int q0 = start[piece ? max(blo, 0) : blo + K2], q1 = start[piece ? blo + nb : K2];
            for (int c0 = q0; c0 < q1; c0 += ST) {
                const int cn = min(ST, q1 - c0);
                if (c0 != q0 || piece) group_sync(bar, NG);   // the chunk before is read
                for (int e = tid; e < cn; e += NG) {
                    const T *w = ew + (size_t)(c0 + e) * 6 * P;
                    T *o = st.w + e * (DIP ? 4 : 2) * P;
                    if (DIP) {
                        const int m = c.b.order[c0 + e];
                        const T q = eq[c0 + e], wz = w[4 * P + jz], dz = w[5 * P + jz];
                        const T vx = q * (T)(c.dipole[m] * g.KL[0]) * wz;
                        const T vy = q * (T)(c.dipole[(size_t)c.n + m] * g.KL[1]) * wz;
                        const T vz = q * (T)(c.dipole[2 * (size_t)c.n + m] * g.KL[2]) * dz;
#pragma unroll
                        for (int j = 0; j < P; ++j) {
                            o[j] = w[j];
                            o[P + j] = w[P + j];
                            o[2 * P + j] = vy * w[3 * P + j] + vz * w[2 * P + j];
                            o[3 * P + j] = vx * w[2 * P + j];
                        }
                    } else {
                        const T qz = eq[c0 + e] * w[4 * P + jz];
#pragma unroll
                        for (int j = 0; j < P; ++j) {
                            o[j] = w[j];
                            o[P + j] = qz * w[2 * P + j];
                        }
                    }
                    const int4 base = c.b.base[c0 + e];
                    const int ybin = base.y - blo >= K2 ? base.y - blo - K2 : base.y - blo;
                    st.bx[e] = (int)((unsigned)ybin << 24) | base.x;
                }
                group_sync(bar, NG);
                if (grp < RG)
                    for (int r = (tid >> 5) * RG + grp; r < nrow; r += NG / 32 * RG) {
                        // this row's bins, y - P + 1 .. y, are one or two runs of the list
                        const int y = y0 + r, ylo = y - P + 1;
                        T *h = hi + (size_t)r * stride;
                        float *lw = lo + (size_t)r * stride;
                        for (int half = ylo < 0 ? 0 : 1; half < 2; ++half) {
                            const int b0 = half ? max(ylo, 0) : ylo + K2, b1 = half ? y : K2 - 1;
                            const int i0 = b0 - blo - (b0 - blo >= K2 ? K2 : 0), i1 = b1 - blo - (b1 - blo >= K2 ? K2 : 0);
                            const int e0 = max(st.run[i0].x - c0, 0), e1 = min(st.run[i1].y - c0, cn);
                            if (e0 >= e1) continue;
                            int pk = st.bx[e0];
#pragma unroll 1
                            for (int e = e0; e < e1; ++e) {
                                const int nx = st.bx[min(e + 1, e1 - 1)];
                                int jy = y - blo - (int)((unsigned)pk >> 24);
                                jy += jy < 0 ? K2 : 0;
                                int x = (pk & 0xffffff) + l;
                                x -= x >= K1 ? K1 : 0;
                                const T *w = st.w + e * (DIP ? 4 : 2) * P;
                                const T v = w[(DIP ? 2 : 1) * P + jy], wx = w[l];
                                if (DIP) {
                                    h[x] = fma(v, wx, fma(w[3 * P + jy], w[P + l], h[x]));
                                } else if (F32) {
                                    const T u = v * wx, a = h[x], s = a + u, bp = s - a;
                                    lw[x] += (float)((a - (s - bp)) + (u - bp));
                                    h[x] = s;
                                } else {
                                    h[x] = fma(v, wx, h[x]);
                                }
                                pk = nx;
                                __syncwarp(mask);   // the next particle's lanes may read this point
                            }
                        }
                    }
            }
        }
    }
}

}  // namespace tcp
