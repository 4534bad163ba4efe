// Reconstruction of a batch from its spikes and the templates, and the
// reconstruction's adjoint (lss_recon_forward / lss_recon_backward).
//
// Kilosort subtracts each accepted spike from the batch as
//   Xres[:, x_i + m - nt/2] -= a_i * sum_k U[y_i, k, :] wPCA[k, m]
// (template_matching.py:195-198, the einsum('ijk,jl->kil', U[iY], W) term), so
// the reconstruction is
//   R[c, s] = sum_i a_i sum_k U[y_i, k, c] wPCA[k, s - x_i + nt/2].
// With the assignments (x_i, y_i, a_i) fixed, R is linear in U and in wPCA;
// for an upstream gradient G = dL/dR the adjoint is
//   P_i[k, c]   = sum_m wPCA[k, m] G[c, x_i + m - nt/2]   (the temporal-basis
//                 convolution of G, recomputed per spike: nothing is stored
//                 by the forward pass)
//   dL/dU[t]    = sum_{i: y_i = t} a_i P_i
//   dL/dwPCA    = sum_i a_i sum_c U[y_i, :, c] G[c, x_i + (.) - nt/2]
//   dL/da_i     = sum_{k, c} U[y_i, k, c] P_i[k, c]
// Both passes are deterministic (fixed orders, no atomics). F = float or double
// (the finite-difference checks run the same kernels in FP64).
//
// The backward pass needs each spike's window of G only twice, an element at a
// time: with S_t[c, m] = sum_{i: y_i = t} a_i G[c, x_i + m - nt/2],
//   dL/dU[t]  = wPCA S_t^T,   dL/dwPCA = sum_t U[t] S_t,
//   dL/da_i   = sum_{c, m} (sum_k U[y_i, k, c] wPCA[k, m]) G[c, x_i + m - nt/2],
// so the K-fold contractions are taken once per template instead of per spike.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "lss.h"
#include "lss_kernels.cuh"

namespace lss {

constexpr int RF_CH = 128;     // channels per CTA (four groups of 32, one per warp)
constexpr int RF_THREADS = 256;
constexpr int RF_JC = 4;       // columns per lane
constexpr int RB_THREADS = 512;
constexpr int RB_WARPS = RB_THREADS / 32;
constexpr int RB_SP = 64;      // spikes whose dL/da shares are kept before they are summed over the cluster
constexpr int RB_MAXZ = 8;     // CTAs of a cluster (portable limit)

__device__ __forceinline__ int lower_bound_i(const int32_t* a, int n, int v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// 8 channels by JC columns of sums: += u[c] * b[j], one FMA per term
template <typename F, int JC>
struct Outer {
    F v[8][JC];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
            for (int j = 0; j < JC; ++j) v[c][j] = F(0);
    }
    __device__ __forceinline__ void add(const F* u, const F (&b)[JC]) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
            for (int j = 0; j < JC; ++j) v[c][j] += u[c] * b[j];
    }
    __device__ __forceinline__ F at(int c, int j) const { return v[c][j]; }
};
template <int JC>
struct Outer<float, JC> {  // channels in pairs
    unsigned long long v[4][JC];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int j = 0; j < JC; ++j) v[c][j] = 0ull;
    }
    __device__ __forceinline__ void add(const float* u, const float (&b)[JC]) {
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(u), q = *reinterpret_cast<const ulonglong2*>(u + 4);
#pragma unroll
        for (int j = 0; j < JC; ++j) {
            unsigned long long bb;
            asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(b[j]));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[0][j]) : "l"(p.x), "l"(bb));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[1][j]) : "l"(p.y), "l"(bb));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[2][j]) : "l"(q.x), "l"(bb));
            asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v[3][j]) : "l"(q.y), "l"(bb));
        }
    }
    __device__ __forceinline__ float at(int c, int j) const {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v[c / 2][j]));
        return c % 2 ? b : a;
    }
};

// R[c, col] by the definition, over the spikes [lo, hi), none of which adds to a
// column outside its window.
template <typename F>
__device__ __noinline__ F recon_one(const F* __restrict__ U, const F* __restrict__ W, int K, int C, int nt,
                                    const int32_t* __restrict__ xs, const int32_t* __restrict__ ys,
                                    const F* __restrict__ as, int lo, int hi, int c, int64_t col) {
    F acc = F(0);
    for (int i = lo; i < hi; ++i) {
        const int64_t m = col - xs[i] + nt / 2;
        if (m < 0 || m >= nt) continue;
        F w = F(0);
        for (int k = 0; k < K; ++k) w += U[((int64_t)ys[i] * K + k) * C + c] * W[k * nt + m];
        acc += as[i] * w;
    }
    return acc;
}

// xs/ys/as: spikes sorted by x. A warp owns 32 columns of 32 channels, a lane 8
// channels by 4 columns (8 apart) in registers, and takes the tile's spikes in time
// order, skipping the ones whose window misses its columns:
// acc[c, s] += U[y, k, c] * (a W[k, m]). U rows of SP spikes at a time are copied to
// shared memory while the SP before them are added, W is staged once with 32 zeros
// on either side. Shared memory returns 128 bytes per cycle to a warp also where
// lanes read the same value: 8 x 4 outputs take 12 cycles of it beside 8 of FMAs (in
// pairs of channels for floats); one column by 32 channels took 32 beside 8.
// 9000 spikes at 384 channels x 60000 samples are 2.5 GFLOP that must be done and
// 3.9 GFLOP done (a window covers 61 of the 92 columns it is taken over), over 92 MB
// written: 180 us, against 296 us with one column per lane and 232 us with 8 x 8
// outputs (two CTAs per SM instead of three, 61 of 124 columns).
// The zeros beside W are no zeros beside an infinite or NaN amplitude or template
// value: a sum that is not finite at the end is taken again by the definition.
template <typename F, int SP>
__global__ void __launch_bounds__(RF_THREADS, sizeof(F) == 4 ? 3 : 1)
    k_recon_fwd(const F* __restrict__ U, const F* __restrict__ W, int K, int C, int nt, const int32_t* __restrict__ xs,
                const int32_t* __restrict__ ys, const F* __restrict__ as, int n, F* __restrict__ R, int64_t N) {
    constexpr int JC = RF_JC, CW = 8 * JC, COLS = 2 * CW;     // a warp's columns, the CTA's
    extern __shared__ __align__(16) unsigned char rf_smem[];
    F* Us = reinterpret_cast<F*>(rf_smem);        // [2][SP][K][RF_CH]
    F* Ws = Us + 2 * SP * K * RF_CH;               // [K][nt + 2 CW]
    __shared__ int s_x[2][SP];
    __shared__ F s_a[2][SP];
    const int h = nt / 2, wp = nt + 2 * CW;
    const int64_t t0 = (int64_t)blockIdx.x * COLS;
    const int c0 = blockIdx.y * RF_CH;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wc = (warp >> 1) * 32 + (lane >> 3) * 8;     // the lane's channels, from c0
    const int64_t w0 = t0 + (warp & 1) * CW;               // the warp's first column
    const int64_t col = w0 + (lane & 7);                   // the lane's
    const bool on = c0 + (warp >> 1) * 32 < C && w0 < N;
    for (int e = threadIdx.x; e < K * wp; e += RF_THREADS) {
        const int k = e / wp, m = e % wp - CW;
        Ws[e] = (m >= 0 && m < nt) ? W[k * nt + m] : F(0);
    }
    // spikes whose window [x - h, x - h + nt) meets [t0, t0 + COLS)
    const int lo = lower_bound_i(xs, n, (int)(t0 - (nt - 1 - h)));
    const int hi = lower_bound_i(xs, n, (int)(t0 + COLS + h));
    Outer<F, JC> acc;
    acc.clear();
    // SP spikes from i0 on: a warp per row (spike, component) of U, copied asynchronously (past C: zeros)
    auto stage = [&](int i0, int buf) {
        const int ns = min(SP, hi - i0);
        for (int row = warp; row < ns * K; row += RF_THREADS / 32) {
            const int q = row / K;
            const F* src = U + ((int64_t)ys[i0 + q] * K + (row - q * K)) * C;
            F* dst = Us + (buf * SP * K + row) * RF_CH;
#pragma unroll
            for (int c = lane; c < RF_CH; c += 32) {
                const bool in = c0 + c < C;
                asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(dst + c)),
                             "l"(src + (in ? c0 + c : 0)), "n"((int)sizeof(F)), "r"(in ? (int)sizeof(F) : 0)
                             : "memory");
            }
        }
        if (threadIdx.x < ns) {
            s_x[buf][threadIdx.x] = xs[i0 + threadIdx.x];
            s_a[buf][threadIdx.x] = as[i0 + threadIdx.x];
        }
    };
    if (lo < hi) stage(lo, 0);
    int buf = 0;
    for (int i0 = lo; i0 < hi; i0 += SP, buf ^= 1) {
        const int ns = min(SP, hi - i0);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();  // the group is there; the one before it has been added, its buffer is free
        if (i0 + SP < hi) stage(i0 + SP, buf ^ 1);
        if (!on) continue;
        for (int q = 0; q < ns; ++q) {
            const int64_t d = w0 - s_x[buf][q] + h;        // lag of the warp's first column
            if (d <= -CW || d >= nt) continue;
            const F a = s_a[buf][q];
            const F* wq = Ws + (int)d + CW + (lane & 7);
            const F* uq = Us + (buf * SP + q) * K * RF_CH + wc;
            for (int k = 0; k < K; ++k) {
                F b[JC];
#pragma unroll
                for (int j = 0; j < JC; ++j) b[j] = a * wq[k * wp + 8 * j];
                acc.add(uq + k * RF_CH, b);
            }
        }
    }
    if (on) {
        F* out = R + (int64_t)(c0 + wc) * N + col;
        F z = F(0);  // NaN once an output is not finite
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
            for (int j = 0; j < JC; ++j)
                if (c0 + wc + c < C && col + 8 * j < N) {
                    const F v = acc.at(c, j);
                    out[(int64_t)c * N + 8 * j] = v;
                    z += F(0) * v;
                }
        if (z != F(0)) {
#pragma unroll 1
            for (int e = 0; e < 8 * JC; ++e) {
                const int c = e / JC, j = e % JC;
                if (c0 + wc + c >= C || col + 8 * j >= N) continue;
                F* p = out + (int64_t)c * N + 8 * j;
                if (!isfinite(*p)) *p = recon_one(U, W, K, C, nt, xs, ys, as, lo, hi, c0 + wc + c, col + 8 * j);
            }
        }
    }
}


// A template's gradients again where the sums over its spikes were NaN: by the
// definition, which contracts a spike's window before its amplitude is taken (an
// infinite amplitude times a window of both signs is a NaN in S_t, and an infinite
// gradient). A sum that turns NaN here too is not taken further. One CTA; 0.8 us of the
// backward pass below when nothing is redone.
template <typename F>
__device__ __noinline__ void redo_nan(const F* __restrict__ U, const F* __restrict__ W, int K, int C, int nt,
                                      const int32_t* __restrict__ x, const F* __restrict__ amp,
                                      const int32_t* __restrict__ order, const int32_t* __restrict__ tstart,
                                      const F* __restrict__ G, int64_t N, F* dU, F* Qt, F* damp, int t) {
    const int j0 = tstart[t], j1 = tstart[t + 1];
    auto g = [&](int i, int c, int m) {  // G in spike i's window
        const int64_t s = (int64_t)x[i] + m - nt / 2;
        return s >= 0 && s < N ? G[(int64_t)c * N + s] : F(0);
    };
    auto dot = [&](int i, int k, int c) {  // P_i[k, c]
        F p = F(0);
        for (int m = 0; m < nt && p == p; ++m) p += W[k * nt + m] * g(i, c, m);
        return p;
    };
    const F* Ut = U + (int64_t)t * K * C;
    for (int e = threadIdx.x; e < K * C; e += RB_THREADS) {
        F* p = dU + (int64_t)t * K * C + e;
        if (*p == *p) continue;
        F v = F(0);
        for (int j = j0; j < j1 && v == v; ++j) v += amp[order[j]] * dot(order[j], e / C, e % C);
        *p = v;
    }
    for (int e = threadIdx.x; e < K * nt; e += RB_THREADS) {
        F* p = Qt + (int64_t)t * K * nt + e;
        if (*p == *p) continue;
        F v = F(0);
        for (int j = j0; j < j1 && v == v; ++j) {
            F q = F(0);
            for (int c = 0; c < C && q == q; ++c) q += Ut[e / nt * C + c] * g(order[j], c, e % nt);
            v += amp[order[j]] * q;
        }
        *p = v;
    }
    const int lane = threadIdx.x & 31;
    for (int j = j0 + threadIdx.x / 32; damp && j < j1; j += RB_WARPS) {  // a warp per spike
        F* p = damp + order[j];
        if (*p == *p) continue;
        F v = F(0);
        for (int e = lane; e < K * C && v == v; e += 32) v += Ut[e] * dot(order[j], e / C, e % C);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) *p = v;
    }
}

// A cluster of Z CTAs per template t; order[tstart[t] .. tstart[t+1]) are its
// spikes. CTA z takes channel chunks z, z + Z, ...: a warp's channels w + 16 j (j <
// CJ), lags lane + 32u (u < NM) of a window in registers, S and the template's
// waveform beside them, so a spike costs one coalesced read and two FMAs per
// element; a spike's window is fetched while the one before it is added. The
// clusters' shared memories are then summed in rank order. 9000 spikes x 384
// channels x 61 samples are 843 MB of windows (the 92 MB gradient stays in L2), read
// and added in 270 us; 470 us with 8 warps per CTA, no window ahead and a check per
// element.
template <typename F, int NM>
__global__ void __launch_bounds__(RB_THREADS, sizeof(F) == 4 ? 2 : 1) k_recon_bwd(const F* __restrict__ U, const F* __restrict__ W, int K,
                                                          int C, int nt, const int32_t* __restrict__ x,
                                                          const F* __restrict__ amp, const int32_t* __restrict__ order,
                                                          const int32_t* __restrict__ tstart, const F* __restrict__ G,
                                                          int64_t N, F* __restrict__ dU, F* __restrict__ Qt,
                                                          F* __restrict__ damp) {
    constexpr int CJ = 8 / NM, CH = RB_WARPS * CJ;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char rb_smem[];
    const int ntp = nt | 1;
    F* Ws = reinterpret_cast<F*>(rb_smem);        // [K][nt]
    F* Us = Ws + K * nt;                           // [K][CH]  U[t] of the chunk
    F* S = Us + K * CH;                            // [CH][ntp]
    F* Qp = S + CH * ntp;                          // [K][nt] this CTA's share of U[t] S_t
    F* red = Qp + K * nt;                          // [RB_SP][RB_WARPS] shares of dL/da_i by warp
    __shared__ int s_i[RB_SP], s_x[RB_SP];
    __shared__ F s_a[RB_SP];
    const int Z = (int)cl.num_blocks(), z = (int)cl.block_rank();
    const int t = blockIdx.x / Z;
    const int h = nt / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int e = threadIdx.x; e < K * nt; e += RB_THREADS) {
        Ws[e] = W[e];
        Qp[e] = F(0);
    }
    const int j0 = tstart[t], j1 = tstart[t + 1];
    const int nchunk = (C + CH - 1) / CH;
    for (int it = 0; it * Z < nchunk; ++it) {
        const int c0 = (it * Z + z) * CH;  // past C: the CTA only takes part in the sums
        __syncthreads();
        for (int e = threadIdx.x; e < K * CH; e += RB_THREADS) {
            const int k = e / CH, c = e % CH;
            Us[e] = (c0 + c < C) ? U[((int64_t)t * K + k) * C + c0 + c] : F(0);
        }
        __syncthreads();
        F s[CJ][NM], wv[CJ][NM];
#pragma unroll
        for (int j = 0; j < CJ; ++j)
#pragma unroll
            for (int u = 0; u < NM; ++u) {
                const int m = lane + 32 * u;
                F v = F(0);
                if (m < nt)
                    for (int k = 0; k < K; ++k) v += Us[k * CH + warp + RB_WARPS * j] * Ws[k * nt + m];
                wv[j][u] = v;
                s[j][u] = F(0);
            }
        for (int b0 = j0; b0 < j1; b0 += RB_SP) {
            const int nb = min(RB_SP, j1 - b0);
            __syncthreads();
            if (threadIdx.x < nb) {
                const int i = order[b0 + threadIdx.x];
                s_i[threadIdx.x] = i;
                s_x[threadIdx.x] = x[i];
                s_a[threadIdx.x] = amp[i];
            }
            __syncthreads();
            // spike q's window of G in this warp's rows
            auto load = [&](int q, F (&v)[CJ][NM]) {
                if (q >= nb) return;
                const int64_t x0 = (int64_t)s_x[q] - h;
                const F* g = G + (int64_t)(c0 + warp) * N + x0 + lane;
                if (x0 >= 0 && x0 + nt <= N && c0 + CH <= C) {
#pragma unroll
                    for (int j = 0; j < CJ; ++j, g += RB_WARPS * N)
#pragma unroll
                        for (int u = 0; u < NM; ++u) v[j][u] = lane + 32 * u < nt ? __ldg(g + 32 * u) : F(0);
                } else {
#pragma unroll
                    for (int j = 0; j < CJ; ++j, g += RB_WARPS * N)
#pragma unroll
                        for (int u = 0; u < NM; ++u) {
                            const int64_t p = x0 + lane + 32 * u;
                            const bool in = lane + 32 * u < nt && c0 + warp + RB_WARPS * j < C && p >= 0 && p < N;
                            v[j][u] = in ? __ldg(g + 32 * u) : F(0);
                        }
                }
            };
            // what it adds to the window sums; this lane's share of dL/da
            auto add = [&](int q, const F (&v)[CJ][NM]) {
                const F a = s_a[q];
                F d = F(0);
#pragma unroll
                for (int j = 0; j < CJ; ++j)
#pragma unroll
                    for (int u = 0; u < NM; ++u) {
                        s[j][u] += a * v[j][u];
                        d += wv[j][u] * v[j][u];
                    }
                return d;
            };
            F va[CJ][NM], vb[CJ][NM];  // the next spike's window is on its way while one is added
            load(0, va);
            for (int q = 0; q < nb; q += 2) {
                load(q + 1, vb);
                const F da = add(q, va);
                load(q + 2, va);
                const F db = q + 1 < nb ? add(q + 1, vb) : F(0);
                if (damp) {  // both sums over the lanes: the lower half of the warp takes the first
                    F d = (lane & 16 ? db : da) + __shfl_xor_sync(0xffffffffu, lane & 16 ? da : db, 16);
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
                    if ((lane & 15) == 0 && q + (lane >> 4) < nb) red[(q + (lane >> 4)) * RB_WARPS + warp] = d;
                }
            }
            if (damp) {
                // dL/da_i: over ranks and warps in order; later chunks add on
                cl.sync();
                if (z == 0 && threadIdx.x < nb) {
                    F d = it ? damp[s_i[threadIdx.x]] : F(0);
                    for (int r = 0; r < Z; ++r) {
                        const F* rr = cl.map_shared_rank(red, r) + threadIdx.x * RB_WARPS;
                        for (int w = 0; w < RB_WARPS; ++w) d += rr[w];
                    }
                    damp[s_i[threadIdx.x]] = d;
                }
                cl.sync();
            }
        }
#pragma unroll
        for (int j = 0; j < CJ; ++j)
#pragma unroll
            for (int u = 0; u < NM; ++u)
                if (lane + 32 * u < nt) S[(warp + RB_WARPS * j) * ntp + lane + 32 * u] = s[j][u];
        __syncthreads();
        for (int e = threadIdx.x; e < K * CH; e += RB_THREADS) {
            const int k = e / CH, c = e % CH;
            if (c0 + c >= C) continue;
            F v = F(0);
            for (int m = 0; m < nt; ++m) v += Ws[k * nt + m] * S[c * ntp + m];
            dU[((int64_t)t * K + k) * C + c0 + c] = v;
        }
        for (int e = threadIdx.x; e < K * nt; e += RB_THREADS) {
            const int k = e / nt, m = e % nt;
            F v = F(0);
            for (int c = 0; c < CH; ++c) v += Us[k * CH + c] * S[c * ntp + m];
            Qp[e] += v;
        }
    }
    cl.sync();
    bool odd = false;
    if (z == 0)
        for (int e = threadIdx.x; e < K * nt; e += RB_THREADS) {
            F v = F(0);
            for (int r = 0; r < Z; ++r) v += cl.map_shared_rank(Qp, r)[e];
            Qt[(int64_t)t * K * nt + e] = v;
            odd |= !isfinite(v);
        }
    cl.sync();  // the other ranks' shared memory is read until here
    // (what is not finite in S_t or in the template is in Qt, which sums over all channels)
    if (z == 0 && __syncthreads_or(odd)) redo_nan(U, W, K, C, nt, x, amp, order, tstart, G, N, dU, Qt, damp, t);
}

// dW[e] = sum_t Qt[t, e]: 32 columns per CTA, the templates strided over 8 rows
// of threads, whose sums are combined in order
template <typename F>
__global__ void __launch_bounds__(256) k_reduce_templates(const F* __restrict__ Qt, int T, int KN, F* __restrict__ dW) {
    __shared__ F part[8][32];
    const int e = blockIdx.x * 32 + threadIdx.x;
    F s = F(0);
    if (e < KN)
        for (int t = threadIdx.y; t < T; t += 8) s += Qt[(int64_t)t * KN + e];
    part[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && e < KN) {
        for (int r = 1; r < 8; ++r) s += part[r][threadIdx.x];
        dW[e] = s;
    }
}

template <typename F>
static cudaError_t recon_fwd(const void* U, const void* W, int K, int C, int nt, const int32_t* xs, const int32_t* ys,
                             const void* as, int n, void* R, int64_t N, cudaStream_t s) {
    constexpr int SP = sizeof(F) == 4 ? 8 : 4, COLS = 16 * RF_JC;
    const size_t smem = sizeof(F) * ((size_t)2 * SP * K * RF_CH + (size_t)K * (nt + COLS));
    const cudaError_t e = allow_shared_memory<k_recon_fwd<F, SP>>();
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((N + COLS - 1) / COLS), (unsigned)((C + RF_CH - 1) / RF_CH));
    k_recon_fwd<F, SP><<<grid, RF_THREADS, smem, s>>>(static_cast<const F*>(U), static_cast<const F*>(W), K, C, nt, xs,
                                                      ys, static_cast<const F*>(as), n, static_cast<F*>(R), N);
    return cudaGetLastError();
}

// NM: lags per lane (ceil(nt / 32) rounded up to a power of two)
template <typename F, int NM>
static cudaError_t recon_bwd_nm(const F* U, const F* W, int T, int K, int C, int nt, const int32_t* x, const F* amp,
                                const int32_t* order, const int32_t* tstart, const F* G, int64_t N, F* dU, F* work,
                                F* damp, cudaStream_t s) {
    constexpr int CH = RB_WARPS * (8 / NM);
    const size_t smem = sizeof(F) * (2 * (size_t)K * nt + (size_t)K * CH + (size_t)CH * (nt | 1) + RB_SP * RB_WARPS);
    // (always: with the static arrays a size just below 48 KB needs it too)
    const cudaError_t e = allow_shared_memory<k_recon_bwd<F, NM>>();
    if (e != cudaSuccess) return e;
    const int Z = std::min(RB_MAXZ, (C + CH - 1) / CH);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)T * (unsigned)Z);
    lc.blockDim = dim3(RB_THREADS);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)Z;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_recon_bwd<F, NM>, U, W, K, C, nt, x, amp, order, tstart, G, N, dU, work, damp);
}

template <typename F>
static cudaError_t recon_bwd(const void* U, const void* W, int T, int K, int C, int nt, const int32_t* x,
                             const void* amp, const int32_t* order, const int32_t* tstart, const void* G, int64_t N,
                             void* dU, void* dW, void* damp, void* work, cudaStream_t s) {
    // channels and components are bounded as the shared memory of one CTA per template would bound them
    if (sizeof(F) * (2 * (size_t)K * nt + 2 * (size_t)K * C + (size_t)32 * (nt + 1) + 256) > 227 * 1024)
        return cudaErrorInvalidValue;
    auto run = [&](auto kind) {
        return recon_bwd_nm<F, decltype(kind)::value>(
            static_cast<const F*>(U), static_cast<const F*>(W), T, K, C, nt, x, static_cast<const F*>(amp), order, tstart,
            static_cast<const F*>(G), N, static_cast<F*>(dU), static_cast<F*>(work), static_cast<F*>(damp), s);
    };
    const cudaError_t e = nt <= 32    ? run(std::integral_constant<int, 1>())
                          : nt <= 64  ? run(std::integral_constant<int, 2>())
                          : nt <= 128 ? run(std::integral_constant<int, 4>())
                                      : run(std::integral_constant<int, 8>());
    if (e != cudaSuccess) return e;
    const int KN = K * nt;
    k_reduce_templates<F><<<(KN + 31) / 32, dim3(32, 8), 0, s>>>(static_cast<const F*>(work), T, KN, static_cast<F*>(dW));
    return cudaGetLastError();
}

}  // namespace lss

using namespace lss;

static int recon_args_ok(int32_t dtype, int32_t T, int32_t K, int32_t C, int32_t nt, int64_t n, int64_t N) {
    if (dtype != 0 && dtype != 1) return 0;
    if (T <= 0 || K <= 0 || K > 16 || C <= 0 || nt <= 0 || nt > 255 || n < 0 || n > INT32_MAX || N <= 0) return 0;
    return 1;
}

extern "C" {

int lss_recon_forward(int32_t dtype, const void* U, const void* wPCA, int32_t T, int32_t K, int32_t C, int32_t nt,
                      const int32_t* x_sorted, const int32_t* y, const void* amp, int64_t n, void* R, int64_t N,
                      void* stream) {
    if (!recon_args_ok(dtype, T, K, C, nt, n, N) || !U || !wPCA || !R || (n > 0 && (!x_sorted || !y || !amp))) {
        lss::set_thread_error("lss_recon_forward: bad argument");
        return LSS_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const cudaError_t e = dtype == 0 ? recon_fwd<float>(U, wPCA, K, C, nt, x_sorted, y, amp, (int)n, R, N, s)
                                     : recon_fwd<double>(U, wPCA, K, C, nt, x_sorted, y, amp, (int)n, R, N, s);
    if (e != cudaSuccess) {
        lss::set_thread_error(cudaGetErrorString(e));
        return LSS_ERR_CUDA;
    }
    return LSS_OK;
}

int lss_recon_backward(int32_t dtype, const void* U, const void* wPCA, int32_t T, int32_t K, int32_t C, int32_t nt,
                       const int32_t* x, const void* amp, const int32_t* order_by_template,
                       const int32_t* template_start, const void* dR, int64_t N, void* dU, void* dwPCA, void* damp,
                       void* work, void* stream) {
    if (!recon_args_ok(dtype, T, K, C, nt, 0, N) || !U || !wPCA || !x || !amp || !order_by_template ||
        !template_start || !dR || !dU || !dwPCA || !work) {
        lss::set_thread_error("lss_recon_backward: bad argument");
        return LSS_ERR_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const cudaError_t e =
        dtype == 0 ? recon_bwd<float>(U, wPCA, T, K, C, nt, x, amp, order_by_template, template_start, dR, N, dU,
                                      dwPCA, damp, work, s)
                   : recon_bwd<double>(U, wPCA, T, K, C, nt, x, amp, order_by_template, template_start, dR, N, dU,
                                       dwPCA, damp, work, s);
    if (e != cudaSuccess) {
        lss::set_thread_error(cudaGetErrorString(e));
        return LSS_ERR_CUDA;
    }
    return LSS_OK;
}

}  // extern "C"
