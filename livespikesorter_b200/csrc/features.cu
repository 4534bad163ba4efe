// Residual, PC features and spike records of one batch.
//
// * Xres = X minus every accepted spike's waveform, applied in the order the
//   reference applies them (round by round; within a round the +-nt/2
//   windows of distinct peaks never overlap): template_matching.py:197.
// * PC features xfeat[i, j, k] = sum_m Xres[iCC[j, iU[y_i]], x_i + m - nt/2]
//   * wPCA[k, m] + amp_i * Ucc[j, y_i, k]: template_matching.py:50-51
//   (compute_xfeat_kernel, OnlineSpikesV2.cu:112-187, which indexes the
//   residual as [n, C] although it is stored [C, n]; this follows Kilosort).
// * records: time = (x - nt) + ibatch*NT - nt/2 + nt0min, dropping negative
//   times of batch 0 (template_matching.py:53-68), in run_matching order.
#include "lss_kernels.cuh"
#include "mp_common.cuh"

#include <algorithm>
#include <climits>

namespace lss {

// projection-row element as float: the FP32 path's tf32 parts or the BF16
// path's bf16 parts (hi + lo is the projection to 2^-23 or 2^-17 relative)
__device__ __forceinline__ float pval(const float* p) { return *p; }
__device__ __forceinline__ float pval(const __nv_bfloat16* p) { return __bfloat162float(*p); }

constexpr int XR_COLS = 128;
constexpr int XR_CH = 32;
constexpr int XR_LIST_MAX = 1024;

__global__ void __launch_bounds__(XR_COLS) k_xres(const float* __restrict__ X, int64_t ldx, int32_t C, int32_t N,
                                                  int32_t nt, const float* __restrict__ wave,
                                                  const int32_t* __restrict__ sp_x,
                                                  const int32_t* __restrict__ sp_y,
                                                  const float* __restrict__ sp_amp,
                                                  const int32_t* __restrict__ round_start, int32_t rounds,
                                                  float* __restrict__ Xres, int64_t ldr, int32_t* status) {
    __shared__ int l_x[XR_LIST_MAX], l_y[XR_LIST_MAX];
    __shared__ float l_a[XR_LIST_MAX];
    __shared__ int r_cnt[XR_COLS], r_off[XR_COLS + 1];
    const int h = nt / 2;
    const int s0 = blockIdx.x * XR_COLS;
    const int wlo = s0 - h, whi = s0 + XR_COLS - 1 + h;
    int nlist = 0;
    // spikes touching the tile, in round order; rounds handled XR_COLS at a time
    for (int rb = 0; rb < rounds; rb += XR_COLS) {
        const int r = rb + threadIdx.x;
        int lo = 0, cnt = 0;
        if (r < rounds) {
            int a = round_start[r], bnd = round_start[r + 1];
            int b2 = bnd;
            while (a < b2) {  // first spike with x >= wlo
                const int m = (a + b2) >> 1;
                if (sp_x[m] < wlo) a = m + 1; else b2 = m;
            }
            lo = a;
            int e = a;
            while (e < bnd && sp_x[e] <= whi) ++e;
            cnt = e - a;
        }
        r_cnt[threadIdx.x] = cnt;
        __syncthreads();
        if (threadIdx.x < 32) {
            constexpr int PL = XR_COLS / 32;
            int v[PL], o = 0;
#pragma unroll
            for (int i = 0; i < PL; ++i) {
                v[i] = o;
                o += r_cnt[threadIdx.x * PL + i];
            }
            const int inc = warp_inc_scan(o, threadIdx.x);
#pragma unroll
            for (int i = 0; i < PL; ++i) r_off[threadIdx.x * PL + i] = inc - o + v[i];
            if (threadIdx.x == 31) r_off[XR_COLS] = inc;
        }
        __syncthreads();
        for (int k = 0; k < cnt; ++k) {
            const int dst = nlist + r_off[threadIdx.x] + k;
            if (dst < XR_LIST_MAX) {
                l_x[dst] = sp_x[lo + k];
                l_y[dst] = sp_y[lo + k];
                l_a[dst] = sp_amp[lo + k];
            }
        }
        nlist += r_off[XR_COLS];
        __syncthreads();
    }
    if (nlist > XR_LIST_MAX) {
        if (threadIdx.x == 0) atomicOr(status, STATUS_LIST);
        nlist = XR_LIST_MAX;
    }
    const int s = s0 + threadIdx.x;
    if (s >= N) return;
    {
        const int c0 = blockIdx.y * XR_CH, nc = min(XR_CH, C - c0);
        float v[XR_CH];
#pragma unroll
        for (int k = 0; k < XR_CH; ++k) v[k] = (k < nc) ? X[(int64_t)(c0 + k) * ldx + s] : 0.f;
        for (int e = 0; e < nlist; ++e) {
            const int d = s - l_x[e];
            if (d < -h || d > h) continue;
            const float a = l_a[e];
            const float* wp = wave + ((int64_t)l_y[e] * C + c0) * nt + (d + h);
#pragma unroll
            for (int k = 0; k < XR_CH; ++k)
                if (k < nc) v[k] = __fsub_rn(v[k], __fmul_rn(a, wp[(int64_t)k * nt]));
        }
#pragma unroll
        for (int k = 0; k < XR_CH; ++k)
            if (k < nc) Xres[(int64_t)(c0 + k) * ldr + s] = v[k];
    }
}

cudaError_t launch_xres(const float* X, int64_t ldx, int32_t C, int32_t N, int32_t nt, const float* wave,
                        const int32_t* sp_x, const int32_t* sp_y, const float* sp_amp,
                        const int32_t* round_start, int32_t rounds,
                        float* Xres, int64_t ldr, int32_t* status, cudaStream_t s) {
    const dim3 grid((N + XR_COLS - 1) / XR_COLS, (C + XR_CH - 1) / XR_CH);
    k_xres<<<grid, XR_COLS, 0, s>>>(X, ldx, C, N, nt, wave, sp_x, sp_y, sp_amp, round_start, rounds, Xres,
                                     ldr, status);
    return cudaGetLastError();
}

// Records: one CTA computes every kept spike's output slot with ballot scans
// (spikes aligned before the recording start are dropped, which only happens
// in the first batch), then a grid writes the slots and their PC features.
//
// Record time t = (x - nt) + ibatch * NT + shift - nt/2 + nt0min
// (template_matching.py:54-59; shift = 0 for Kilosort's batches). With
// rc.counters the spike count is read from the device, with rc.ibatch_dev the
// batch index too, and with rc.slots > 0 batch b writes slot b % slots of
// output arrays that hold `slots` batches of `capacity` records each (the
// streaming loop's result rings).
__device__ __forceinline__ int64_t rec_time(int x, int64_t ibatch, const RecordClock& rc) {
    return (int64_t)(x - rc.nt) + ibatch * (int64_t)rc.NT + rc.shift - rc.nt / 2 + rc.nt0min;
}

__global__ void __launch_bounds__(1024) k_records_scan(const int32_t* __restrict__ sp_x, int32_t n, RecordClock rc,
                                                       int32_t* __restrict__ slot, int64_t* out_count) {
    __shared__ int wsum[32];
    __shared__ int s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (rc.counters) n = rc.counters[0];
    const int64_t ibatch = rc.ibatch_dev ? *rc.ibatch_dev : rc.ibatch;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int i = c0 + threadIdx.x;
        bool keep = false;
        if (i < n) keep = rec_time(sp_x[i], ibatch, rc) >= 0;
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) wsum[warp] = __popc(bal);
        __syncthreads();
        if (warp == 0) {
            const int c = wsum[lane];
            int inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            wsum[lane] = inc - c;
        }
        __syncthreads();
        if (i < n) slot[i] = keep ? s_base + wsum[warp] + __popc(bal & ((1u << lane) - 1u)) : -1;
        __syncthreads();
        if (threadIdx.x == 1023) s_base += wsum[31] + __popc(bal);
        __syncthreads();
    }
    if (threadIdx.x == 0) out_count[rc.slots > 0 ? ibatch % rc.slots : 0] = s_base;
}

__global__ void k_records_write(const int32_t* __restrict__ sp_x, const int32_t* __restrict__ sp_y,
                                const float* __restrict__ sp_amp, const float* __restrict__ tF,
                                const int32_t* __restrict__ slot, int32_t n, int32_t feat_len, RecordClock rc,
                                int64_t* out_time, int32_t* out_tmpl, float* out_amp, float* out_pc,
                                int64_t capacity) {
    if (rc.counters) n = rc.counters[0];
    const int64_t ibatch = rc.ibatch_dev ? *rc.ibatch_dev : rc.ibatch;
    const int64_t base = rc.slots > 0 ? (ibatch % rc.slots) * capacity : 0;
    const int row = 3 + feat_len;  // time, template, amplitude, features
    const int64_t total = (int64_t)n * row;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / row;
        const int f = (int)(e % row);
        const int o = slot[i];
        if (o < 0 || o >= capacity) continue;
        const int64_t q = base + o;
        if (f == 0) out_time[q] = rec_time(sp_x[i], ibatch, rc);
        else if (f == 1) out_tmpl[q] = sp_y[i];
        else if (f == 2) out_amp[q] = sp_amp[i];
        else if (out_pc && tF) out_pc[q * feat_len + (f - 3)] = tF[i * feat_len + (f - 3)];
    }
}

cudaError_t launch_records(const int32_t* sp_x, const int32_t* sp_y, const float* sp_amp, const float* tF,
                           int32_t* slot, int32_t n, int32_t feat_len, const RecordClock& rc, int64_t* out_time,
                           int32_t* out_tmpl, float* out_amp, float* out_pc, int64_t capacity, int64_t* out_count,
                           cudaStream_t s) {
    // n: the spike count, or (rc.counters != null) an upper bound that sizes the write grid
    if (!rc.presorted) k_records_scan<<<1, 1024, 0, s>>>(sp_x, n, rc, slot, out_count);
    const int64_t total = (int64_t)n * (3 + (tF ? feat_len : 0));
    if (total > 0) {
        const int64_t blocks = std::min<int64_t>((total + 255) / 256, rc.counters ? 1184 : INT32_MAX);
        k_records_write<<<(unsigned)blocks, 256, 0, s>>>(sp_x, sp_y, sp_amp, tF, slot, n, tF ? feat_len : 0, rc,
                                                         out_time, out_tmpl, out_amp, tF ? out_pc : nullptr,
                                                         capacity);
    }
    return cudaGetLastError();
}

__global__ void k_st_out(const int32_t* __restrict__ sp_x, const int32_t* __restrict__ sp_y,
                         const float* __restrict__ sp_amp, int32_t n, int64_t* st, float* amps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    st[2 * (int64_t)i] = sp_x[i];
    st[2 * (int64_t)i + 1] = sp_y[i];
    amps[i] = sp_amp[i];
}

cudaError_t launch_st_out(const int32_t* sp_x, const int32_t* sp_y, const float* sp_amp, int32_t n,
                          int64_t* st, float* amps, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_st_out<<<(n + 255) / 256, 256, 0, s>>>(sp_x, sp_y, sp_amp, n, st, amps);
    return cudaGetLastError();
}



// ---------------------------------------------------------------------------
// PC features without a residual array (used by lss_sort_batch, where the
// whitening is folded into the templates). With Xh the highpassed batch and
// Mw = M @ Wrot, Kilosort's
//   xfeat[i, j, k] = sum_m Xres[ch, x_i + m - nt/2] * wPCA[k, m] + amp_i * Ucc[j, y_i, k]
// (template_matching.py:50-51, ch = iCC[j, iU[y_i]]) is evaluated as
//   sum_c' Mw[ch, c'] * sum_m wPCA[k, m] Xh[c', x_i + m - nt/2]
//   - sum_{spikes i', |x_i - x_i'| < nt} amp_i' * sum_k' U[y_i', k', ch] * R[k, k', x_i - x_i']
//   + amp_i * Ucc[j, y_i, k]
// with R[k, k', d] = sum_m wPCA[k, m] wPCA[k', m + d] (the waveform of spike i'
// projected on the basis at lag d). Same linear algebra, different order.
// One CTA per spike; channels are staged 64 at a time.
// ---------------------------------------------------------------------------
constexpr int FT_CH = 64;
constexpr int FT_LIST = 512;
constexpr int FT_NQ = 32;  // neighbours per staged chunk

template <typename PT>
__device__ __forceinline__ void pc_features_one(
    int i, int rounds, const float* __restrict__ Xh, int64_t ldx, int32_t C, int32_t nt, int32_t K, int32_t nC,
    int32_t T, const float* __restrict__ wpca, const float* __restrict__ Mw, const float* __restrict__ U,
    const float* __restrict__ R, const int64_t* __restrict__ iCC, const int64_t* __restrict__ iU,
    const float* __restrict__ Ucc, const int32_t* __restrict__ sp_x, const int32_t* __restrict__ sp_y,
    const float* __restrict__ sp_amp, const int32_t* __restrict__ round_start, float* __restrict__ tF,
    int32_t* status, const PT* __restrict__ Phi, const PT* __restrict__ Plo, int64_t ldp) {
    extern __shared__ float sm[];
    const int ntp = nt + 1;
    float* ws = sm;                          // [K][nt]
    float* xs = ws + K * nt;                 // [FT_CH][ntp]
    float* pc = xs + FT_CH * ntp;            // [FT_CH][K]
    float* mw = pc + FT_CH * K;              // [nC][FT_CH]
    // the projection-row path reuses the front of the buffer (see below)
    const int front = max(K * nt + FT_CH * ntp + FT_CH * K + nC * FT_CH, C * K + nC * C + 4 * nC * K);
    float* acc = sm + front;                 // [nC*K]
    __shared__ int s_ch[64];
    __shared__ int l_x[FT_LIST], l_y[FT_LIST];
    __shared__ float l_a[FT_LIST];
    __shared__ int s_n;
    __shared__ int s_cnt[256];
    const int x = sp_x[i], y = sp_y[i];
    const int h = nt / 2;
    for (int e = threadIdx.x; e < K * nt; e += blockDim.x) ws[e] = wpca[e];
    if (threadIdx.x < nC) s_ch[threadIdx.x] = (int)iCC[(int64_t)threadIdx.x * C + iU[y]];
    for (int e = threadIdx.x; e < nC * K; e += blockDim.x) acc[e] = 0.f;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    // neighbours (any round, round order) whose waveform window overlaps this
    // spike's window; rounds are scanned blockDim.x at a time
    for (int rb = 0; rb < rounds; rb += blockDim.x) {
        const int r = rb + threadIdx.x;
        int lo = 0, cnt = 0;
        if (r < rounds) {
            const int b = round_start[r + 1];
            int hi2 = b;
            lo = round_start[r];
            while (lo < hi2) {
                const int m = (lo + hi2) >> 1;
                if (sp_x[m] <= x - nt) lo = m + 1; else hi2 = m;
            }
            int e = lo;
            while (e < b && sp_x[e] < x + nt) ++e;
            cnt = e - lo;
        }
        // exclusive prefix of the counts over the block (warp scans, then the
        // warp totals), offset by the entries listed so far
        {
            const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += u;
            }
            __shared__ int s_wtot[8];
            if (lane == 31) s_wtot[wp] = inc;
            __syncthreads();
            int before = s_n;
            for (int w2 = 0; w2 < wp; ++w2) before += s_wtot[w2];
            s_cnt[threadIdx.x] = before + inc - cnt;
            __syncthreads();
            if (threadIdx.x == blockDim.x - 1) s_n = before + inc;
            __syncthreads();
        }
        for (int q = 0; q < cnt; ++q) {
            const int slot = s_cnt[threadIdx.x] + q;
            if (slot < FT_LIST) {
                l_x[slot] = sp_x[lo + q];
                l_y[slot] = sp_y[lo + q];
                l_a[slot] = sp_amp[lo + q];
            }
        }
        __syncthreads();
    }
    if (Phi) {
        // the spike's projection row P[x, :] = hi + lo and the nC rows of Mw,
        // then each (j, k) dot product split over 4 threads, combined in order
        float* prow = sm;                  // [C*K]
        float* mwr = prow + C * K;         // [nC][C]
        float* red = mwr + nC * C;         // [4*nC*K]
        __syncthreads();
        const int64_t o = (int64_t)x * ldp;
        for (int e = threadIdx.x; e < C * K; e += blockDim.x) prow[e] = __fadd_rn(pval(Phi + o + e), pval(Plo + o + e));
        for (int e = threadIdx.x; e < nC * C; e += blockDim.x) {
            const int j = e / C, c = e % C;
            mwr[e] = Mw[(int64_t)s_ch[j] * C + c];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < 4 * nC * K; e += blockDim.x) {
            const int f = e >> 2, part = e & 3;
            const int j = f / K, k = f % K;
            float v = 0.f;
            for (int c = part; c < C; c += 4) v = fmaf(mwr[j * C + c], prow[c * K + k], v);
            red[e] = v;
        }
        __syncthreads();
        for (int f = threadIdx.x; f < nC * K; f += blockDim.x)
            acc[f] = __fadd_rn(__fadd_rn(red[4 * f], red[4 * f + 1]), __fadd_rn(red[4 * f + 2], red[4 * f + 3]));
    }
    for (int c0 = 0; c0 < (Phi ? 0 : C); c0 += FT_CH) {
        const int nc = min(FT_CH, C - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < nc * nt; e += blockDim.x) {
            const int c = e / nt, m = e % nt;
            xs[c * ntp + m] = Xh[(int64_t)(c0 + c) * ldx + x - h + m];
        }
        for (int e = threadIdx.x; e < nC * nc; e += blockDim.x) {
            const int j = e / nc, c = e % nc;
            mw[j * FT_CH + c] = Mw[(int64_t)s_ch[j] * C + c0 + c];
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nc * K; e += blockDim.x) {
            const int c = e / K, k = e % K;
            float p = 0.f;
            for (int m = 0; m < nt; ++m) p = fmaf(ws[k * nt + m], xs[c * ntp + m], p);
            pc[c * K + k] = p;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < nC * K; e += blockDim.x) {
            const int j = e / K, k = e % K;
            float v = acc[e];
            for (int c = 0; c < nc; ++c) v = fmaf(mw[j * FT_CH + c], pc[c * K + k], v);
            acc[e] = v;
        }
    }
    __syncthreads();
    const int nl = min(s_n, FT_LIST);
    if (threadIdx.x == 0 && s_n > FT_LIST) atomicOr(status, STATUS_LIST);
    // neighbours' projected waveforms, FT_NQ at a time:
    //   contrib[q][j][k] = sum_k' U[y_q, k', ch_j] * R[k, k', x - x_q]
    // all loads of a chunk are independent, then each (j, k) sums its column
    // over q in list order
    float* contrib = acc + nC * K;  // [FT_NQ][nC*K]
    const int F = nC * K;
    const int nd = 2 * nt - 1;
    float v = 0.f;
    const int e_own = threadIdx.x;  // (j, k) owned by this thread when < F
    if (e_own < F) v = acc[e_own];
    for (int q0 = 0; q0 < nl; q0 += FT_NQ) {
        const int nq = min(FT_NQ, nl - q0);
        __syncthreads();
        for (int task = threadIdx.x; task < nq * F; task += blockDim.x) {
            const int q = task / F, f = task % F;
            const int j = f / K, k = f % K;
            const int d = x - l_x[q0 + q];
            const float* rk = R + ((int64_t)k * K) * nd + (d + nt - 1);
            const float* uy = U + (int64_t)l_y[q0 + q] * K * C + s_ch[j];
            float sub = 0.f;
            for (int kk = 0; kk < K; ++kk) sub = fmaf(__ldg(uy + (int64_t)kk * C), __ldg(rk + (int64_t)kk * nd), sub);
            contrib[q * F + f] = sub;
        }
        __syncthreads();
        if (e_own < F)
            for (int q = 0; q < nq; ++q) v = __fsub_rn(v, __fmul_rn(l_a[q0 + q], contrib[q * F + e_own]));
    }
    if (e_own < F) {
        const int j = e_own / K, k = e_own % K;
        v = __fadd_rn(v, __fmul_rn(sp_amp[i], Ucc[((int64_t)j * T + y) * K + k]));
        tF[(int64_t)i * F + e_own] = v;
    }
}

// Projection-row path for ten nearest channels, K = KPC components known at
// compile time. A CTA (one per SM) takes the spikes of `cols` columns, a piece of
// them at a time: it first lists, in matching order, every spike within nt of the
// piece (a round's spikes are in time order: a thread finds a round's share by
// bisection, a warp copies it); then a warp takes a spike at a time. A piece whose
// list would not fit is halved, a sparse one is followed by a wider one, so that the
// time grows with the spikes whatever the length of the batch. Lanes own quads of
// channels (whole lines of P and of the Mw rows per load, three quads in flight; a
// lane per feature reads ten lines per load and was bound by the L1) and
// sum all ten channels' features over them; the partial sums are combined and
// dealt out together, a lane keeping half the features at every step (the same
// additions as a butterfly per feature: 62 shuffles instead of 300 for 60
// features). Each lane then finishes its FP features: the neighbours' projected
// waveforms, FS_NB loaded together and subtracted in list order, and amp * Ucc. A
// neighbour whose template is exactly zero on all of the spike's channels (urange:
// a template's first and last channel that is not) subtracts nothing and is not
// loaded; templates are local, on a 384-channel probe three of four are skipped.
// 384 channels, 19.9k spikes of 800 templates: 0.17 ms with the BF16 path's rows, 0.21
// with the FP32 path's (0.40 with a search of every round per spike, five butterfly
// steps per feature and a neighbour at a time). 32 channels, 0.68 spikes per sample:
// 0.5 ms at 60000 samples, 2.4 at 300000, 9.0 at 1200000 (with one list for the CTA's
// whole slice, and every spike read where it did not fit: 0.5, 176 and 2660).
constexpr int FS_LIST = 1024;   // spikes listed per piece (more than a spike's neighbours may be: see fw_list)
constexpr int FS_WARPS = 16;    // most warps of a CTA
constexpr int FS_MIN_COLS = 16; // least columns of a CTA
// neighbours per spike (all rounds, within +-nt), more are refused
constexpr int fw_list(int K) { return K == 6 ? 256 : FT_LIST; }
static_assert(FT_LIST < FS_LIST, "one column's list holds every spike's neighbours, or the batch is refused");
constexpr int FS_NC = 10;
constexpr int FS_NB = 4;        // neighbours whose templates are loaded together

// four projection values (hi or lo parts)
__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(u.x));
    const float2 b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// One halving step: lanes with bit OFF of their number clear keep v[0 .. N),
// the others v[N .. 2N), each plus its partner's.
template <int N, int OFF>
__device__ __forceinline__ void halve(float* v, int lane) {
    const bool up = lane & OFF;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float keep = up ? v[N + i] : v[i], give = up ? v[i] : v[N + i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, OFF);
    }
}

// Of a round's spikes [lo, hi), in time order, the ones in columns [s0, s1): both ends
// at once, since a load of either chain takes 300 cycles.
__device__ __forceinline__ void columns_of(const int32_t* __restrict__ sp_x, int s0, int s1, int& lo, int& hi) {
    int a0 = lo, b0 = hi, a1 = lo, b1 = hi;  // the first spike at or after s0 (s1) is in [a0, b0] ([a1, b1])
    while (a0 < b0 || a1 < b1) {
        const int m0 = (a0 + b0) >> 1, m1 = (a1 + b1) >> 1;
        const int x0 = a0 < b0 ? __ldg(sp_x + m0) : 0, x1 = a1 < b1 ? __ldg(sp_x + m1) : 0;
        if (a0 < b0) {
            if (x0 < s0) a0 = m0 + 1; else b0 = m0;
        }
        if (a1 < b1) {
            if (x1 < s1) a1 = m1 + 1; else b1 = m1;
        }
    }
    lo = a0;
    hi = a1;
}

template <int KPC, typename PT>
__global__ void __launch_bounds__(32 * FS_WARPS, 1) k_pc_features(
    int32_t C, int32_t nt, int32_t T, const float* __restrict__ Mw, const float* __restrict__ Ut,
    const int2* __restrict__ urange, const float* __restrict__ R, const int64_t* __restrict__ iCC,
    const int64_t* __restrict__ iU, const float* __restrict__ Ucc, const int32_t* __restrict__ sp_x,
    const int32_t* __restrict__ sp_y, const float* __restrict__ sp_amp, const int32_t* __restrict__ round_start,
    int32_t rounds, const int32_t* __restrict__ counters, float* __restrict__ tF,
    int32_t* status, const PT* __restrict__ Phi, const PT* __restrict__ Plo, int64_t ldp, int32_t cols) {
    constexpr int NC = FS_NC, F = NC * KPC, FP = (F + 31) / 32;
    constexpr bool ONE_J = KPC % FP == 0;  // a lane's features belong to one channel
    constexpr int NB = ONE_J ? FS_NB : FS_NB / 2;  // (registers)
    extern __shared__ __align__(16) float fs_sm[];
    constexpr int NW = FS_WARPS, NT = 32 * NW;
    float* Rs = fs_sm;  // [lag][k'][k]: R[k, k', lag]
    __shared__ int l_x[FS_LIST], l_y[FS_LIST], l_i[FS_LIST], l_own[FS_LIST];
    __shared__ float l_a[FS_LIST];
    __shared__ int s_lo[NT], s_off[NT + 1], s_wtot[NW];  // of a round: its first listed spike, where it goes
    __shared__ int s_at, s_w;  // the piece
    __shared__ int s_n, s_own, s_next;  // its spikes listed and owned, the next to take
    __shared__ int s_ch[FS_WARPS][NC];  // the spike's channels
    const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
    const int nd = 2 * nt - 1;
    if (counters) rounds = counters[1];
    if (threadIdx.x == 0) {
        s_at = blockIdx.x * cols;
        s_w = cols;
    }
    for (int p = wl; p < KPC * KPC; p += NW)  // a warp per pair of components; they arrive while the spikes are listed
        for (int d = lane; d < nd; d += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(Rs + d * (KPC * KPC) + (p % KPC) * KPC + p / KPC)),
                         "l"(R + (int64_t)p * nd + d)
                         : "memory");
    __syncthreads();
    // (what a piece is lives in shared memory: no register is held for it while spikes are worked on)
    for (;;) {
        const int s0 = s_at, w = min(s_w, (int)(blockIdx.x + 1) * cols - s0);
        if (w <= 0) break;
        if (threadIdx.x == 0) {
            s_own = 0;
            s_next = NW;
        }
        // ---- the spikes near the piece's columns, in matching order
        int n_list = 0;
        for (int rb = 0; rb < rounds; rb += NT) {
            const int r = rb + threadIdx.x;
            int lo = 0, cnt = 0;
            if (r < rounds) {
                lo = __ldg(round_start + r);
                cnt = __ldg(round_start + r + 1);
                columns_of(sp_x, s0 - nt + 1, s0 + w - 1 + nt, lo, cnt);
                cnt -= lo;
            }
            const int inc = warp_inc_scan(cnt, lane);
            if (lane == 31) s_wtot[wl] = inc;
            __syncthreads();
            int before = n_list, total = n_list;
#pragma unroll
            for (int v = 0; v < NW; ++v) {
                if (v < wl) before += s_wtot[v];
                total += s_wtot[v];
            }
            s_lo[threadIdx.x] = lo;
            s_off[threadIdx.x] = before + inc - cnt;
            if (threadIdx.x == 0) s_off[NT] = total;
            __syncthreads();
            n_list = total;
            if (n_list > FS_LIST) break;
            for (int q = wl; q < min(NT, rounds - rb); q += NW) {  // a warp per round
                const int at = s_off[q], ne = s_off[q + 1] - at, i0 = s_lo[q];
                for (int e = lane; e < ne; e += 32) {
                    const int i = i0 + e, xe = __ldg(sp_x + i);
                    l_x[at + e] = xe;
                    l_y[at + e] = __ldg(sp_y + i);
                    l_a[at + e] = __ldg(sp_amp + i);
                    l_i[at + e] = i;
                    if (xe >= s0 && xe < s0 + w) l_own[atomicAdd(&s_own, 1)] = at + e;
                }
            }
            __syncthreads();
        }
        if (n_list > FS_LIST) {
            if (w == 1) {  // a spike of this column has more neighbours than may be
                bool own = false;
                for (int r = threadIdx.x; r < rounds; r += NT) {
                    int lo = __ldg(round_start + r), hi = __ldg(round_start + r + 1);
                    columns_of(sp_x, s0, s0 + 1, lo, hi);
                    own |= lo < hi;
                }
                if (own) atomicOr(status, STATUS_LIST);
            }
            if (threadIdx.x == 0) {
                if (w == 1) ++s_at;
                s_w = (w + 1) / 2;
            }
            __syncthreads();
            continue;
        }
        if (threadIdx.x == 0) s_n = n_list;
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        for (int o = wl; o < s_own;) {
            // the o-th spike of these columns
            const int e = l_own[o], i = l_i[e], x = l_x[e], y = l_y[e];
            const float amp = l_a[e];
            int nx = 0;
            if (lane == 0) nx = atomicAdd(&s_next, 1);
            o = __shfl_sync(0xffffffffu, nx, 0);
            const int64_t u = iU[y];
            int chl = 0;  // lane j < NC holds channel j's index
            if (lane < NC) chl = (int)iCC[(int64_t)lane * C + u];
            const int ch_min = __reduce_min_sync(0xffffffffu, lane < NC ? chl : INT_MAX);
            const int ch_max = __reduce_max_sync(0xffffffffu, lane < NC ? chl : -1);
            __syncwarp();
            if (lane < NC) s_ch[wl][lane] = chl;
            __syncwarp();
            // ---- sums over channels: acc[j * K + k] = sum_c Mw[ch_j, c] * P[x, c*K + k]
            float acc[32 * FP];
#pragma unroll
            for (int f = 0; f < 32 * FP; ++f) acc[f] = 0.f;
            {
                const PT* ph = Phi + (int64_t)x * ldp;
                const PT* pl = Plo + (int64_t)x * ldp;
                if ((C & 3) == 0) {  // (rows of P and Mw are then whole 16-byte pieces)
#pragma unroll 3
                    for (int c = 4 * lane; c < C; c += 128) {
                        float pv[4 * KPC];
#pragma unroll
                        for (int e = 0; e < 4 * KPC; e += 4) {
                            const float4 h = ld4(ph + c * KPC + e), l = ld4(pl + c * KPC + e);
                            pv[e] = __fadd_rn(h.x, l.x);
                            pv[e + 1] = __fadd_rn(h.y, l.y);
                            pv[e + 2] = __fadd_rn(h.z, l.z);
                            pv[e + 3] = __fadd_rn(h.w, l.w);
                        }
#pragma unroll
                        for (int j = 0; j < NC; ++j) {
                            const float4 mv = ld4(Mw + (int64_t)s_ch[wl][j] * C + c);
#pragma unroll
                            for (int k = 0; k < KPC; ++k) {
                                float v = acc[j * KPC + k];
                                v = fmaf(mv.x, pv[k], v);
                                v = fmaf(mv.y, pv[KPC + k], v);
                                v = fmaf(mv.z, pv[2 * KPC + k], v);
                                acc[j * KPC + k] = fmaf(mv.w, pv[3 * KPC + k], v);
                            }
                        }
                    }
                } else {
                    for (int c = lane; c < C; c += 32) {
                        float pv[KPC];
#pragma unroll
                        for (int k = 0; k < KPC; ++k) pv[k] = __fadd_rn(pval(ph + c * KPC + k), pval(pl + c * KPC + k));
#pragma unroll
                        for (int j = 0; j < NC; ++j) {
                            const float mv = __ldg(Mw + (int64_t)s_ch[wl][j] * C + c);
#pragma unroll
                            for (int k = 0; k < KPC; ++k) acc[j * KPC + k] = fmaf(mv, pv[k], acc[j * KPC + k]);
                        }
                    }
                }
            }
            halve<16 * FP, 16>(acc, lane);
            halve<8 * FP, 8>(acc, lane);
            halve<4 * FP, 4>(acc, lane);
            halve<2 * FP, 2>(acc, lane);
            halve<FP, 1>(acc, lane);
            // ---- this lane's features f = lane * FP + q
            int jf[FP], kf[FP], cf[FP];
#pragma unroll
            for (int q = 0; q < FP; ++q) {
                const int f = min(lane * FP + q, F - 1);
                jf[q] = f / KPC;
                kf[q] = f % KPC;
                cf[q] = s_ch[wl][jf[q]];
            }
            // ---- neighbours (any round, matching order) whose window overlaps x's
            int nl = 0;
            const int n_list = s_n;
            for (int b0 = 0; b0 < n_list; b0 += 32) {
                const int q = b0 + lane;
                int xq = INT_MIN, yq = 0;
                float aq = 0.f;
                if (q < n_list) {
                    xq = l_x[q];
                    if (xq > x - nt && xq < x + nt) {
                        yq = l_y[q];
                        aq = l_a[q];
                    }
                }
                const bool near = xq > x - nt && xq < x + nt;
                nl += __popc(__ballot_sync(0xffffffffu, near));
                bool some = near;  // (an infinite amplitude times zero is not zero)
                if (near && fabsf(aq) < INFINITY) {
                    const int2 ur = __ldg(urange + yq);
                    some = ur.x <= ch_max && ur.y >= ch_min;
                }
                unsigned m = __ballot_sync(0xffffffffu, some);
                while (m) {
                    // the next NB neighbours (an = 0 past the last: it subtracts nothing)
                    int d[NB];
                    float an[NB], uv[NB][ONE_J ? 1 : FP][KPC];
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        const int src = m ? __ffs(m) - 1 : 0;
                        const int yn = __shfl_sync(0xffffffffu, yq, src);
                        const float ab = __shfl_sync(0xffffffffu, aq, src);
                        const int xb = __shfl_sync(0xffffffffu, xq, src);
                        const bool on = m != 0u;
                        m &= m - 1u;
                        d[b] = on ? x - xb + nt - 1 : -1;
                        an[b] = ab;
                        if (on) {
#pragma unroll
                            for (int q = 0; q < (ONE_J ? 1 : FP); ++q) {
                                const float* uy = Ut + ((int64_t)yn * C + cf[q]) * KPC;
                                if constexpr (KPC % 2 == 0) {
#pragma unroll
                                    for (int kk = 0; kk < KPC; kk += 2) {
                                        const float2 t = __ldg(reinterpret_cast<const float2*>(uy + kk));
                                        uv[b][q][kk] = t.x;
                                        uv[b][q][kk + 1] = t.y;
                                    }
                                } else {
#pragma unroll
                                    for (int kk = 0; kk < KPC; ++kk) uv[b][q][kk] = __ldg(uy + kk);
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        if (d[b] >= 0) {
#pragma unroll
                            for (int q = 0; q < FP; ++q) {
                                const float* rk = Rs + d[b] * (KPC * KPC) + kf[q];
                                float sub = 0.f;
#pragma unroll
                                for (int kk = 0; kk < KPC; ++kk) sub = fmaf(uv[b][ONE_J ? 0 : q][kk], rk[kk * KPC], sub);
                                acc[q] = __fsub_rn(acc[q], __fmul_rn(an[b], sub));
                            }
                        }
                }
            }
            if (nl > fw_list(KPC) && lane == 0) atomicOr(status, STATUS_LIST);
#pragma unroll
            for (int q = 0; q < FP; ++q) {
                const int f = lane * FP + q;
                if (f < F)
                    tF[(int64_t)i * F + f] =
                        __fadd_rn(acc[q], __fmul_rn(amp, Ucc[((int64_t)jf[q] * T + y) * KPC + kf[q]]));
            }
        }
        __syncthreads();  // the list has been read
        if (threadIdx.x == 0) {
            const int done = min(s_w, (int)(blockIdx.x + 1) * cols - s_at);
            s_at += done;
            s_w = s_n < FS_LIST / 2 ? min(2 * done, cols) : done;
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// CTA per spike, grid-stride over the spikes; with counters != null the spike
// and round counts are read from the matching pursuit's device counters
// (graph-captured batches, whose launch does not know them).
template <typename PT>
__global__ void __launch_bounds__(256) k_pc_features_folded(
    const float* __restrict__ Xh, int64_t ldx, int32_t C, int32_t nt, int32_t K, int32_t nC, int32_t T,
    const float* __restrict__ wpca, const float* __restrict__ Mw, const float* __restrict__ U,
    const float* __restrict__ R, const int64_t* __restrict__ iCC, const int64_t* __restrict__ iU,
    const float* __restrict__ Ucc, const int32_t* __restrict__ sp_x, const int32_t* __restrict__ sp_y,
    const float* __restrict__ sp_amp, const int32_t* __restrict__ round_start, int32_t rounds, int32_t n,
    const int32_t* __restrict__ counters, float* __restrict__ tF, int32_t* status, const PT* __restrict__ Phi,
    const PT* __restrict__ Plo, int64_t ldp) {
    if (counters) {
        n = counters[0];
        rounds = counters[1];
    }
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        pc_features_one(i, rounds, Xh, ldx, C, nt, K, nC, T, wpca, Mw, U, R, iCC, iU, Ucc, sp_x, sp_y, sp_amp,
                        round_start, tF, status, Phi, Plo, ldp);
        __syncthreads();
    }
}

template <int KPC, typename PT>
static cudaError_t launch_pcs(int32_t C, int32_t N, int32_t nt, int32_t T, const float* Mw, const float* Ut, const int2* urange, const float* R,
                              const int64_t* iCC, const int64_t* iU, const float* Ucc, const int32_t* sp_x,
                              const int32_t* sp_y, const float* sp_amp, const int32_t* round_start, int32_t rounds,
                              const int32_t* counters, float* tF,
                              int32_t* status, const PT* Phi, const PT* Plo, int64_t ldp, size_t smem, cudaStream_t s) {
    const cudaError_t e = allow_shared_memory<k_pc_features<KPC, PT>>();
    if (e != cudaSuccess) return e;
    // one CTA per SM
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cols = std::max(FS_MIN_COLS, (N + sms - 1) / std::max(sms, 1));
    k_pc_features<KPC, PT><<<(N + cols - 1) / cols, 32 * FS_WARPS, smem, s>>>(C, nt, T, Mw, Ut, urange, R, iCC, iU, Ucc, sp_x, sp_y,
                                                                          sp_amp, round_start, rounds, counters, tF, status,
                                                                          Phi, Plo, ldp, cols);
    return cudaGetLastError();
}

template <typename PT>
static cudaError_t launch_pcf(const float* Xh, int64_t ldx, int32_t C, int32_t nt, int32_t K, int32_t nC, int32_t T,
                              int32_t N, const float* wpca, const float* Mw, const float* U, const float* Ut,
                              const int2* urange, const float* R, const int64_t* iCC, const int64_t* iU, const float* Ucc,
                              const int32_t* sp_x, const int32_t* sp_y, const float* sp_amp,
                              const int32_t* round_start, int32_t rounds, int32_t n,
                              const int32_t* counters, float* tF, int32_t* status, const PT* Phi, const PT* Plo,
                              int64_t ldp, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    // ten channels: a CTA per SM while the basis correlations fit beside the lists in shared memory; else a CTA per
    // spike
    const size_t rs = 4 * (size_t)(2 * nt - 1) * K * K;
    if (Phi && nC == FS_NC && K >= 1 && K <= 8 && rs <= 180 * 1024) {
#define LSS_PCS(k)                                                                                                       \
    case k:                                                                                                              \
        return launch_pcs<k, PT>(C, N, nt, T, Mw, Ut, urange, R, iCC, iU, Ucc, sp_x, sp_y, sp_amp, round_start, rounds, counters, \
                                 tF, status, Phi, Plo, ldp, rs, s)
        switch (K) {
            LSS_PCS(1);
            LSS_PCS(2);
            LSS_PCS(3);
            LSS_PCS(4);
            LSS_PCS(5);
            LSS_PCS(6);
            LSS_PCS(7);
            LSS_PCS(8);
        }
#undef LSS_PCS
    }
    if (nC * K > 256) return cudaErrorInvalidValue;  // one (j, k) per thread
    const size_t front = std::max<size_t>((size_t)K * nt + (size_t)FT_CH * (nt + 1) + (size_t)FT_CH * K +
                                              (size_t)nC * FT_CH,
                                          (size_t)C * K + (size_t)nC * C + 4 * (size_t)nC * K);
    const size_t smem = sizeof(float) * (front + (size_t)nC * K + (size_t)FT_NQ * nC * K);
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_shared_memory<k_pc_features_folded<PT>>();
        if (e != cudaSuccess) return e;
    }
    // n: the spike count, or (counters != null) the grid size
    k_pc_features_folded<PT><<<n, 256, smem, s>>>(Xh, ldx, C, nt, K, nC, T, wpca, Mw, U, R, iCC, iU, Ucc, sp_x,
                                                  sp_y, sp_amp, round_start, rounds, n, counters, tF, status, Phi, Plo,
                                                  ldp);
    return cudaGetLastError();
}

cudaError_t launch_pc_features_folded(const float* Xh, int64_t ldx, int32_t C, int32_t nt, int32_t K, int32_t nC,
                                      int32_t T, int32_t N, const float* wpca, const float* Mw, const float* U,
                                      const float* Ut, const int2* urange, const float* R, const int64_t* iCC, const int64_t* iU,
                                      const float* Ucc, const int32_t* sp_x, const int32_t* sp_y, const float* sp_amp,
                                      const int32_t* round_start,
                                      int32_t rounds, int32_t n, const int32_t* counters, float* tF,
                                      int32_t* status, const void* Phi, const void* Plo, int32_t p_bf16, int64_t ldp,
                                      cudaStream_t s) {
    if (p_bf16)
        return launch_pcf<__nv_bfloat16>(Xh, ldx, C, nt, K, nC, T, N, wpca, Mw, U, Ut, urange, R, iCC, iU, Ucc, sp_x, sp_y, sp_amp,
                                         round_start, rounds, n, counters, tF, status,
                                         static_cast<const __nv_bfloat16*>(Phi),
                                         static_cast<const __nv_bfloat16*>(Plo), ldp, s);
    return launch_pcf<float>(Xh, ldx, C, nt, K, nC, T, N, wpca, Mw, U, Ut, urange, R, iCC, iU, Ucc, sp_x, sp_y, sp_amp, round_start,
                             rounds, n, counters, tF, status, static_cast<const float*>(Phi),
                             static_cast<const float*>(Plo), ldp, s);
}

// acc |= *st (errors of asynchronous batches, collected until lss_sync)
__global__ void k_status_or(const int32_t* st, int32_t* acc) {
    if (*st) atomicOr(acc, *st);
}

cudaError_t launch_status_or(const int32_t* st, int32_t* acc, cudaStream_t s) {
    k_status_or<<<1, 1, 0, s>>>(st, acc);
    return cudaGetLastError();
}

}  // namespace lss
