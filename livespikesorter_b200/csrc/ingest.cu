// Ingest of one padded batch: int16 rows -> channel mean removal -> median
// common-average reference -> circular highpass.
//
// Semantics follow kilosort/io.py:584-637 (padded_batch_to_torch) and
// io.py:757-777 (BinaryFiltered.filter up to the whitening); the whitening and
// drift GEMM runs in gemm_fp32.cu. LiveSpikeSorter's equivalents are
// meanRemove / median_remove_kernel / highpassFilter
// (myGPUhelpers.cu:98-118,471-534; OnlineSpikesV2.cu:976-1026).
//
// HBM layout: raw int16 [n_rows, ld_raw] (the file's interleaved rows), output
// float [C, ldx] channel-major with time contiguous, so every later stage reads
// 128-byte rows.
#include "lss_kernels.cuh"
#include "mp_common.cuh"

namespace lss {

__device__ __forceinline__ int64_t src_row(int64_t s, const IngestMap& m, int64_t base) {
    if (m.base_dev) {
        const int64_t r = base + s;
        return r < 0 ? 0 : r % m.ring_rows;
    }
    int64_t j = s - m.lead;
    if (j < 0) j = 0;
    if (j >= m.nsamp) {
        if (m.zero_tail) return -1;
        j = m.nsamp - 1;
    }
    return j;
}

// Per-channel integer sums over the padded batch (exact: raw samples are
// integers, so the mean is the correctly rounded quotient of an exact sum).
// Grid: one CTA per `cols` columns (a multiple of 8); a warp per column at a time with
// channels lane + 32q in registers (the loads of two columns in flight), per-lane int
// sums combined across the CTA's warps in shared memory, one 64-bit atomic per channel
// and CTA. Bound by the latency of its loads: 64 columns per CTA fill the chip in a
// long batch, fewer in a short one (384 x 60122 in 19 us, 422 columns in 2.5 us, against 69 and 34 us with
// 256 columns per CTA and a branch per load).
template <int NQ>
__global__ void __launch_bounds__(256) k_chan_sums(const int16_t* __restrict__ raw, int32_t ld_raw,
                                                   const int32_t* __restrict__ chan_map, int32_t C, int64_t N,
                                                   IngestMap map, int cols, long long* __restrict__ sums) {
    __shared__ int part[8][NQ * 32];
    const int64_t s0 = (int64_t)blockIdx.x * cols;
    const int64_t s1 = min(N, s0 + cols);
    const int64_t base = map.base_dev ? *map.base_dev : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int acc[NQ];
    int ch[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int c = lane + 32 * q;
        acc[q] = 0;
        ch[q] = (c < C) ? (chan_map ? chan_map[c] : c) : 0;
    }
    constexpr int P = NQ <= 12 ? 2 : 1;  // columns in flight
    for (int64_t sc = s0 + warp; sc < s1; sc += 8 * P) {
        int16_t v[P][NQ];
        int mask[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const int64_t r = sc + 8 * p < s1 ? src_row(sc + 8 * p, map, base) : -1;
            const int16_t* row = raw + max(r, (int64_t)0) * ld_raw;
            mask[p] = r >= 0 ? -1 : 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) v[p][q] = row[ch[q]];  // no branch: all loads in flight (lanes past C: unused)
        }
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int q = 0; q < NQ; ++q) acc[q] += v[p][q] & mask[p];
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) part[warp][lane + 32 * q] = acc[q];
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        int t = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += part[w][c];
        atomicAdd((unsigned long long*)&sums[c], (unsigned long long)(long long)t);
    }
}

template <int NQ>
static void launch_sums_t(const int16_t* raw, int32_t ld_raw, const int32_t* chan_map, int32_t C, int64_t N,
                          IngestMap map, long long* sums, cudaStream_t s) {
    const int cols = (int)std::min<int64_t>(64, std::max<int64_t>(8, N / (4 * 148) / 8 * 8));
    const int grid = (int)((N + cols - 1) / cols);
    k_chan_sums<NQ><<<grid, 256, 0, s>>>(raw, ld_raw, chan_map, C, N, map, cols, sums);
}

cudaError_t launch_chan_sums(const int16_t* raw, int32_t ld_raw, const int32_t* chan_map, int32_t C,
                             int64_t N, IngestMap map, long long* sums, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(sums, 0, sizeof(long long) * C, s);
    if (e != cudaSuccess) return e;
    const int nq = (C + 31) / 32;
    if (nq <= 2) launch_sums_t<2>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else if (nq <= 4) launch_sums_t<4>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else if (nq <= 8) launch_sums_t<8>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else if (nq <= 12) launch_sums_t<12>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else if (nq <= 16) launch_sums_t<16>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else if (nq <= 24) launch_sums_t<24>(raw, ld_raw, chan_map, C, N, map, sums, s);
    else launch_sums_t<32>(raw, ld_raw, chan_map, C, N, map, sums, s);
    return cudaGetLastError();
}

// Order-preserving float -> uint32 key.
__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unkey(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// Lower median (sorted index (C-1)/2, torch.median's choice) of a warp's C values,
// v[q] of lane l being value l + 32 q (padding +inf; no NaN and no -0), found by
// counting: two pivots about the mean, 1.7 standard errors of the median apart for
// normal values, leave about 20 of 384 values between them; a further pair of pivots
// tightens the bracket, by rank on even turns and halving the floats in it on odd
// ones, until at most 32 values are left. Those are packed one per lane and each
// counts the ones not above it. About 300 instructions per column of 384; a search
// bit by bit over the floats takes 32 counts, 1150.
template <int NQ>
__device__ __forceinline__ float lower_median(const float (&v)[NQ], int C, float mean, float& d0, float* cand,
                                              int lane) {
    const int kth = (C - 1) / 2;
    const float big = 3.0e38f;  // above every value in magnitude
    float flo = -big, fhi = big;
    int clo = 0, chi = C;  // values not above flo, fhi; clo <= kth < chi
    if (C > 32) {
        if (d0 < 0.f) {  // the warp's first column
            float dev = 0.f;
#pragma unroll
            for (int q = 0; q < NQ; ++q) dev += (lane + 32 * q < C) ? fabsf(v[q] - mean) : 0.f;
            // sums of at most 32 values below 2^18, in eighths: 32 lanes of them fit
            const float total = 0.125f * (float)__reduce_add_sync(0xffffffffu, (unsigned)(8.f * fminf(dev, 8388608.f)));
            d0 = fmaxf(31.f * total / ((float)C * (float)C), 0.01f);
        }
        float d = d0;
        float p1 = mean - d, p2 = mean + d;
        for (int turn = 0; turn < 128; ++turn) {
            unsigned cnt = 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) cnt += (v[q] <= p1 ? 1u : 0u) + (v[q] <= p2 ? 0x10000u : 0u);
            cnt = __reduce_add_sync(0xffffffffu, cnt);
            const int n1 = (int)(cnt & 0xffffu), n2 = (int)(cnt >> 16);
            if (n1 > kth) {
                fhi = p1;
                chi = n1;
            } else {
                flo = p1;
                clo = n1;
                if (n2 > kth) {
                    fhi = p2;
                    chi = n2;
                } else {
                    flo = p2;
                    clo = n2;
                }
            }
            if (chi - clo <= 32) break;
            const uint32_t klo = fkey(flo), khi = fkey(fhi);
            if (khi - klo <= 1) return fhi;  // nothing but fhi itself
            if (flo == -big || fhi == big) {
                d *= 3.f;
                p1 = (flo == -big) ? fhi - d : flo + 0.4f * d;
                p2 = (flo == -big) ? fhi - 0.4f * d : flo + d;
            } else if (turn & 1) {
                p1 = p2 = unkey(klo + (khi - klo) / 2);
            } else {
                const float w = (fhi - flo) / (float)(chi - clo);
                const float est = flo + w * ((float)(kth - clo) + 0.5f);
                p1 = est - 10.f * w;
                p2 = est + 10.f * w;
            }
            // strictly inside the bracket, in order
            p1 = fminf(fmaxf(p1, unkey(klo + 1)), unkey(khi - 1));
            p2 = fminf(fmaxf(p2, p1), unkey(khi - 1));
        }
        if (chi - clo > 32) return fhi;  // (the bracket halves every other turn: not reached)
    }
    __syncwarp();
    cand[lane] = big;
    __syncwarp();
    unsigned in = 0;  // of the chi - clo values in the bracket, this lane's
#pragma unroll
    for (int q = 0; q < NQ; ++q) in |= (v[q] > flo && v[q] <= fhi) ? 1u << q : 0u;
    const int mine = __popc(in);
    float* dst = cand + warp_inc_scan(mine, lane) - mine;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
        if (in >> q & 1u) *dst++ = v[q];
    __syncwarp();
    const float x = cand[lane];
    int le = 0;
    for (int i = 0; i < chi - clo; i += 4) {
        const float4 o = *reinterpret_cast<const float4*>(cand + i);
        le += (o.x <= x) + (o.y <= x) + (o.z <= x) + (o.w <= x);
    }
    const uint32_t key = le > kth - clo ? fkey(x) : 0xFFFFFFFFu;
    return unkey(__reduce_min_sync(0xffffffffu, key));
}

// CAR tile: COLS time columns x C channels staged in shared memory, a warp per column
// at a time (NQ = values per lane >= C/32): its channels' loads in flight together, the
// median taken off, then the tile is written back as rows of COLS samples. Tiles of 32
// columns (128-byte rows); of 8 in batches that give the chip less than one CTA per SM
// of those (384 x 60122 in 62 us, 422 columns in 4.9 us; bit-wise search and 32 columns: 169 and 28 us).
template <int NQ, int COLS>
__global__ void __launch_bounds__(256, NQ <= 12 ? 4 : 1) k_car(const int16_t* __restrict__ raw, int32_t ld_raw,
                                             const int32_t* __restrict__ chan_map, int32_t C,
                                             int64_t N, IngestMap map, float sign,
                                             const long long* __restrict__ sums, int do_car,
                                             float* __restrict__ X1, int64_t ldx) {
    extern __shared__ __align__(16) float sm[];
    float* cand = sm + 32 * (threadIdx.x >> 5);  // [8 warps][32]
    float* tile = sm + 8 * 32;                   // [C][COLS + 1]
    float* mean = tile + (size_t)C * (COLS + 1);  // [NQ * 32]
    int* chan = reinterpret_cast<int*>(mean + NQ * 32);  // [NQ * 32]
    const int64_t s0 = (int64_t)blockIdx.x * COLS;
    const int ncol = (int)min((int64_t)COLS, N - s0);
    const double invN = 1.0 / (double)N;
    const int64_t base = map.base_dev ? *map.base_dev : 0;
    for (int c = threadIdx.x; c < NQ * 32; c += 256) {
        mean[c] = c < C ? (float)((double)sign * (double)sums[c] * invN) : 0.f;
        chan[c] = c >= C ? 0 : chan_map ? chan_map[c] : c;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float invC = 1.f / (float)C;
    float mbar = 0.f;  // mean of the channel means (where the search starts from)
#pragma unroll
    for (int q = 0; q < NQ; ++q) mbar += mean[lane + 32 * q];
#pragma unroll
    for (int o = 16; o; o >>= 1) mbar += __shfl_xor_sync(0xffffffffu, mbar, o);
    mbar *= invC;
    float d0 = -1.f;
    for (int j = warp; j < ncol; j += 8) {
        const int64_t r = src_row(s0 + j, map, base);
        const int16_t* row = raw + max(r, (int64_t)0) * ld_raw;
        const int mask = r >= 0 ? -1 : 0;
        int16_t x[NQ];
        float v[NQ];
        int sx = 0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) x[q] = row[chan[lane + 32 * q]];  // (lanes past C: unused)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const bool on = lane + 32 * q < C;
            const int xi = x[q] & mask;
            sx += on ? xi : 0;
            v[q] = on ? __fsub_rn(sign * (float)xi, mean[lane + 32 * q]) : INFINITY;
        }
        float mj = 0.f;
        if (do_car) {
            sx = __reduce_add_sync(0xffffffffu, sx);
            mj = lower_median<NQ>(v, C, sign * (float)sx * invC - mbar, d0, cand, lane);
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int c = lane + 32 * q;
            if (c < C) tile[c * (COLS + 1) + j] = do_car ? __fsub_rn(v[q], mj) : v[q];
        }
    }
    __syncthreads();
    // rows of whole 16-byte pieces (ldx and s0 are multiples of 4)
    for (int idx = threadIdx.x; idx < C * (COLS / 4); idx += 256) {
        const int j = idx % (COLS / 4) * 4, c = idx / (COLS / 4);
        const float* t = tile + c * (COLS + 1) + j;
        float* o = X1 + (int64_t)c * ldx + s0 + j;
        if (j + 4 <= ncol) {
            *reinterpret_cast<float4*>(o) = make_float4(t[0], t[1], t[2], t[3]);
        } else {
            for (int u = 0; u < ncol - j; ++u) o[u] = t[u];
        }
    }
}

template <int NQ, int COLS>
static cudaError_t launch_car_cols(const int16_t* raw, int32_t ld_raw, const int32_t* chan_map, int32_t C, int64_t N,
                                   IngestMap map, float sign, const long long* sums, int do_car, float* X1, int64_t ldx,
                                   cudaStream_t s) {
    const size_t smem = sizeof(float) * (8 * 32 + (size_t)C * (COLS + 1) + 2 * NQ * 32);
    const cudaError_t e = allow_shared_memory<k_car<NQ, COLS>>();
    if (e != cudaSuccess) return e;
    k_car<NQ, COLS><<<(unsigned)((N + COLS - 1) / COLS), 256, smem, s>>>(raw, ld_raw, chan_map, C, N, map, sign, sums,
                                                                         do_car, X1, ldx);
    return cudaGetLastError();
}

template <int NQ>
static cudaError_t launch_car_t(const int16_t* raw, int32_t ld_raw, const int32_t* chan_map, int32_t C, int64_t N,
                                IngestMap map, float sign, const long long* sums, int do_car, float* X1, int64_t ldx,
                                cudaStream_t s) {
    if (N < 148 * 32) return launch_car_cols<NQ, 8>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    return launch_car_cols<NQ, 32>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
}

cudaError_t launch_car(const int16_t* raw, int32_t ld_raw, const int32_t* chan_map, int32_t C, int64_t N,
                       IngestMap map, float sign, const long long* sums, int do_car, float* X1,
                       int64_t ldx, cudaStream_t s) {
    const int nq = (C + 31) / 32;
    if (nq <= 2) return launch_car_t<2>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    if (nq <= 4) return launch_car_t<4>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    if (nq <= 8) return launch_car_t<8>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    if (nq <= 12) return launch_car_t<12>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    if (nq <= 16) return launch_car_t<16>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    if (nq <= 24) return launch_car_t<24>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
    return launch_car_t<32>(raw, ld_raw, chan_map, C, N, map, sign, sums, do_car, X1, ldx, s);
}

// Circular highpass: Xh[c, i] = sum_{d=-L..L} taps[d+L] * X1[c, (i+d) mod N].
// This equals fftshift(real(ifft(fft(X) * conj(fft(h_N))))) of
// kilosort/preprocessing.py:138-154 + io.py:771-774 with the impulse response
// truncated where its tail mass is below 2^-30 of its L1 norm (the host picks
// L; the tail then contributes less than the FP32 rounding of the transform).
// CTA: one channel, HP_TILE outputs; thread: 8 consecutive outputs with a
// sliding register window over the staged input.
constexpr int HP_TILE = 1024;
constexpr int HP_THREADS = HP_TILE / 8;
__global__ void __launch_bounds__(HP_THREADS) k_highpass(const float* __restrict__ X1, int64_t ldx, int64_t N,
                                                         const float* __restrict__ taps, int32_t L,
                                                         float* __restrict__ Xh) {
    extern __shared__ float sm[];
    const int ntap = 2 * L + 1;
    const int ntap_pad = (ntap + 7) & ~7;
    float* tp = sm;                      // [ntap_pad] (zero padded)
    float* xs = sm + ntap_pad;           // [HP_TILE + ntap_pad + 8]
    const int c = blockIdx.y;
    const int64_t i0 = (int64_t)blockIdx.x * HP_TILE;
    const float* xrow = X1 + (int64_t)c * ldx;
    for (int e = threadIdx.x; e < ntap_pad; e += blockDim.x) tp[e] = (e < ntap) ? taps[e] : 0.f;
    const int nx = HP_TILE + ntap_pad + 8;
    for (int p = threadIdx.x; p < nx; p += blockDim.x) {
        int64_t g = i0 - L + p;
        g %= N;
        if (g < 0) g += N;
        xs[p] = xrow[g];
    }
    __syncthreads();
    float acc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = 0.f;
    const int o = threadIdx.x * 8;
    float w[16];
#pragma unroll
    for (int r = 0; r < 8; ++r) w[r] = xs[o + r];
    for (int eb = 0; eb < ntap_pad; eb += 8) {
#pragma unroll
        for (int r = 0; r < 8; ++r) w[8 + r] = xs[o + eb + 8 + r];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float t = tp[eb + u];
#pragma unroll
            for (int r = 0; r < 8; ++r) acc[r] = fmaf(t, w[r + u], acc[r]);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) w[r] = w[8 + r];
    }
    float* yrow = Xh + (int64_t)c * ldx;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int64_t i = i0 + o + r;
        if (i < N) yrow[i] = acc[r];
    }
}

cudaError_t launch_highpass(const float* X1, int64_t ldx, int32_t C, int64_t N, const float* taps, int32_t L,
                            float* Xh, cudaStream_t s) {
    const int ntap_pad = ((2 * L + 1) + 7) & ~7;
    const size_t smem = sizeof(float) * ((size_t)ntap_pad + HP_TILE + ntap_pad + 8);
    const cudaError_t e = allow_shared_memory<k_highpass>();
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((N + HP_TILE - 1) / HP_TILE), (unsigned)C);
    k_highpass<<<grid, HP_THREADS, smem, s>>>(X1, ldx, N, taps, L, Xh);
    return cudaGetLastError();
}



// ---------------------------------------------------------------------------
// The same circular highpass by overlap-save FFT convolution (used when the
// truncated impulse response has L <= 1024). One CTA filters two channels at
// once as the real and imaginary parts of a 4096-point complex signal (the
// filter is real, so both come out of one transform): the block x[start-L ..
// start-L+4096) (indices mod N) is transformed by a radix-16 Stockham FFT in
// registers and shared memory, multiplied by H = conj(FFT(g)) where g holds the taps wrapped
// around index 0 (a circular correlation), and transformed back; its outputs
// L .. 4096-L-1 are exact (their taps never wrap inside the block).
// ---------------------------------------------------------------------------
constexpr int HF = 4096;

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(__fsub_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)),
                       __fadd_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}

// Shared-memory index with one pad slot per 16 points (radix-16 passes write
// with stride 16: the pad spreads those writes over the banks).
__device__ __forceinline__ int pad16(int i) { return i + (i >> 4); }
constexpr int HFP = HF + HF / 16;

__device__ __forceinline__ void dft4(float2& x0, float2& x1, float2& x2, float2& x3) {
    const float2 s02 = make_float2(x0.x + x2.x, x0.y + x2.y), d02 = make_float2(x0.x - x2.x, x0.y - x2.y);
    const float2 s13 = make_float2(x1.x + x3.x, x1.y + x3.y), d13 = make_float2(x1.x - x3.x, x1.y - x3.y);
    x0 = make_float2(s02.x + s13.x, s02.y + s13.y);
    x1 = make_float2(d02.x + d13.y, d02.y - d13.x);  // d02 - i*d13
    x2 = make_float2(s02.x - s13.x, s02.y - s13.y);
    x3 = make_float2(d02.x - d13.y, d02.y + d13.x);  // d02 + i*d13
}

// In-register 16-point forward DFT, natural order in and out (n = 4 n1 + n2,
// k = k1 + 4 k2: four 4-point DFTs, twiddles exp(-2 pi i n2 k1 / 16), four
// more 4-point DFTs).
__device__ __forceinline__ void dft16(float2 v[16]) {
    const float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, r2 = 0.70710678118654752f;
    const float2 W[10] = {{1.f, 0.f}, {c1, -s1}, {r2, -r2}, {s1, -c1}, {0.f, -1.f},
                          {-s1, -c1}, {-r2, -r2}, {-c1, -s1}, {-1.f, 0.f}, {-c1, s1}};
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) dft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
    // v[4 k1 + n2] now holds y[n2][k1]
#pragma unroll
    for (int n2 = 1; n2 < 4; ++n2)
#pragma unroll
        for (int k1 = 1; k1 < 4; ++k1) v[4 * k1 + n2] = cmul(v[4 * k1 + n2], W[n2 * k1]);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // v[4 k1 + k2] holds X[k1 + 4 k2]: transpose to natural order
    float2 t[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1)
#pragma unroll
        for (int k2 = 0; k2 < 4; ++k2) t[k1 + 4 * k2] = v[4 * k1 + k2];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = t[i];
}

// The radix-16 Stockham passes (L = 1, 16, 256), one butterfly per thread
// (blockDim.x == HF / 16), in place. Thread j takes the points j + 256 i of every
// pass and leaves those of the last one, so the first pass starts from registers and
// the last ends in them: the samples, the product with H and the outputs never pass
// through shared memory, which a block crosses four times instead of sixteen. The
// twiddle of point i is read from a table laid out [i][k] (i = 1..15, k < L),
// neighbouring threads at neighbouring places; exp(-2 pi i n / 4096) by its n
// put a warp's lanes on up to 30 lines per load.
template <int L>
__device__ __forceinline__ void twiddle(float2 v[16], const float2* __restrict__ tw) {
    const int k = threadIdx.x & (L - 1);
#pragma unroll
    for (int i = 1; i < 16; ++i) v[i] = cmul(v[i], __ldg(tw + i * L + k));
}

template <int L>
__device__ __forceinline__ void put(float2* a, const float2 v[16]) {
    constexpr int lg = (L == 1) ? 0 : 4, step = (L == 1) ? 1 : 17;  // pad16(base + L * i) - pad16(base) = step * i
    const int j = threadIdx.x, base = (j >> lg) * 16 * L + (j & (L - 1));
    a += pad16(base);
#pragma unroll
    for (int i = 0; i < 16; ++i) a[step * i] = v[i];
    __syncthreads();
}

__device__ __forceinline__ void get(const float2* a, float2 v[16]) {
    a += pad16(threadIdx.x);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = a[pad16((HF / 16) * i)];
}

__device__ __forceinline__ void fft4096(float2 v[16], float2* a, const float2* __restrict__ tw) {
    dft16(v);
    put<1>(a, v);
    get(a, v);
    twiddle<16>(v, tw + 16 * 256);
    dft16(v);
    __syncthreads();
    put<16>(a, v);
    get(a, v);
    twiddle<256>(v, tw);
    dft16(v);
}

constexpr int HF_THREADS = HF / 16;

// Bound by its FP32 adds and multiplies (about 50 us at the full rate for 384 x 60122) with the shared-memory
// passes beside them: 93 us, against 242 with every pass through shared memory. Two CTAs per SM: the 16 points, their
// twiddles and a butterfly's temporaries take 128 registers (118 and 116 us with four and three CTAs, which spill).
__global__ void __launch_bounds__(HF_THREADS, 2) k_highpass_fft(const float* __restrict__ X1, int64_t ldx, int32_t C,
                                                               int64_t N, int32_t L, const float2* __restrict__ H,
                                                               const float2* __restrict__ tw, float* __restrict__ Xh) {
    extern __shared__ float2 A[];  // [HFP]: one padded 4096-point buffer, transformed in place
    const int c1 = 2 * blockIdx.y, c2 = c1 + 1;
    const bool two = c2 < C;
    const int64_t start = (int64_t)blockIdx.x * (HF - 2 * L);
    const float* x1 = X1 + (int64_t)c1 * ldx;
    const float* x2 = X1 + (int64_t)(two ? c2 : c1) * ldx;
    float2 v[16];
    if (start - L >= 0 && start - L + HF <= N) {
        x1 += start - L + threadIdx.x;
        x2 += start - L + threadIdx.x;
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i].x = x1[i * HF_THREADS];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i].y = two ? x2[i * HF_THREADS] : 0.f;
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) {  // the ends wrap around
            int g = ((int)(start - L) + (int)threadIdx.x + i * HF_THREADS) % (int)N;
            if (g < 0) g += (int)N;
            v[i] = make_float2(x1[g], two ? x2[g] : 0.f);
        }
    }
    fft4096(v, A, tw);
    // conj(Z * H): the second forward transform then gives conj(F * y)
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 z = cmul(v[i], __ldg(H + threadIdx.x + i * HF_THREADS));
        v[i] = make_float2(z.x, -z.y);
    }
    __syncthreads();
    fft4096(v, A, tw);
    const float inv = 1.f / (float)HF;
    const int nend = (int)min((int64_t)(HF - L), N - start + L);
    float* y1 = Xh + (int64_t)c1 * ldx + (start - L + threadIdx.x);
    float* y2 = y1 + ldx;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int n = threadIdx.x + i * HF_THREADS;
        if (n >= L && n < nend) {
            y1[i * HF_THREADS] = v[i].x * inv;
            if (two) y2[i * HF_THREADS] = -v[i].y * inv;
        }
    }
}

cudaError_t launch_highpass_fft(const float* X1, int64_t ldx, int32_t C, int64_t N, int32_t L, const float2* H,
                                const float2* tw, float* Xh, cudaStream_t s) {
    if (L > 1024) return cudaErrorInvalidValue;
    const size_t smem = HFP * sizeof(float2);
    const cudaError_t e = allow_shared_memory<k_highpass_fft>();
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((N + (HF - 2 * L) - 1) / (HF - 2 * L)), (unsigned)((C + 1) / 2));
    k_highpass_fft<<<grid, HF_THREADS, smem, s>>>(X1, ldx, C, N, L, H, tw, Xh);
    return cudaGetLastError();
}

}  // namespace lss
