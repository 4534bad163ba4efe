// FP32 SIMT GEMM, C[M,N] = A[M,K] @ B[K,N], all row-major.
//
// Used by the FP32 parity path for the whitening/drift product
// ((M @ Wrot) @ X, kilosort/io.py:782-789; cublasSgemm in
// OnlineSpikesV2.cu:767-778) and the template score GEMM
// (einsum('ijk,kjl->il'), template_matching.py:146;
// cross_correlation_kernel, myGPUhelpers.cu:262-336).
// Each output is a single FP32 FMA chain over k in ascending order, so the
// result is deterministic and independent of the launch shape.
//
// Tiling: BM x BN outputs per CTA of 256 threads, TM x TN per thread in quads 64
// apart (conflict-free 16-byte shared-memory reads), slabs of GBK in two shared
// buffers: the next slab's B rows are copied asynchronously and its A values held
// in registers while the current one is consumed. Two outputs of a row go through
// one packed FMA (f32x2: each value rounded on its own, so every output is the
// same chain), with A's values doubled in registers: a warp's shared-memory reads
// arrive at 128 bytes per cycle also where lanes read the same value, and 8x16
// outputs per thread take 24 cycles of them per k against 32 of FMAs (8x8 with A
// stored doubled: 24 against 16, 523 us below). Bound by the FP32 pipe in the
// large case: 384 x 384 x 60122 in 391 us, 45 TFLOP/s of the 74 that the FMA units
// give (8x8 scalar outputs: 771 us). The folded operand of 800 templates x 6 x 384
// takes 62 us and the C x C product 20 us (117 and 42 us), bound by the latency of
// few CTAs.
#include "lss_kernels.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace lss {

constexpr int GBK = 16;

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ unsigned long long dup2(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}

// Stores take four adjacent outputs (m, n .. n + 3) of an N-column product.
struct StorePlain {
    static constexpr bool FOLDED = false;
    float* Cm;
    int64_t ldc;
    int vec;  // floats per piece that every row is aligned for: 4, 2 or 1
    __device__ void operator()(int m, int n, int N, const float (&v)[4]) const {
        float* p = Cm + (int64_t)m * ldc + n;
        if (vec == 4 && n + 4 <= N) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else if (vec == 2 && n + 4 <= N) {
            *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
            *reinterpret_cast<float2*>(p + 2) = make_float2(v[2], v[3]);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (n + u < N) p[u] = v[u];
        }
    }
};

// Folded-template layout of the score GEMM: row m = t*K + k, column n = c'
// goes to [t, c'*K + k] of a row-stride-ldk array, as the bf16 split
// hi = bf16(v), lo = bf16(v - hi) or as the tf32 split hi = rna(v),
// lo = rna(v - hi) (both exact tf32 values).
struct StoreFolded {
    static constexpr bool FOLDED = true;
    int K;
    int64_t ldk;
    __nv_bfloat16* out16;
    __nv_bfloat16* out16lo;
    float* hi;
    float* lo;
    __device__ __forceinline__ void one(int64_t o, float v) const {
        if (out16) {
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            out16[o] = h;
            if (out16lo) out16lo[o] = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(h)));
        }
        if (hi) {
            uint32_t r;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
            const float h = __uint_as_float(r);
            hi[o] = h;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(__fsub_rn(v, h)));
            lo[o] = __uint_as_float(r);
        }
    }
};

template <int BM, int BN, class Store>
__global__ void __launch_bounds__(256) k_sgemm(const float* __restrict__ A, int64_t lda, const float* __restrict__ B,
                                               int64_t ldb, int M, int N, int K, int vecA, int vecB, Store store) {
    constexpr int TM = BM / 16, TN = BN / 16;      // outputs per thread
    constexpr int QM = TM / 4, QN = TN / 4;        // ... in quads
    constexpr int NA = BM * GBK / 4 / 256;         // float4s of an A slab per thread
    constexpr int NBV = BN * GBK / 4 / 256;        // ... of a B slab
    __shared__ __align__(16) float smem[2 * GBK * (BM + BN)];
    float(*As)[GBK][BM] = reinterpret_cast<float(*)[GBK][BM]>(smem);
    float(*Bs)[GBK][BN] = reinterpret_cast<float(*)[GBK][BN]>(smem + 2 * GBK * BM);
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid & 15, ty = tid >> 4;
    float4 ra[NA];
    auto load_a = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int idx = tid + 256 * i, kq = idx / BM * 4, gm = m0 + idx % BM, gk = k0 + kq;
            const float* p = A + (int64_t)gm * lda + gk;
            if (vecA && gm < M && gk + 4 <= K) {
                ra[i] = __ldg(reinterpret_cast<const float4*>(p));
            } else {
                const bool in = gm < M;
                ra[i] = make_float4(in && gk < K ? p[0] : 0.f, in && gk + 1 < K ? p[1] : 0.f, in && gk + 2 < K ? p[2] : 0.f,
                                    in && gk + 3 < K ? p[3] : 0.f);
            }
        }
    };
    auto store_a = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int idx = tid + 256 * i, kq = idx / BM * 4, mm = idx % BM;
            const float v[4] = {ra[i].x, ra[i].y, ra[i].z, ra[i].w};
#pragma unroll
            for (int u = 0; u < 4; ++u) As[buf][kq + u][mm] = v[u];
        }
    };
    auto copy_b = [&](int k0, int buf) {
#pragma unroll
        for (int i = 0; i < NBV; ++i) {
            const int idx = tid + 256 * i, kk = idx / (BN / 4), nn = idx % (BN / 4) * 4;
            const int gk = k0 + kk, gn = n0 + nn;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(&Bs[buf][kk][nn]);
            const float* p = B + (int64_t)min(gk, K - 1) * ldb;
            if (vecB && gn + 4 <= N) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(p + gn), "r"(gk < K ? 16 : 0)
                             : "memory");
            } else {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool in = gk < K && gn + u < N;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4u * u), "l"(p + (in ? gn + u : 0)),
                                 "r"(in ? 4 : 0)
                                 : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    auto step = [&](int buf, int kk) {
        unsigned long long av[TM], bv[TN / 2];
#pragma unroll
        for (int q = 0; q < QM; ++q) {
            const float4 p = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4 + 64 * q]);
            av[4 * q] = dup2(p.x);
            av[4 * q + 1] = dup2(p.y);
            av[4 * q + 2] = dup2(p.z);
            av[4 * q + 3] = dup2(p.w);
        }
#pragma unroll
        for (int q = 0; q < QN; ++q) {
            const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(&Bs[buf][kk][tx * 4 + 64 * q]);
            bv[2 * q] = p.x;
            bv[2 * q + 1] = p.y;
        }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], av[i], bv[j]);
    };
    const int nslab = (K + GBK - 1) / GBK;
    load_a(0);
    copy_b(0, 0);
    for (int t = 0; t < nslab; ++t) {
        const int buf = t & 1;
        store_a(buf);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // slab t is there; slab t - 1 has been consumed, its buffer is free
        if (t + 1 < nslab) {
            load_a((t + 1) * GBK);
            copy_b((t + 1) * GBK, buf ^ 1);
        }
        if (K - t * GBK >= GBK) {
#pragma unroll
            for (int kk = 0; kk < GBK; ++kk) step(buf, kk);
        } else {
            for (int kk = 0; kk < K - t * GBK; ++kk) step(buf, kk);  // no terms past K: the chain is exactly k = 0 .. K-1
        }
    }
    if constexpr (Store::FOLDED) {
        // rows (t, k) of the tile side by side along k: through shared memory, to be written in runs of K values
        static_assert(BM * 65 <= 2 * GBK * (BM + BN), "64 staged columns");
        const int t0 = m0 / store.K, t1 = (min(m0 + BM, M) - 1) / store.K;
#pragma unroll
        for (int q = 0; q < QN; ++q) {
            __syncthreads();
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float* p = smem + (ty * 4 + (i & 3) + (i >> 2) * 64) * 65 + tx * 4;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(p[0]), "=f"(p[1]) : "l"(acc[i][2 * q]));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(p[2]), "=f"(p[3]) : "l"(acc[i][2 * q + 1]));
            }
            __syncthreads();
            const int run = 64 * store.K;
            for (int t = t0; t <= t1; ++t) {
                for (int e = tid; e < run; e += 256) {
                    const int nn = e / store.K, m = t * store.K + e - nn * store.K - m0, n = n0 + 64 * q + nn;
                    if (m >= 0 && m < BM && n < N)
                        store.one(t * store.ldk + (int64_t)n * store.K + (m0 + m - t * store.K), smem[m * 65 + nn]);
                }
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int gm = m0 + ty * 4 + (i & 3) + (i >> 2) * 64;
            if (gm >= M) continue;
#pragma unroll
            for (int q = 0; q < QN; ++q) {
                float v[4];
                asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(acc[i][2 * q]));
                asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2]), "=f"(v[3]) : "l"(acc[i][2 * q + 1]));
                store(gm, n0 + tx * 4 + 64 * q, N, v);
            }
        }
    }
}

template <int BM, int BN, class Store>
static cudaError_t launch_tiles(const float* A, int64_t lda, const float* B, int64_t ldb, int M, int N, int K, Store store,
                                cudaStream_t s) {
    auto vec = [](const float* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && (ld & 3) == 0; };
    dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)((M + BM - 1) / BM));
    k_sgemm<BM, BN><<<grid, 256, 0, s>>>(A, lda, B, ldb, M, N, K, (int)vec(A, lda), (int)vec(B, ldb), store);
    return cudaGetLastError();
}

cudaError_t launch_sgemm(const float* A, int64_t lda, const float* B, int64_t ldb, float* Cm, int64_t ldc,
                         int M, int N, int K, cudaStream_t s) {
    auto rows_on = [&](unsigned bytes) { return reinterpret_cast<uintptr_t>(Cm) % bytes == 0 && ldc * 4 % bytes == 0; };
    const StorePlain st{Cm, ldc, rows_on(16) ? 4 : rows_on(8) ? 2 : 1};
    // A 64x64 tile reads two shared values per FMA pair of a thread and is bound by that at half the FMA rate; a
    // 128x256 tile is not, but is eight times the work: fewer of them than half the SMs, and the small tile's
    // spread over the chip is worth as much. 64-row tiles where the last 128 rows would be at most half full.
    if ((int64_t)((N + 255) / 256) * ((M + 127) / 128) < 74) return launch_tiles<64, 64>(A, lda, B, ldb, M, N, K, st, s);
    if ((M + 127) / 128 * 128 - M >= 64) return launch_tiles<64, 256>(A, lda, B, ldb, M, N, K, st, s);
    return launch_tiles<128, 256>(A, lda, B, ldb, M, N, K, st, s);
}

cudaError_t launch_sgemm_folded(const float* U, const float* Mw, int32_t T, int32_t K, int32_t C, int64_t ldk,
                                __nv_bfloat16* out16, __nv_bfloat16* out16lo, float* hi, float* lo, cudaStream_t s) {
    // rows t*K + k of U [T, K, C] (row-major, stride C) times Mw [C, C]
    return launch_tiles<64, 128>(U, C, Mw, C, T * K, C, C, StoreFolded{K, ldk, out16, out16lo, hi, lo}, s);
}

}  // namespace lss
