// Device helpers shared by the two matching-pursuit kernels (mp.cu: the
// rounds that update every row; mp_lazy.cu: the rounds that update a tile of
// the score field only when it can take part in a decision).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lss_kernels.cuh"

namespace lss {

constexpr unsigned MP_SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ bool grid_sync(unsigned int* bar, int32_t* status) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile unsigned int* vgen = bar + 1;
        const unsigned int gen = *vgen;
        __threadfence();
        const unsigned int arrived = atomicAdd(bar, 1u);
        int ok = 1;
        if (arrived == gridDim.x - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            unsigned int spins = 0;
            while (*vgen == gen) {
                ++spins;
                if ((spins & 255u) == 0u && (*(volatile int32_t*)status & STATUS_TIMEOUT)) {
                    ok = 0;
                    break;
                }
                if (spins > MP_SPIN_LIMIT) {
                    atomicOr(status, STATUS_TIMEOUT);
                    ok = 0;
                    break;
                }
                if (spins > 64) __nanosleep(32);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// L2 residency: the score field is read-modify-written every round and fits
// in L2 for a few hundred templates, while each spike's ctc slice is read once
// per spike, so the field is kept (evict_last) and ctc streamed (evict_first).
__device__ __forceinline__ uint64_t policy_keep() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t policy_stream() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float ld_keep(const float* a, uint64_t pol) {
    float v;
    asm volatile("ld.global.cg.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_keep(float* a, float v, uint64_t pol) {
    asm volatile("st.global.cg.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(a), "f"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ float ld_stream(const float* a, uint64_t pol) {
    float v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(a), "l"(pol));
    return v;
}

// Phase clock of the rounds (thread 0 of each CTA): time in the peak phase,
// waiting after it, in the update phase and waiting after it, summed over the
// rounds; added to phase[0..3] in ns (sums over CTAs) with the slowest CTA's
// peak and update totals in phase[4], phase[5]. Laps read the SM's cycle
// counter (the global timer takes about half a microsecond per read); the
// totals are scaled by the global timer's span over the cycles' span.
// The clock lives in shared memory, so that no register is held for it.
struct PhaseClock {
    static constexpr int WORDS = 7;
    unsigned long long* s;  // [WORDS] shared: last lap, four sums, first cycle, first time
    __device__ __forceinline__ static unsigned long long now() {
        unsigned long long v;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
        return v;
    }
    __device__ __forceinline__ void start() {
        s[6] = now();
        s[0] = s[5] = (unsigned long long)clock64();
        for (int i = 1; i < 5; ++i) s[i] = 0;
    }
    __device__ __forceinline__ void lap(int i) {
        const unsigned long long u = (unsigned long long)clock64();
        s[1 + i] += u - s[0];
        s[0] = u;
    }
    __device__ __forceinline__ void flush(unsigned long long* phase) const {
        if (!phase) return;
        const double ns = (double)(now() - s[6]) / (double)max(1ull, (unsigned long long)clock64() - s[5]);
        unsigned long long t[4];
        for (int i = 0; i < 4; ++i) {
            t[i] = (unsigned long long)((double)s[1 + i] * ns);
            atomicAdd(phase + i, t[i]);
        }
        atomicMax(phase + 4, t[0]);
        atomicMax(phase + 5, t[2]);
    }
};

__device__ __forceinline__ float cf_of(float b, float nmv) {
    const float r = fmaxf(b, 0.f);
    return __fdiv_rn(__fmul_rn(r, r), nmv);
}

__device__ __forceinline__ unsigned long long pack_key(float cf, int t) {
    return ((unsigned long long)__float_as_uint(cf) << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned)t);
}


// Running maximum of Cf = fl(fl(r*r) / nm) (r = relu(b)) with the first index
// on ties. The correctly rounded quotient is formed only for candidates:
// a = fl(fl(r*r) * fl(1/nm)) is within 3.01 ulp of it, so a < best*(1 - 8 ulp)
// proves the exact value is below best (checked only while best is a normal
// number, where the relative bounds hold).
struct ColMax {
    float best = -1.f;
    float thr = -1.f;  // rounded-down best * (1 - 2^-21)
    int bi = 0;
    __device__ __forceinline__ void consider(float b, float nmv, float inv, int t) {
        const float r = fmaxf(b, 0.f);
        const float sq = __fmul_rn(r, r);
        if (__fmul_rn(sq, inv) < thr) return;
        const float cf = __fdiv_rn(sq, nmv);
        if (cf > best) {
            best = cf;
            bi = t;
            thr = (cf >= 1e-30f) ? __fmul_rd(cf, 0.99999952316f) : -1.f;
        }
    }
};

// Best Cf of column s over rows [t0, t1), loads issued eight rows at a time.
__device__ __forceinline__ void column_best(const float* __restrict__ B, int64_t ldb, const float* s_nm,
                                            const float* s_inv, int s, int t0, int t1, ColMax& m) {
    const float* bp = B + (int64_t)t0 * ldb + s;
    int t = t0;
    for (; t + 8 <= t1; t += 8, bp += 8 * ldb) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldcg(bp + u * ldb);
#pragma unroll
        for (int u = 0; u < 8; ++u) m.consider(v[u], s_nm[t + u], s_inv[t + u], t + u);
    }
    for (; t < t1; ++t, bp += ldb) m.consider(__ldcg(bp), s_nm[t], s_inv[t], t);
}

// Inclusive warp scan.
__device__ __forceinline__ int warp_inc_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

}  // namespace lss
