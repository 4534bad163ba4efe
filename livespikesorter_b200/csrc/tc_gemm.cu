// Template scores on the 5th-generation tensor cores (tcgen05), BF16 inputs,
// FP32 accumulation in tensor memory:
//   B[t, s] = sum_kk B0T[s, kk] * U_p[t, kk]      (kk = c*K + k)
// i.e. einsum('ijk,kjl->il', U, conv1d(X, wPCA)) of
// kilosort/template_matching.py:145-146 (cross_correlation_kernel,
// myGPUhelpers.cu:262-336, in the reference).
//
// Shape: samples are the MMA's M (128 per tile, one TMEM lane each), templates
// its N (up to 256 TMEM columns per pass, two accumulators in turn), the
// (channel, component) pairs its K (64 per pipeline stage = one 128-byte
// swizzle row of bf16). Both operands are K-major, loaded by TMA with 128B
// swizzle into a multi-stage shared-memory ring guarded by mbarriers.
//
// Warp roles (192 threads): warp 0 issues TMA, warp 1 owns TMEM and issues the
// MMAs (one elected lane), warps 2-5 drain the accumulator: each thread owns
// one sample (TMEM lane) and stores its 16 scores of a tile of the deferred rounds
// as 64 adjacent bytes (or, as rows, a template's scores 128 bytes at a time across
// a warp). Where they are wanted, the same thread forms the column maximum of
// Cf = relu(B)^2 / nm over all templates, exactly as the rounds do.
//
// Every mbarrier wait is bounded; on expiry the CTA raises an abort flag,
// drains what it issued and frees its tensor memory before returning.
#include "lss_kernels.cuh"

#include <cuda.h>

#include <algorithm>
#include <cstdio>

namespace lss {
namespace tc {

constexpr int BM = 128;               // samples per tile
constexpr int MAX_NP = 512;           // TMEM columns: two accumulators of up to 256 templates
constexpr int MAX_STAGES = 6;
constexpr int SPLIT_W = 128;          // templates per work item in split mode
constexpr int MAPPED_SPLIT_W = 64;    // ... for a re-check of a few mapped rows
constexpr int THREADS = 192;

// Element kinds of the score GEMM (TcOp).
//  BF16  : one MMA term, 128-byte rows (64 bf16 per k-block), 128B swizzle.
//  TF32x3: FP32-class accuracy from tf32 splits x = hi + lo:
//          D += A_hi B_hi + A_hi B_lo + A_lo B_hi, 64-byte rows (16 floats per
//          k-block), 64B swizzle; A and B each have a hi and a lo tile.
//  BF16x3: the same three terms with bf16 splits hi = bf16(x), lo = bf16(x - hi)
//          (about 2^-16 relative per product), 64-byte rows (32 bf16 per
//          k-block), 64B swizzle: half the operand bytes and tensor time of
//          TF32x3.
template <int OP>
struct Kind {
    static constexpr bool SPLIT = OP != TC_BF16;                   // hi and lo tiles per operand
    static constexpr uint32_t ROW = SPLIT ? 64u : 128u;            // bytes per operand row in a stage
    static constexpr int BKE = OP == TC_TF32X3 ? 16 : (OP == TC_BF16X3 ? 32 : 64);  // elements per k-block
    static constexpr int SUB = ROW / 32;                           // 32-byte MMA K steps per k-block
    static constexpr int PARTS = SPLIT ? 2 : 1;
    static constexpr uint32_t A_TILE = BM * ROW;                   // bytes of one A tile
    static constexpr uint32_t ATOM = 8 * ROW;                      // swizzle atom (8 rows)
    static constexpr uint64_t LAYOUT = SPLIT ? 4 : 2;              // UMMA layout: SWIZZLE_64B / SWIZZLE_128B
    static constexpr uint32_t FMT = OP == TC_TF32X3 ? 2u : 1u;     // operand format: TF32 (2) or BF16 (1)
};

struct Args {
    int N, T, Tpad, KB;
    int stages, b_rows;
    int nacc;                 // accumulator buffers in TMEM
    float* Bout;
    int64_t ldb;
    const float* nm;
    float* cfmax;
    int32_t* imax;
    int nt;
    int32_t* status;
    const int32_t* rowmap;    // GEMM row r scores sample rowmap[r / map_rows] * map_rows + r % map_rows (null: r)
    int map_rows;
    const int32_t* count_dev; // rows = min(N, count_dev[0] * map_rows) (null: N)
    const int32_t* perm;      // template of each operand row (null: the row's number)
    int tile_blocks;          // > 0: Bout as the deferred rounds' tiles, that many row blocks
    int ncols;                // samples in the batch (edge columns are the first/last nt)
    float* cf2;               // (error bounds) largest upper bound of any other template
    int pass_w;               // templates per pass (at most 256)
    bool split;               // one work item per (sample tile, pass) instead of per tile
    bool maxima;              // column maxima are wanted (the deferred rounds take theirs from the tiles)
    unsigned long long* keys; // split mode: one work item per (sample tile, pass); column maxima are
                              // combined as atomicMax of (Cf bits << 32 | ~t) (null: a CTA owns whole rows)
    // error bounds (BF16 path): |B - B_fp32| <= eps * un[t] * sqrt(pn2[s]) per score; per column
    // the epilogue writes cf_lo (lower bound of the best template's Cf), cf_hi (upper bound of
    // the column maximum) and, in cf2, the largest upper bound of any other template
    const float* un;
    const float* pn2;
    float eps;
    float* cf_lo;
    float* cf_hi;
    // split mode with error bounds: per (pass, column) partials, finished by
    // k_bounds_finalize: part_keys [npass][ncols] best key of the pass; part
    // [npass][4][ncols] lo of the pass's best, largest hi, its template, second hi
    unsigned long long* part_keys;
    float* part;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait (about 2 s of wall time); false when the CTA is aborting or
// the budget expired (then the abort flag and STATUS_TIMEOUT are raised).
static __device__ __noinline__ bool mbar_wait_long(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                                   int32_t* status) {
    const uint64_t t0 = globaltimer();
    for (uint32_t i = 0;; ++i) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 255u) == 255u) {
            if (*abort_flag) return false;
            if (globaltimer() - t0 > 2000000000ull) break;
        }
    }
    *abort_flag = 1;
    atomicOr(status, STATUS_TIMEOUT);
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int32_t* status) {
    return mbar_try(bar, parity) || mbar_wait_long(bar, parity, abort_flag, status);
}

// Wait (bounded, no abort check) for a phase that is known to complete.
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    const uint64_t t0 = globaltimer();
    while (!mbar_try(bar, parity) && globaltimer() - t0 < 2000000000ull) {
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// K-major operand with swizzled rows: 8-row atoms of ATOM bytes. The low word holds
// the address in 16-byte units, so that an operand elsewhere in shared memory is one
// addition away.
template <int OP>
__device__ __forceinline__ uint32_t operand_desc(uint32_t addr) {
    return ((addr >> 4) & 0x3FFFu) | (1u << 16);
}
template <int OP>
__device__ __forceinline__ uint64_t operand_at(uint32_t desc, uint32_t bytes) {
    using KD = Kind<OP>;
    constexpr uint32_t hi = (KD::ATOM >> 4) | (1u << 14) | (uint32_t)(KD::LAYOUT << 29);
    return (uint64_t)hi << 32 | (desc + (bytes >> 4));
}

// Instruction descriptor: F32 accumulator, BF16 (1) or TF32 (2) operands,
// both K-major, M = 128.
template <int OP>
__device__ __forceinline__ uint32_t instr_desc(int n) {
    const uint32_t fmt = Kind<OP>::FMT;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

template <int OP>
__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                    uint32_t accumulate) {
    if constexpr (OP == TC_TF32X3) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
            : "memory");
    }
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void st_keep(float* a, float v, uint64_t pol) {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(a), "f"(v), "l"(pol) : "memory");
}

// 8 consecutive floats (32-byte aligned), kept in L2 like st_keep
__device__ __forceinline__ void st_keep8(float* a, const uint32_t* v) {
    asm volatile("st.global.L2::evict_last.v8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "l"(a)
                 : "memory");
}

// Running column maximum of Cf = fl(fl(r*r) / nm) over a thread's scores, and
// the largest and second largest upper bounds of Cf. One warp per scheduler runs
// the epilogue, so nothing here branches: the quick quotient q = fl(fl(r*r) *
// fl(1/nm)) errs by 3.01 * 2^-24, the running state is the largest q, its row and
// score and the second largest q, and the exact quotient is formed once at the
// end; only where the two are within 8 * 2^-24 are the rows looked at again. (A
// branching form, with an exact quotient at every new maximum, bounded the BF16x3
// GEMM at about 650 cycles per score: with rows in probe order the scores rise
// step by step towards each unit. BF16x3 scores and re-check of 384 channels x 800
// templates x 60122 columns: 1.57 -> 0.84 ms.)
struct ColMax {
    float q1 = -1.f, q2 = -1.f, vb = 0.f;
    int tb = 0;
    float hi1 = 0.f, hi2 = 0.f;
    int thi1 = -1;
    __device__ __forceinline__ void consider(float v, float inv, int t) {
        const float r = fmaxf(v, 0.f);
        const float q = __fmul_rn(__fmul_rn(r, r), inv);
        q2 = fmaxf(q2, fminf(q1, q));
        const bool up = q > q1;
        q1 = fmaxf(q1, q);
        vb = up ? v : vb;
        tb = up ? t : tb;
    }
    // upper bound of the FP32 path's Cf for B within +-dB: directed rounding,
    // then a margin for the reciprocal and the rounded squares
    __device__ __forceinline__ void bound(float v, float dB, float inv, int t) {
        const float bh = fmaxf(__fadd_ru(v, dB), 0.f);
        const float hi = __fmul_ru(__fmul_ru(__fmul_ru(bh, bh), inv), 1.000001f);
        hi2 = fmaxf(hi2, fminf(hi1, hi));
        thi1 = hi > hi1 ? t : thi1;
        hi1 = fmaxf(hi1, hi);
    }
};

// Stage layout: [A_hi | A_lo] [B_hi rows | B_lo rows] (lo tiles only for the split kinds).
template <int OP>
__global__ void __launch_bounds__(THREADS, 1)
    k_score_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmAlo,
               const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmBlo, Args a) {
    using KD = Kind<OP>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t a_bytes = KD::PARTS * KD::A_TILE;
    const uint32_t b_part = (uint32_t)a.b_rows * KD::ROW;
    const uint32_t stage_bytes = a_bytes + KD::PARTS * b_part;
    uint8_t* tail = smem + (size_t)a.stages * stage_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail);  // full[S], empty[S], acc_full[2], acc_empty[2], drain
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * a.stages + 5);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* s_nm = reinterpret_cast<float*>(tmem_slot + 4);
    float* s_inv = s_nm + a.Tpad;
    float* s_un = s_inv + a.Tpad;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s0 = smem_u32(smem);
    auto full_bar = [&](int s) { return smem_u32(bars + s); };
    auto empty_bar = [&](int s) { return smem_u32(bars + a.stages + s); };
    auto accf_bar = [&](int i) { return smem_u32(bars + 2 * a.stages + i); };
    auto acce_bar = [&](int i) { return smem_u32(bars + 2 * a.stages + 2 + i); };
    const uint32_t drain_bar = smem_u32(bars + 2 * a.stages + 4);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(accf_bar(i), 1);
            mbar_init(acce_bar(i), 4);
        }
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int t = threadIdx.x; t < a.Tpad; t += THREADS) {
        const float v = (t < a.T) ? a.nm[t] : 1.f;
        s_nm[t] = v;
        s_inv[t] = __frcp_rn(v);
        s_un[t] = (a.un && t < a.T) ? a.un[t] : 0.f;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(MAX_NP)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    const int rows = a.count_dev ? min(a.N, a.count_dev[0] * a.map_rows) : a.N;
    const int ntiles = (rows + BM - 1) / BM;
    const int PW = a.pass_w;
    const int npass = (a.Tpad + PW - 1) / PW;
    const bool split = a.split;
    const int items = split ? ntiles * npass : ntiles;

    if (warp == 0) {
        if (lane == 0) {
            // ---------------- TMA producer
            int stage = 0;
            uint32_t ph = 0;
            uint32_t last_ph[MAX_STAGES];
            bool pending[MAX_STAGES] = {};
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int tile = split ? it / npass : it;
                const int pb = split ? it % npass : 0, pe = split ? pb + 1 : npass;
                for (int p = pb; p < pe && ok; ++p) {
                    const int row = p * PW;
                    int kx = 0;
                    for (int kb = 0; kb < a.KB; ++kb, kx += KD::BKE) {
                        const uint32_t full = full_bar(stage);
                        if (!mbar_wait(empty_bar(stage), ph ^ 1u, abort_flag, a.status)) { ok = false; break; }
                        const uint32_t sa = s0 + stage * stage_bytes;
                        const uint32_t sb = sa + a_bytes;
                        mbar_expect_tx(full, stage_bytes);
                        tma_load_2d(sa, &tmA, kx, tile * BM, full);
                        if (KD::SPLIT) tma_load_2d(sa + KD::A_TILE, &tmAlo, kx, tile * BM, full);
                        tma_load_2d(sb, &tmB, kx, row, full);
                        if (KD::SPLIT) tma_load_2d(sb + b_part, &tmBlo, kx, row, full);
                        last_ph[stage] = ph;
                        pending[stage] = true;
                        if (++stage == a.stages) { stage = 0; ph ^= 1u; }
                    }
                }
            }
            if (!ok) {
                // aborting: let every load this thread issued land before the CTA exits
                for (int s = 0; s < a.stages; ++s)
                    if (pending[s]) mbar_drain(full_bar(s), last_ph[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---------------- MMA issuer. A k-block's six MMAs of 208 templates
            // take 650 cycles; waiting, building every MMA's descriptors and
            // issuing took this thread 830 at any width. With the descriptors'
            // low words kept, the waits' timers out of line and a fifth stage a
            // block takes 770 (400 templates x 60122 samples, 3xTF32: 518 -> 438
            // us, 418 at the measured peak; BF16x3 at 800: 682 -> 654 us, where
            // the error bounds' epilogue waits beside it).
            const uint32_t desc_a = operand_desc<OP>(s0), desc_b = operand_desc<OP>(s0 + a_bytes);
            int stage = 0;
            uint32_t ph = 0;
            uint32_t acc_ph[2] = {0, 0};
            int acc = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
                const int pb = split ? it % npass : 0, pe = split ? pb + 1 : npass;
                for (int p = pb; p < pe && ok; ++p) {
                    const int np = min(PW, a.Tpad - p * PW);
                    if (!mbar_wait(acce_bar(acc), acc_ph[acc] ^ 1u, abort_flag, a.status)) { ok = false; break; }
                    fence_after();
                    const uint32_t dcol = tmem + (uint32_t)(acc * 256);
                    const uint32_t idesc = instr_desc<OP>(np);
                    for (int kb = 0; kb < a.KB; ++kb) {
                        if (!mbar_wait(full_bar(stage), ph, abort_flag, a.status)) { ok = false; break; }
                        fence_after();
                        const uint32_t da = desc_a + stage * (stage_bytes >> 4), db = desc_b + stage * (stage_bytes >> 4);
#pragma unroll
                        for (int ks = 0; ks < KD::SUB; ++ks) {
                            const uint64_t ad = operand_at<OP>(da, ks * 32), bd = operand_at<OP>(db, ks * 32);
                            const uint32_t acc_on = (kb | ks) != 0;
                            if (KD::SPLIT) {
                                const uint64_t adl = operand_at<OP>(da, KD::A_TILE + ks * 32);
                                const uint64_t bdl = operand_at<OP>(db + (b_part >> 4), ks * 32);
                                mma<OP>(dcol, adl, bd, idesc, acc_on);  // A_lo B_hi
                                mma<OP>(dcol, ad, bdl, idesc, 1u);      // A_hi B_lo
                                mma<OP>(dcol, ad, bd, idesc, 1u);       // A_hi B_hi
                            } else {
                                mma<OP>(dcol, ad, bd, idesc, acc_on);
                            }
                        }
                        mma_commit(empty_bar(stage));
                        if (++stage == a.stages) { stage = 0; ph ^= 1u; }
                    }
                    if (!ok) break;
                    mma_commit(accf_bar(acc));
                    acc_ph[acc] ^= 1u;
                    acc = (acc + 1) % a.nacc;
                }
            }
            if (!ok) {
                *abort_flag = 1;
                // aborting: wait for every MMA already issued before the memory is released
                mma_commit(drain_bar);
                mbar_drain(drain_bar, 0);
            }
        }
    } else {
        // ---------------- epilogue: warps 2..5, one sample per thread
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        // the score field is re-read by the matching pursuit right after: keep it in L2
        uint64_t pol;
        asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
        const int row = q * 32 + lane;
        uint32_t acc_ph[2] = {0, 0};
        int acc = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const int tile = split ? it / npass : it;
            const int pb = split ? it % npass : 0, pe = split ? pb + 1 : npass;
            const int gr = tile * BM + row;
            const int n = (a.rowmap && gr < rows) ? a.rowmap[gr / a.map_rows] * a.map_rows + gr % a.map_rows : gr;
            const bool valid = gr < rows && n < a.ncols;
            const bool edge = (n < a.nt) || (n >= a.ncols - a.nt);
            const bool bounds = a.un != nullptr;
            ColMax m;
            // bound of this column's score errors per unit template norm
            const float epsp = (bounds && valid) ? __fmul_ru(a.eps, __fsqrt_ru(a.pn2[n])) : 0.f;
            float* tile0 = a.Bout + ((int64_t)(n >> 5) * a.tile_blocks * 32 + (n & 31)) * MPB_ROWS;  // (tiles) this column's first rows
            for (int p = pb; p < pe; ++p) {
                const int np = min(PW, a.Tpad - p * PW);
                if (!mbar_wait(accf_bar(acc), acc_ph[acc], abort_flag, a.status)) { ok = false; break; }
                fence_after();
                const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * 256);
                for (int c = 0; c < np; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(tbase + (uint32_t)c, r);
                    const int t0 = p * PW + c;  // operand row (probe order)
                    if (valid) {
                        if (a.tile_blocks) {
                            // this thread's column of one tile: 64 bytes
                            static_assert(MPB_ROWS == 16, "one tile per 16 operand rows");
                            st_keep8(tile0 + (int64_t)(t0 >> 4) * 32 * MPB_ROWS, r);
                            st_keep8(tile0 + (int64_t)(t0 >> 4) * 32 * MPB_ROWS + 8, r + 8);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (t0 + j < a.T)
                                    st_keep(a.Bout + (int64_t)(a.perm ? __ldg(a.perm + t0 + j) : t0 + j) * a.ldb + n,
                                            __uint_as_float(r[j]), pol);
                        }
                    }
                    // (rows past T are zero in the operand, their nm 1 and norm 0: never a maximum)
                    if (a.maxima) {
                        if (bounds) {
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const float2 inv = *reinterpret_cast<const float2*>(s_inv + t0 + j);
                                const float2 un = *reinterpret_cast<const float2*>(s_un + t0 + j);
                                const float v0 = __uint_as_float(r[j]), v1 = __uint_as_float(r[j + 1]);
                                m.consider(v0, inv.x, t0 + j);
                                m.bound(v0, __fmul_ru(epsp, un.x), inv.x, t0 + j);
                                m.consider(v1, inv.y, t0 + j + 1);
                                m.bound(v1, __fmul_ru(epsp, un.y), inv.y, t0 + j + 1);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const float2 inv = *reinterpret_cast<const float2*>(s_inv + t0 + j);
                                m.consider(__uint_as_float(r[j]), inv.x, t0 + j);
                                m.consider(__uint_as_float(r[j + 1]), inv.y, t0 + j + 1);
                            }
                        }
                    }
                }
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acce_bar(acc));
                acc_ph[acc] ^= 1u;
                acc = (acc + 1) % a.nacc;
            }
            if (ok && valid && a.maxima) {
                // the best Cf and its first template
                float best = 0.f, lo_best = 0.f;
                int bi = 0;
                if (!edge) {
                    auto cf_of = [&](float v, int t) {
                        const float rl = fmaxf(v, 0.f);
                        return __fdiv_rn(__fmul_rn(rl, rl), s_nm[t]);
                    };
                    auto id_of = [&](int t) { return a.perm ? __ldg(a.perm + t) : t; };
                    best = cf_of(m.vb, m.tb);
                    bi = id_of(m.tb);
                    if (!(m.q1 >= 1e-30f && m.q2 < __fmul_rd(m.q1, 0.99999952316f))) {
                        // several rows may be the best: each in turn, read back as this thread wrote it
                        const int t_end = min(a.T, pe * PW);
                        best = -1.f;
                        for (int t = pb * PW; t < t_end; ++t) {
                            const int id = id_of(t);
                            const float v = a.tile_blocks ? __ldcg(tile0 + (int64_t)(t >> 4) * 32 * MPB_ROWS + (t & 15))
                                                          : __ldcg(a.Bout + (int64_t)id * a.ldb + n);
                            const float cf = cf_of(v, t);
                            if (cf > best || (cf == best && id < bi)) {
                                best = cf;
                                bi = id;
                                m.tb = t;
                                m.vb = v;
                            }
                        }
                    }
                    if (bounds) {
                        // lower bound of the best template's Cf in the FP32 path
                        const float bl = fmaxf(__fsub_rd(m.vb, __fmul_ru(epsp, s_un[m.tb])), 0.f);
                        lo_best = __fmul_rd(__fmul_rd(__fmul_rd(bl, bl), s_inv[m.tb]), 0.999999f);
                        if (m.thi1 >= 0) m.thi1 = id_of(m.thi1);
                    }
                }
                if (split && bounds) {
                    const int64_t nc = a.ncols;
                    a.part_keys[pb * nc + n] =
                        ((unsigned long long)__float_as_uint(best) << 32) | (unsigned long long)(~(uint32_t)bi);
                    a.part[(pb * 4 + 0) * nc + n] = lo_best;
                    a.part[(pb * 4 + 1) * nc + n] = edge ? 0.f : m.hi1;
                    a.part[(pb * 4 + 2) * nc + n] = __int_as_float(edge ? -1 : m.thi1);
                    a.part[(pb * 4 + 3) * nc + n] = edge ? 0.f : m.hi2;
                } else if (split) {
                    atomicMax(a.keys + n, ((unsigned long long)__float_as_uint(best) << 32) | (unsigned long long)(~(uint32_t)bi));
                } else {
                    a.cfmax[n] = best;
                    a.imax[n] = bi;
                    if (bounds) {
                        a.cf2[n] = edge ? 0.f : ((m.thi1 == bi) ? m.hi2 : m.hi1);
                        a.cf_lo[n] = lo_best;
                        a.cf_hi[n] = edge ? 0.f : m.hi1;
                    }
                }
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MAX_NP) : "memory");
    }
}

// Split mode: column maxima from the combined keys (the keys are left for the
// next user to clear).
__global__ void k_keys_to_maxima(const unsigned long long* __restrict__ keys, int N, float* __restrict__ cfmax,
                                 int32_t* __restrict__ imax) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const unsigned long long k = keys[n];
    cfmax[n] = __uint_as_float((uint32_t)(k >> 32));
    imax[n] = (int32_t)(~(uint32_t)k);
}

// Split mode with error bounds: per column, the passes' partials combined into
// what the unsplit epilogue writes: the best (Cf, first template) over the
// passes, the lower bound of that template's Cf, the largest upper bound and,
// in cf2, the largest upper bound of any other template.
__global__ void k_bounds_finalize(const unsigned long long* __restrict__ part_keys, const float* __restrict__ part,
                                  int npass, int N, int nt, float* __restrict__ cfmax, int32_t* __restrict__ imax,
                                  float* __restrict__ cf_lo, float* __restrict__ cf_hi, float* __restrict__ cf2) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    unsigned long long best = 0ull;
    int pbest = 0;
    for (int p = 0; p < npass; ++p) {
        const unsigned long long k = part_keys[(int64_t)p * N + n];
        if (k > best) {
            best = k;
            pbest = p;
        }
    }
    const int tb = (int)(~(uint32_t)best);
    float hi = 0.f, other = 0.f;
    for (int p = 0; p < npass; ++p) {
        const float h1 = part[((int64_t)p * 4 + 1) * N + n];
        const int t1 = __float_as_int(part[((int64_t)p * 4 + 2) * N + n]);
        const float h2 = part[((int64_t)p * 4 + 3) * N + n];
        hi = fmaxf(hi, h1);
        other = fmaxf(other, (t1 == tb) ? h2 : h1);
    }
    const bool edge = (n < nt) || (n >= N - nt);
    cfmax[n] = edge ? 0.f : __uint_as_float((uint32_t)(best >> 32));
    imax[n] = edge ? 0 : tb;
    cf_lo[n] = edge ? 0.f : part[((int64_t)pbest * 4 + 0) * N + n];
    cf_hi[n] = edge ? 0.f : hi;
    cf2[n] = edge ? 0.f : other;
}

// The same for the mapped columns of a re-check (rowmap, count on the device).
__global__ void k_keys_to_maxima_mapped(const unsigned long long* __restrict__ keys, const int32_t* __restrict__ rowmap,
                                        const int32_t* __restrict__ count_dev, int map_rows, int max_rows,
                                        float* __restrict__ cfmax, int32_t* __restrict__ imax) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= min(max_rows, count_dev[0] * map_rows)) return;
    const int n = rowmap[i / map_rows] * map_rows + i % map_rows;
    const unsigned long long k = keys[n];
    cfmax[n] = __uint_as_float((uint32_t)(k >> 32));
    imax[n] = (int32_t)(~(uint32_t)k);
}

}  // namespace tc

// ---------------------------------------------------------------- host side
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeTiled>(p);
    }
    return fn;
}

// 2-D tensor [rows, cols] (cols contiguous, row pitch in elements) of the
// kind's element type, box [box_rows, one swizzled row]: 128 B rows with 128B
// swizzle (BF16) or 64 B rows with 64B swizzle (TF32x3, BF16x3).
static bool make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int64_t pitch, int box_rows,
                     int op) {
    PFN_encodeTiled enc = get_encode();
    if (!enc) return false;
    const bool f32 = op == TC_TF32X3;
    const int64_t esz = f32 ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || ((pitch * esz) & 15) || box_rows < 8 || box_rows > 256 ||
        (box_rows & 7))
        return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(pitch * esz)};
    cuuint32_t box[2] = {(cuuint32_t)(op == TC_BF16 ? 64 : 64 / esz), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1u, 1u};
    return enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
               dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               op == TC_BF16 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A pass wider than 256 templates (two boxes, one accumulator) is planned only by
// lss_create's check of the template count; launch_tc refuses it.
TcPlan tc_plan(int T, int op, int pass_w) {
    TcPlan p{};
    p.Tpad = (T + 15) / 16 * 16;
    p.pass_w = std::min(pass_w, tc::MAX_NP);
    const int np0 = std::min(p.pass_w, p.Tpad);
    p.box_rows = (np0 <= 256) ? np0 : ((np0 + 1) / 2 + 7) / 8 * 8;
    int b_rows = 0;  // largest pass rounded up to whole boxes
    for (int off = 0; off < p.Tpad; off += p.pass_w) {
        const int np = std::min(p.pass_w, p.Tpad - off);
        b_rows = std::max(b_rows, (np + p.box_rows - 1) / p.box_rows * p.box_rows);
    }
    p.b_rows = b_rows;
    const size_t row = op == TC_BF16 ? 128 : 64, parts = op == TC_BF16 ? 1 : 2;
    const size_t stage = parts * (tc::BM * row + (size_t)b_rows * row);
    auto bytes = [&](int stages) { return 1024 + stages * stage + 8 * (2 * stages + 5) + 16 + 12 * (size_t)p.Tpad; };
    const size_t tail = 8 * (2 * 4 + 5) + 16 + 12 * (size_t)p.Tpad;
    const size_t budget = 227 * 1024 - 1024 - tail;
    p.stages = (int)std::min<size_t>(4, budget / stage);
    while (p.stages >= 4 && p.stages < tc::MAX_STAGES && bytes(p.stages + 1) <= 227 * 1024) ++p.stages;
    p.nacc = (np0 <= 256) ? 2 : 1;
    p.smem = bytes(p.stages);
    p.kblock = op == TC_TF32X3 ? 16 : (op == TC_BF16X3 ? 32 : 64);
    return p;
}

template <int OP>
static cudaError_t launch_tc(const void* A, const void* Alo, int64_t ldk, int N, const void* Bm, const void* Blo, int T,
                             int CKpad, const float* nm, float* Bout, int64_t ldb, float* cfmax, int32_t* imax, int nt,
                             int32_t* status, int grid, cudaStream_t s, const TcExtra& ex) {
    // Few sample tiles (short streaming batches): one work item per (tile,
    // pass of SPLIT_W templates) so that more SMs share the templates; the
    // column maxima are then combined through 64-bit keys. (Passes as narrow as
    // give every SM one take as long for one probe, 57 us for 422 samples x 800
    // templates, and slow four probes that share the device down by a sixth.)
    // A re-check of mapped rows (rowmap, count on the device) is usually one
    // or two tiles: its templates are split the same way, in narrower passes.
    const int ntiles = (N + tc::BM - 1) / tc::BM;
    // templates in passes of at most 256 TMEM columns (equal widths): two
    // accumulators alternate, so one pass's epilogue drains while the next
    // pass's MMAs run, and the smaller stages leave room for five of them
    const int tpad = (T + 15) / 16 * 16;
    const int npass = (tpad + 255) / 256;
    const int even_w = ((tpad + npass - 1) / npass + 15) / 16 * 16;
    // (the deferred rounds take the column maxima from the tiles' keys: none are formed here)
    const bool maxima = !(ex.tile_blocks && !ex.un && !ex.rowmap);
    const bool split_map = ex.keys && ex.rowmap && ex.count_dev && !ex.un && T > tc::MAPPED_SPLIT_W;
    const bool split_short = (ex.keys || !maxima) && !ex.un && !ex.rowmap && 2 * ntiles < grid && T > tc::SPLIT_W;
    // Several passes over a full batch: one work item per (tile, pass), so that
    // a tile's passes run on consecutive CTAs at the same time and its sample
    // operand is read from DRAM once (tile by tile the passes would stream it
    // once per pass, and 148 tiles in flight do not fit the L2); column maxima
    // through keys, or per-pass partials for the error bounds.
    const bool bounds_part = ex.un && ex.part_keys && ex.part && (int64_t)npass * N <= ex.part_cap;
    const bool split_pass = !split_map && !split_short && !ex.rowmap && npass > 1 &&
                            (((ex.keys || !maxima) && !ex.un) || bounds_part);
    const bool split = split_map || split_short || split_pass;
    const bool part_mode = split_pass && bounds_part;
    const TcPlan p = tc_plan(T, OP, split_map ? tc::MAPPED_SPLIT_W : (split_short ? tc::SPLIT_W : even_w));
    if (p.stages < 2 || p.b_rows > 256 || CKpad % p.kblock) return cudaErrorInvalidValue;
    CUtensorMap ma, malo, mb, mblo;
    if (!make_map(&ma, A, N, CKpad, ldk, tc::BM, OP) || !make_map(&mb, Bm, p.Tpad, CKpad, CKpad, p.box_rows, OP))
        return cudaErrorInvalidValue;
    if (tc::Kind<OP>::SPLIT) {
        if (!make_map(&malo, Alo, N, CKpad, ldk, tc::BM, OP) ||
            !make_map(&mblo, Blo, p.Tpad, CKpad, CKpad, p.box_rows, OP))
            return cudaErrorInvalidValue;
    } else {
        malo = ma;
        mblo = mb;
    }
    tc::Args a{};
    a.N = N;
    a.T = T;
    a.Tpad = p.Tpad;
    a.KB = CKpad / p.kblock;
    a.stages = p.stages;
    a.b_rows = p.b_rows;
    a.nacc = p.nacc;
    a.Bout = Bout;
    a.ldb = ldb;
    a.nm = nm;
    a.cfmax = cfmax;
    a.imax = imax;
    a.nt = nt;
    a.status = status;
    a.rowmap = ex.rowmap;
    a.map_rows = ex.map_rows;
    a.count_dev = ex.count_dev;
    a.perm = ex.perm;
    a.tile_blocks = ex.tile_blocks;
    a.ncols = ex.rowmap ? ex.ncols : N;
    a.cf2 = ex.cf2;
    a.pass_w = p.pass_w;
    a.split = split;
    a.maxima = maxima;
    a.keys = (split && !part_mode) ? ex.keys : nullptr;
    a.part_keys = part_mode ? ex.part_keys : nullptr;
    a.part = part_mode ? ex.part : nullptr;
    a.un = (split && !part_mode) ? nullptr : ex.un;
    a.pn2 = ex.pn2;
    a.eps = ex.eps;
    a.cf_lo = ex.cf_lo;
    a.cf_hi = ex.cf_hi;
    if (a.un && (!a.pn2 || !a.cf2 || !a.cf_lo || !a.cf_hi || ex.rowmap)) return cudaErrorInvalidValue;
    cudaError_t e = allow_shared_memory<tc::k_score_tc<OP>>();
    if (e != cudaSuccess) return e;
    const int items = split ? ntiles * ((p.Tpad + p.pass_w - 1) / p.pass_w) : ntiles;
    if (split && !part_mode && maxima) {
        e = cudaMemsetAsync(ex.keys, 0, (size_t)(split_map ? ex.ncols : N) * sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
    }
    tc::k_score_tc<OP><<<std::min(grid, items), tc::THREADS, p.smem, s>>>(ma, malo, mb, mblo, a);
    if (part_mode)
        tc::k_bounds_finalize<<<(N + 255) / 256, 256, 0, s>>>(ex.part_keys, ex.part, (p.Tpad + p.pass_w - 1) / p.pass_w, N,
                                                              nt, cfmax, imax, ex.cf_lo, ex.cf_hi, ex.cf2);
    else if (split_map)
        tc::k_keys_to_maxima_mapped<<<(N + 255) / 256, 256, 0, s>>>(ex.keys, ex.rowmap, ex.count_dev, ex.map_rows, N,
                                                                    cfmax, imax);
    else if (split && maxima)
        tc::k_keys_to_maxima<<<(N + 255) / 256, 256, 0, s>>>(ex.keys, N, cfmax, imax);
    return cudaGetLastError();
}

cudaError_t launch_score_tc(const __nv_bfloat16* B0T, int64_t ldk, int N, const __nv_bfloat16* Up, int T, int CKpad,
                            const float* nm, float* Bout, int64_t ldb, float* cfmax, int32_t* imax, int nt,
                            int32_t* status, int grid, cudaStream_t s, const TcExtra& ex) {
    return launch_tc<TC_BF16>(B0T, nullptr, ldk, N, Up, nullptr, T, CKpad, nm, Bout, ldb, cfmax, imax, nt, status, grid,
                              s, ex);
}

cudaError_t launch_score_tc_bf16x3(const __nv_bfloat16* B0T_hi, const __nv_bfloat16* B0T_lo, int64_t ldk, int N,
                                   const __nv_bfloat16* Up_hi, const __nv_bfloat16* Up_lo, int T, int CKpad,
                                   const float* nm, float* Bout, int64_t ldb, float* cfmax, int32_t* imax, int nt,
                                   int32_t* status, int grid, cudaStream_t s, const TcExtra& ex) {
    return launch_tc<TC_BF16X3>(B0T_hi, B0T_lo, ldk, N, Up_hi, Up_lo, T, CKpad, nm, Bout, ldb, cfmax, imax, nt, status,
                                grid, s, ex);
}

cudaError_t launch_score_tc_tf32x3(const float* B0T_hi, const float* B0T_lo, int64_t ldk, int N, const float* Up_hi,
                                   const float* Up_lo, int T, int CKpad, const float* nm, float* Bout, int64_t ldb,
                                   float* cfmax, int32_t* imax, int nt, int32_t* status, int grid, cudaStream_t s,
                                   const TcExtra& ex) {
    return launch_tc<TC_TF32X3>(B0T_hi, B0T_lo, ldk, N, Up_hi, Up_lo, T, CKpad, nm, Bout, ldb, cfmax, imax, nt, status,
                                grid, s, ex);
}

}  // namespace lss
