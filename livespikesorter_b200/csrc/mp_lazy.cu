// Greedy matching pursuit that updates a piece of the score field only when
// the piece can take part in a decision. Same rounds, same arithmetic and the
// same spikes and amplitudes as k_mp (mp.cu) and Kilosort's round loop
// (kilosort/template_matching.py:157-198, LiveSpikeSorter's
// kilosortMatchingPursuit, OnlineSpikesV2.cu:873-971).
//
// The field is cut into tiles of 16 template rows (in probe order, so that a
// tile's templates lie close together) by 32 columns, 2 KB each with a column's
// rows adjacent: a warp holds a tile in registers, lane = column, and moves its
// rows, like the rows of ctc at a lag, 32 bytes at a time. A spike (x, y, a)
// changes B[t, s] to fl(B - fl(a * ctc[t, y, s - x + nt])) in the 2nt+1 columns
// around x. Of the field only the columns' best templates are ever looked at,
// and of those only the ones above the threshold: a peak has Cf > Th^2, and a
// column maximum at or below Th^2 changes no decision. So for every tile the
// kernel keeps an upper bound U of relu(B) / sqrt(nm) over the whole tile: the
// bound its exact values give, plus a * max over rows and lags of
// (-ctc / sqrt(nm)) for every spike since, rounded up. While U^2 is below Th^2
// the tile is left alone and the spike stays pending; when U reaches the
// threshold the pending spikes are applied, all of them in the order the rounds
// found them. Every element then sees exactly the reference's operations in the
// reference's order, only later, and a tile that never reaches the threshold
// again is never touched. On a 384-channel probe with 800 templates a batch
// meets 4.8M (spike, tile) pairs, of which 0.64M are applied, in 0.42M loads of
// a tile (3.0 GB, against 23.4 GB when every row is updated).
//
// A spike whose terms leave a tile bit for bit unchanged is not even pending:
// for |B| in [2^e, 2^(e+1)) any |d| < 2^(e-25) leaves fl(B - d) == B, so with
// tmin = min |B| of the tile and h = max over rows and lags of |ctc|, the terms
// are no-ops where fl(a * h) < quarter ulp of tmin.
//
// The two interleaved passes of a round (even-numbered spikes' terms, then the
// odd ones'; with duplicate columns within a pass the last spike wins) become
// an order of the log: the round's even spikes, then its odd ones, each valid
// on [x - nt, hi], hi ending before the next spike of the same parity begins.
//
// Work split: a CTA owns whole 32-column chunks (all their tiles, the keys in
// shared memory), so a tile is only ever read and written by its CTA. CTAs
// exchange 64-bit words that carry their round's tag next to the data, so a
// reader polls the data itself and no fence or barrier counter is needed:
//   * the column maxima within nt of a CTA's edge, read by its neighbours;
//   * the peaks (x, y, a), read by the CTAs whose columns they reach;
//   * each CTA's peak count, read by those, and a round later by every CTA: the
//     round's total ends the loop and numbers the records.
// The parity of a spike is its number in the whole round, but it only orders
// spikes whose windows overlap: a CTA near peaks closer than 2nt reads the counts
// to its left in the same round, the others wait for their neighbours alone.
// (Every CTA reading every count at once cost 10 us of a round's 31 at 800
// templates, the skew between them: 2.23 ms of rounds against 2.00, 0.81 against
// 0.72 at 400. Counts two or three rounds late gain nothing more.)
// Peaks and counts are double-buffered by round parity: before a CTA sends those
// of round r + 2 it has read every CTA's count of round r + 1, each sent after
// its sender had read the peaks and all counts of round r. Column maxima need one
// buffer: their readers' counts are read before the next ones are sent.
// Every wait is bounded (STATUS_TIMEOUT).
#include "lss_kernels.cuh"
#include "mp_common.cuh"

#include <algorithm>
#include <cfloat>
#include <climits>

namespace lss {

constexpr int MPL_THREADS = 1024;
constexpr int MPL_WARPS = MPL_THREADS / 32;
constexpr int MPL_MAX_GRID = 1024;  // (MPL_WARPS warps' lanes: collect)
constexpr int MPL_LOG = 512;          // least log capacity (spikes)
constexpr unsigned MPL_SPIN_LIMIT = 1u << 21;  // polls of a word (about 1.5 s)
constexpr int MPL_REGIONS = 40;       // CTAs whose peaks reach one CTA's columns
constexpr unsigned FULL = 0xffffffffu;
static_assert(MPB_ROWS % 8 == 0, "a column of a tile moves in 32-byte pieces");

// 2^(e - 25) for v in [2^e, 2^(e+1)) (v >= 0): any |d| below it leaves
// fl(v' - d) == v' for every v' with |v'| >= v. Zero when v is zero,
// subnormal, tiny, infinite or NaN (nothing is then skipped).
__device__ __forceinline__ float quarter_ulp(float v) {
    const unsigned e = (__float_as_uint(v) >> 23) & 0xFFu;
    return (e > 25u && e < 255u) ? __uint_as_float((e - 25u) << 23) : 0.f;
}

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Polls *p until its tag (high word) is `tag`; false when the wait gave up.
__device__ __forceinline__ bool poll_word(const unsigned long long* p, unsigned tag, unsigned long long& v,
                                          int32_t* status) {
    for (unsigned spins = 0;; ++spins) {
        v = ld_word(p);
        if ((unsigned)(v >> 32) == tag) return true;
        if ((spins & 255u) == 255u && (*(volatile int32_t*)status & STATUS_TIMEOUT)) return false;
        if (spins > MPL_SPIN_LIMIT) {
            atomicOr(status, STATUS_TIMEOUT);
            return false;
        }
    }
}
// A peak travels in two words: {tag | amplitude} and {12-bit tag | 28-bit x |
// 24-bit template} (the launcher checks the ranges; rounds stay below 2^12).
__device__ __forceinline__ unsigned long long pack_xy(unsigned tag, int x, int y) {
    return ((unsigned long long)(tag & 0xFFFu) << 52) | ((unsigned long long)(unsigned)x << 24) |
           (unsigned long long)(unsigned)y;
}

// Eight rows of a column of a tile (32 bytes). A tile is read and written by
// its own CTA only (between its barriers), so plain loads are coherent; the
// field is kept in L2 as far as it fits, ctc streams through it.
__device__ __forceinline__ void ld_tile8(const float* p, float* v) {
    asm volatile("ld.global.L1::no_allocate.L2::evict_last.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_tile8(float* p, const float* v) {
    asm volatile("st.global.L2::evict_last.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(v[0]), "f"(v[1]),
                 "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(p)
                 : "memory");
}
__device__ __forceinline__ void ld_ctc8(const float* p, float* v) {
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}

// upper bound of relu(B) / sqrt(nm) where the best Cf is cf (Cf = fl(fl(r*r) /
// nm) errs by 2^-23 relative, and by less than 1e-36 absolute where r*r is
// subnormal; the approximate root errs by 2^-23)
__device__ __forceinline__ float bound_of(float cf) {
    float q;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(q) : "f"(cf));
    return __fadd_ru(__fmul_ru(q, 1.000001f), 1e-18f);
}
// true when a bound may belong to a Cf that matters: at or above Th^2 less a
// margin over the peak test's 1e-9 (NaN: true)
__device__ __forceinline__ bool reaches(float ub, float th2) {
    return !(__fadd_ru(__fmul_ru(__fmul_ru(ub, ub), 1.000001f), 2e-9f) < th2);
}


// One CTA per SM: its tiles' keys take most of the shared memory (KSMEM; wider
// slices keep them in global memory).
template <bool KSMEM>
__global__ void __launch_bounds__(MPL_THREADS, 1) k_mp_lazy(MPArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_total, s_pref, s_own, s_base, s_nnew, s_qn, s_qold, s_qnext;
    __shared__ int s_rcnt[MPL_REGIONS];
    __shared__ unsigned long long s_clk[PhaseClock::WORDS];

    const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int N = a.N, T = a.T, nt = a.nt, L2 = 2 * nt + 1, nb = a.nb;
    const int W = a.cols_per_blk, cpc = W / 32, ntile = cpc * nb;
    const int lo = b * W, hi = min(N, lo + W);
    const int nchunk = (hi - lo + 31) / 32;  // chunks that hold columns (every CTA has one)
    const int qend = nchunk * nb, nbg = (nb + 31) / 32, ng = (L2 + MPB_LAGS - 1) / MPB_LAGS;

    // ---- shared memory (mpl_smem_bytes)
    int4* s_log = reinterpret_cast<int4*>(smem_raw);                 // [log_cap] spikes x, hi, template, amplitude
    int4* s_new = s_log + a.log_cap;                                 // [new_cap] this round's
    unsigned long long* s_key = reinterpret_cast<unsigned long long*>(s_new + a.new_cap);  // [nb][W] (KSMEM)
    float* s_vals = reinterpret_cast<float*>(s_key + (KSMEM ? (size_t)nb * W : 0));         // [W + 2nt]
    int* s_ival = reinterpret_cast<int*>(s_vals + W + 2 * nt);       // [W]
    float* s_amp = reinterpret_cast<float*>(s_ival + W);             // [W]
    float* s_nm = s_amp + W;                                         // [nb * MPB_ROWS] by row
    float* s_inv = s_nm + nb * MPB_ROWS;                             // [nb * MPB_ROWS]
    int* s_perm = reinterpret_cast<int*>(s_inv + nb * MPB_ROWS);     // [nb * MPB_ROWS]
    int* s_rowof = s_perm + nb * MPB_ROWS;                           // [T]
    int* s_minp = s_rowof + T;                                       // [nb] smallest template of a block
    float* s_tmin = reinterpret_cast<float*>(s_minp + nb);           // [ntile] min |B| of a tile with nothing pending
    float* s_ub = s_tmin + ntile;                                    // [ntile] bound of relu(B) / sqrt(nm)
    int* s_app = reinterpret_cast<int*>(s_ub + ntile);               // [ntile] first pending log entry, -1: none
    int* s_queue = s_app + ntile;                                    // [ntile]
    unsigned* s_peak = reinterpret_cast<unsigned*>(s_queue + ntile); // [cpc] peak columns of a chunk
    int* s_touch = reinterpret_cast<int*>(s_peak + cpc);             // [cpc] the last round's spikes reach the chunk

    // the key of tile (blk, c) in this lane's column
    auto ld_key = [&](int blk, int c) {
        return KSMEM ? s_key[(size_t)blk * W + c * 32 + lane] : __ldcg(a.bkey + (int64_t)blk * a.ldk + lo + c * 32 + lane);
    };
    auto st_key = [&](int blk, int c, unsigned long long k) {
        if (KSMEM) s_key[(size_t)blk * W + c * 32 + lane] = k;
        else __stcg(a.bkey + (int64_t)blk * a.ldk + lo + c * 32 + lane, k);
    };
    // the rows of tile (blk, c) in this lane's column
    auto tile_at = [&](int blk, int c) { return a.B + (((int64_t)(lo / 32 + c) * nb + blk) * 32 + lane) * MPB_ROWS; };
    // ---- words exchanged with other CTAs: counts [2][G], column maxima
    // [G * W], peaks [2][G * W][2]
    unsigned long long* x_cnt = a.xch;
    unsigned long long* x_val = x_cnt + 2 * G;
    unsigned long long* x_pk = x_val + (int64_t)G * W;
    if (tid < 2) st_word(x_cnt + tid * G + b, 0ull);
    for (int i = tid; i < W; i += MPL_THREADS) {
        st_word(x_val + lo + i, 0ull);
        for (int p = 0; p < 2; ++p) {
            st_word(x_pk + 2 * ((int64_t)p * G * W + lo + i), 0ull);
            st_word(x_pk + 2 * ((int64_t)p * G * W + lo + i) + 1, 0ull);
        }
    }
    for (int i = tid; i < nb * MPB_ROWS; i += MPL_THREADS) {
        const int t = __ldg(a.perm + i);
        s_perm[i] = t;
        const float v = i < T ? __ldg(a.nm + t) : 1.f;
        s_nm[i] = v;
        s_inv[i] = i < T ? __frcp_rn(v) : 0.f;
        if (i < T) s_rowof[t] = i;
    }
    for (int i = tid; i < nb; i += MPL_THREADS) {
        int m = INT_MAX;
        for (int u = i * MPB_ROWS; u < min(T, (i + 1) * MPB_ROWS); ++u) m = min(m, __ldg(a.perm + u));
        s_minp[i] = m;
    }
    for (int q = tid; q < ntile; q += MPL_THREADS) s_app[q] = -1;
    for (int c = tid; c < cpc; c += MPL_THREADS) s_touch[c] = 1;
    if (tid == 0) s_qn = s_qold = s_qnext = s_total = s_pref = s_base = 0;
    __syncthreads();
    int n_app = 0, n_items = 0;  // (spike, tile) updates applied (per warp) and met (per lane)

    // bounds {h, g} of a spike's ctc rows of block blk over the lags at which it
    // meets the chunk that begins at c_lo
    auto lag_bounds = [&](const int4& ev, int c_lo, int blk) {
        const int g0 = max(c_lo - ev.x + nt, 0) / MPB_LAGS, g1 = (min(c_lo + 31, ev.y) - ev.x + nt) / MPB_LAGS;
        const float2* hp = a.hg + ((int64_t)ev.z * ng + g0) * nb + blk;
        float2 m = make_float2(0.f, 0.f), t[5];  // 32 lags lie in at most 5 groups of 8
#pragma unroll
        for (int u = 0; u < 5; ++u) t[u] = g0 + u <= g1 ? __ldg(hp + u * nb) : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 5; ++u) m = make_float2(fmaxf(m.x, t[u].x), fmaxf(m.y, t[u].y));
        return m;
    };
    // smallest |score| of a tile from the lanes' minima
    auto tile_min = [&](float mn, bool act) {
        return __uint_as_float(__reduce_min_sync(FULL, act ? __float_as_uint(mn) : 0x7f800000u));
    };
    // Brings tile q = c * nb + blk up to date with the log's first nlog
    // entries: its rows in registers (lane = column), the pending spikes'
    // terms one spike at a time, then its keys, bound and tmin.
    auto resolve = [&](int q, int nlog) {
        const int c = q / nb, blk = q - c * nb;
        const int r0 = blk * MPB_ROWS, nr = min(MPB_ROWS, T - r0);
        const int c_lo = lo + c * 32, s = c_lo + lane, c_hi = min(c_lo + 31, N - 1);
        const bool act = s < N;
        float v[MPB_ROWS], w[MPB_ROWS];
        float* bp = tile_at(blk, c);
#pragma unroll
        for (int u = 0; u < MPB_ROWS; u += 8) ld_tile8(bp + u, v + u);
        if (nr < MPB_ROWS) {  // rows past T: never the best, never the smallest
#pragma unroll
            for (int u = 0; u < MPB_ROWS; ++u)
                if (u >= nr) v[u] = -INFINITY;
        }
        const int first = s_app[q];
        const bool changed = first >= 0;
        float mn = INFINITY;
        // 32 log entries at a time, lane = entry: hm = the largest |term| that
        // the spike can have in the tile (-1: it does not reach the chunk), so
        // that after each spike the next one that matters is a ballot away
        for (int w0 = first; changed && w0 < nlog; w0 += 32) {
            float hm = -1.f;
            int4 ev = make_int4(0, 0, 0, 0);
            if (w0 + lane < nlog) {
                ev = s_log[w0 + lane];
                if (ev.x - nt <= c_hi && ev.y >= c_lo) hm = fabsf(__fmul_rn(__int_as_float(ev.w), lag_bounds(ev, c_lo, blk).x));
            }
            // the first pending spike is known to change the tile; later ones
            // are tested against the scores that the ones before them left
            float thr = quarter_ulp(tile_min(mn, act));
            unsigned left = __ballot_sync(FULL, w0 == first ? lane == 0 : hm != -1.f && !(hm < thr));
            while (left) {
                const int l = __ffs(left) - 1;
                const int x = __shfl_sync(FULL, ev.x, l), xe = __shfl_sync(FULL, ev.y, l);
                const int y = __shfl_sync(FULL, ev.z, l), aw = __shfl_sync(FULL, ev.w, l);
                const bool cov = act && s >= x - nt && s <= xe;
                const float amp = cov ? __int_as_float(aw) : 0.f;
                const float* cp = a.ctcP + (((int64_t)y * nb + blk) * L2 + (s - x + nt)) * MPB_ROWS;
#pragma unroll
                for (int u = 0; u < MPB_ROWS; u += 8) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) w[u + i] = 0.f;
                    if (cov) ld_ctc8(cp + u, w + u);
                }
                mn = INFINITY;
#pragma unroll
                for (int u = 0; u < MPB_ROWS; ++u) {
                    v[u] = __fsub_rn(v[u], __fmul_rn(amp, w[u]));
                    mn = fminf(mn, fabsf(v[u]));
                }
                ++n_app;
                thr = quarter_ulp(tile_min(mn, act));
                left = __ballot_sync(FULL, hm != -1.f && !(hm < thr)) & ~(FULL >> (31 - l));
            }
        }
        if (!changed) {
#pragma unroll
            for (int u = 0; u < MPB_ROWS; ++u) mn = fminf(mn, fabsf(v[u]));
        }
        if (changed && act) {
#pragma unroll
            for (int u = 0; u < MPB_ROWS; u += 8) st_tile8(bp + u, v + u);
        }
        // ---- the column's best Cf and template: q = fl(fl(r*r) * fl(1/nm))
        // errs by 3.01 * 2^-24, so a row more than 8 * 2^-24 below the largest
        // q is not the best; nearly always one row is left, whose quotient is
        // formed exactly
        float q1 = -1.f, q2 = -1.f, rb = 0.f;
        int ub = 0;
#pragma unroll
        for (int u = 0; u < MPB_ROWS; ++u) {
            const float rl = fmaxf(v[u], 0.f);
            const float qv = __fmul_rn(__fmul_rn(rl, rl), s_inv[r0 + u]);
            q2 = fmaxf(q2, fminf(q1, qv));  // the second largest
            if (qv > q1) {
                q1 = qv;
                rb = rl;
                ub = u;
            }
        }
        unsigned long long k = pack_key(0.f, 0);
        const bool inner = act && s >= nt && s < N - nt;  // Cf[:, :nt] = Cf[:, -nt:] = 0
        if (inner)
            k = rb > 0.f ? pack_key(__fdiv_rn(__fmul_rn(rb, rb), s_nm[r0 + ub]), s_perm[r0 + ub]) : pack_key(0.f, s_minp[blk]);
        // several rows left, or quotients too small for the bound: every row
        // (read back from the field) in turn
        if (inner && rb > 0.f && !(q1 >= 1e-30f && q2 < __fmul_rd(q1, 0.99999952316f))) {
            k = 0ull;
#pragma unroll 1
            for (int u = 0; u < nr; ++u) {
                const float rl = fmaxf(__ldcg(bp + u), 0.f);
                k = max(k, pack_key(__fdiv_rn(__fmul_rn(rl, rl), s_nm[r0 + u]), s_perm[r0 + u]));
            }
        }
        if (act) st_key(blk, c, k);
        const float tm = tile_min(mn, act);
        const unsigned cm = __reduce_max_sync(FULL, act ? (unsigned)(k >> 32) : 0u);
        if (lane == 0) {
            s_tmin[q] = tm;
            s_ub[q] = bound_of(__uint_as_float(cm));
            s_app[q] = -1;
        }
    };
    PhaseClock clk{s_clk};
    int r = 0, nlog = 0;
    // counts of the CTAs [from, to) in the round of `tag`, summed over one warp
    auto sum_counts = [&](int from, int to, unsigned tag, bool& bad) {
        const unsigned long long* w = x_cnt + ((tag - 1u) & 1u) * G;
        int sum = 0;
        for (int i = from + lane; i < to; i += 32) {
            unsigned long long wv;
            bad |= !poll_word(w + i, tag, wv, a.status);
            sum += (int)(unsigned)wv;
        }
        return __reduce_add_sync(FULL, sum);
    };
    // ... of round rr, added up: the number of this CTA's first peak and the
    // total. The last warps take 32 words each (polled one after the other,
    // every word would take the latency of a load)
    auto collect = [&](int rr) {
        bool bad = false;
        const int i = (MPL_WARPS - 1 - warp) * 32 + lane;
        if (i - lane < G) {
            unsigned long long wv = 0ull;
            if (i < G) bad = !poll_word(x_cnt + (rr & 1) * G + i, (unsigned)rr + 1u, wv, a.status);
            const int tot = __reduce_add_sync(FULL, (int)(unsigned)wv);
            const int before = __reduce_add_sync(FULL, i < b ? (int)(unsigned)wv : 0);
            if (lane == 0) {
                atomicAdd(&s_total, tot);
                atomicAdd(&s_pref, before);
            }
        }
        return bad;
    };
    // Round rr is counted: its peaks' records, unless it was the last one
    // (none found) or overflows the list (every CTA sees the same total)
    auto finish = [&](int rr) {
        const int total = s_total, base = s_base;
        if (total == 0) return false;
        if (base + total > a.capacity) {
            if (tid == 0) atomicOr(a.status, STATUS_CAPACITY);
            return false;
        }
        const unsigned long long* pk = x_pk + 2 * ((int64_t)(rr & 1) * G * W + lo);
        for (int k = MPL_THREADS - 1 - tid; k < s_own; k += MPL_THREADS) {
            const unsigned long long w0 = ld_word(pk + 2 * k), w1 = ld_word(pk + 2 * k + 1);
            const int i = base + s_pref + k;
            a.sp_x[i] = (int)((w1 >> 24) & 0xFFFFFFFull);
            a.sp_y[i] = (int)(w1 & 0xFFFFFFull);
            a.sp_amp[i] = __uint_as_float((unsigned)w0);
            if (a.sp_round) a.sp_round[i] = rr;
        }
        if (b == 0 && tid == 0) a.round_start[rr] = base;
        return true;
    };
    int todo_all = 1;  // every tile is due: 1 at the start (keys of the initial field), 2 when the log is full
    for (;; ++r) {
        // ---- the tiles that are due, one warp each
        const int n_old = s_qold, qn = todo_all ? qend : s_qn + n_old;
        for (;;) {
            int i = 0;
            if (lane == 0) i = atomicAdd(&s_qnext, 1);
            i = __shfl_sync(FULL, i, 0);
            if (i >= qn) break;
            const int q = todo_all ? i : s_queue[i < n_old ? i : ntile - 1 - (i - n_old)];
            if (todo_all != 2 || s_app[q] >= 0) resolve(q, nlog);
        }
        if (todo_all == 2) nlog = 0;  // nothing is pending: the log starts again
        if (tid == 0 && r > 0) clk.lap(2);
        __syncthreads();
        if (tid == 0 && r > 0) clk.lap(3);
        if (r == 0) {
            // the exchange words are cleared, the keys ready
            if (!grid_sync(a.bar, a.status)) return;
            if (tid == 0) clk.start();
        }
        if (r >= a.max_rounds) {  // the last round's counts
            bool bad = false;
            if (r > 0) bad = collect(r - 1);
            if (__syncthreads_or(bad)) return;
            if (r == 0) break;
            const bool found = finish(r - 1);
            __syncthreads();
            if (!found) --r;
            else if (tid == 0) s_base += s_total;
            break;
        }
        const unsigned tag = (unsigned)r + 1u;
        unsigned long long* cnt_w = x_cnt + (r & 1) * G;                      // this round's counts
        unsigned long long* pk_w = x_pk + 2 * (int64_t)(r & 1) * G * W;       // ... and peaks
        bool bad = false;
        // ---- column maxima (of the chunks that the last round touched) from the
        // keys of the tiles whose bound reaches the threshold (the others', old
        // ones among them, are below it and change no decision); the ones
        // within nt of the edges go to the neighbours
        for (int c = warp; c < nchunk; c += MPL_WARPS) {
            const int s = lo + c * 32 + lane;
            float v;
            if (s_touch[c]) {
                unsigned long long k = 0ull;
                for (int b0 = 0; b0 < nb; b0 += 32) {
                    unsigned loud = __ballot_sync(FULL, b0 + lane < nb && reaches(s_ub[c * nb + b0 + lane], a.th2));
                    while (loud) {
                        unsigned long long kk[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int blk = b0 + __ffs(loud) - 1;
                            kk[u] = loud && s < N ? ld_key(blk, c) : 0ull;
                            loud &= loud - 1u;
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) k = max(k, kk[u]);
                    }
                }
                v = __uint_as_float((unsigned)(k >> 32));
                s_vals[nt + c * 32 + lane] = v;
                s_ival[c * 32 + lane] = (int)(0xFFFFFFFFu - (unsigned)k);
            } else {
                v = s_vals[nt + c * 32 + lane];
            }
            if (s < N && (s < lo + nt || s >= hi - nt)) st_word(x_val + s, ((unsigned long long)tag << 32) | __float_as_uint(v));
        }
        __syncwarp();
        for (int p = tid; p < 2 * nt; p += MPL_THREADS) {
            const int s = p < nt ? lo - nt + p : hi + p - nt;
            float v = 0.f;
            if (s >= 0 && s < N) {
                unsigned long long wv;
                bad |= !poll_word(x_val + s, tag, wv, a.status);
                v = __uint_as_float((unsigned)wv);
            }
            s_vals[p < nt ? p : (hi - lo) + p] = v;
        }
        // the last round's counts, which the others have had this long to send
        if (r > 0) bad |= collect(r - 1);
        if (__syncthreads_or(bad)) return;
        if (r > 0 && !finish(r - 1)) {
            --r;
            break;
        }
        // ---- P: peaks = (Cmax > Th^2) & (|Cmax - Cfmax| < 1e-9), Cmax the
        // maximum over +-nt. Only a column at the threshold and not below its
        // direct neighbours (less margins above the 1e-9) can pass; for those
        // few the whole warp takes the window
        for (int c = warp; c < nchunk; c += MPL_WARPS) {
            const int i = nt + c * 32 + lane, s = lo + c * 32 + lane;
            bool cand = false;
            if (s < hi) {
                const float v = s_vals[i];
                cand = !(v < a.th2 - 1e-8f) && !(v < s_vals[i - 1] - 1e-8f) && !(v < s_vals[i + 1] - 1e-8f);
            }
            unsigned todo = __ballot_sync(FULL, cand), found = 0u;
            while (todo) {
                const int l = __ffs(todo) - 1;
                todo &= todo - 1u;
                const float* wp = s_vals + c * 32 + l;  // the window of column l begins nt columns before it
                float m = 0.f;
                for (int d = lane; d < L2; d += 32) m = fmaxf(m, wp[d]);
                const float cm = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(m)));
                if (cm > a.th2 && fabsf(__fsub_rn(cm, wp[nt])) < 1e-9f) found |= 1u << l;
            }
            if (lane == 0) s_peak[c] = found;
            if ((found >> lane) & 1u) {
                const int row = s_rowof[s_ival[c * 32 + lane]];
                s_amp[c * 32 + lane] = __fdiv_rn(__ldcg(tile_at(row / MPB_ROWS, c) + row % MPB_ROWS), s_nm[row]);
            }
        }
        if (tid == 0) s_qn = s_qold = s_qnext = 0;
        __syncthreads();
        // ---- publish: this CTA's peaks in time order, their count
        int own = 0;
        for (int c0 = 0; c0 < nchunk; c0 += 32) {
            // lane = chunk: the peaks before it; then chunk c's by warp c % MPL_WARPS
            const int n = c0 + lane < nchunk ? __popc(s_peak[c0 + lane]) : 0;
            const int inc = warp_inc_scan(n, lane);
            for (int c = c0 + (warp - c0 % MPL_WARPS + MPL_WARPS) % MPL_WARPS; c < min(nchunk, c0 + 32); c += MPL_WARPS) {
                const unsigned m = s_peak[c];
                const int at = own + __shfl_sync(FULL, inc - n, c - c0);
                if ((m >> lane) & 1u) {
                    unsigned long long* p = pk_w + 2 * ((int64_t)lo + at + __popc(m & ((1u << lane) - 1u)));
                    st_word(p, ((unsigned long long)tag << 32) | __float_as_uint(s_amp[c * 32 + lane]));
                    st_word(p + 1, pack_xy(tag, lo + c * 32 + lane, s_ival[c * 32 + lane]));
                }
            }
            own += __shfl_sync(FULL, inc, 31);
        }
        if (tid == 0) {
            s_base += s_total;  // (the round before's, recorded)
            s_total = s_pref = 0;
            s_own = own;
            st_word(cnt_w + b, ((unsigned long long)tag << 32) | (unsigned)own);
            clk.lap(0);
        }
        // ---- warp 0: the peaks that reach this CTA's columns, the round's
        // even-numbered ones first. Only peaks within 2nt of one another care
        // about their numbers; elsewhere the counts of the CTAs nearby will do
        if (warp == 0) {
            const int r_lo = max(0, b - (nt + W - 1) / W), r_hi = min(G - 1, b + (3 * nt + W - 1) / W);
            int left = 0, near_n = 0;
            for (int i = r_lo + lane; i <= r_hi; i += 32) {
                unsigned long long wv;
                bad |= !poll_word(cnt_w + i, tag, wv, a.status);
                near_n += (int)(unsigned)wv;
                s_rcnt[i - r_lo] = (int)(unsigned)wv;
            }
            bad = __any_sync(FULL, bad);
            near_n = __reduce_add_sync(FULL, near_n);
            if (lane == 0) clk.lap(1);
            int n_new = 0;
            // peak i of the CTAs r_lo .. r_hi taken together (number left + i of the round)
            auto entry = [&](int i, int& x, int& y, float& am) {
                int reg = r_lo;
                while (i >= s_rcnt[reg - r_lo]) i -= s_rcnt[reg++ - r_lo];
                const unsigned long long* p = pk_w + 2 * ((int64_t)reg * W + i);
                unsigned long long w0 = 0, w1 = 0;
                for (unsigned sp = 0; !bad; ++sp) {
                    w0 = ld_word(p);
                    w1 = ld_word(p + 1);
                    if ((unsigned)(w0 >> 32) == tag && (unsigned)(w1 >> 52) == (tag & 0xFFFu)) break;
                    if (sp > MPL_SPIN_LIMIT) {
                        atomicOr(a.status, STATUS_TIMEOUT);
                        bad = true;
                    }
                }
                am = __uint_as_float((unsigned)w0);
                x = (int)((w1 >> 24) & 0xFFFFFFFull);
                y = (int)(w1 & 0xFFFFFFull);
            };
            // peaks i0 .. i0 + 29 (lanes 30 and 31 only look ahead) of one parity
            auto emit = [&](int pass, int i0, int x, int y, float am) {
                const int i = i0 + lane;
                const int x2 = __shfl_down_sync(FULL, x, 2);  // the next peak of the same parity
                const int ehi = min(min(x + nt, N - 1), x2 - nt - 1);
                const bool mine = lane < 30 && i < near_n && ((left + i) & 1) == pass && x - nt < hi && ehi >= lo &&
                                  ehi >= x - nt;
                const unsigned bal = __ballot_sync(FULL, mine);
                const int dst = n_new + __popc(bal & ((1u << lane) - 1u));
                if (mine && dst < a.new_cap) s_new[dst] = make_int4(x, ehi, y, __float_as_int(am));
                n_new += __popc(bal);
            };
            __syncwarp();
            if (!bad && near_n > 0 && near_n <= 30) {  // one group
                int x = INT_MAX / 2, y = 0;
                float am = 0.f;
                if (lane < near_n) entry(lane, x, y, am);
                const int x1 = __shfl_down_sync(FULL, x, 1);
                const bool close = __any_sync(FULL, lane + 1 < near_n && x1 - x <= 2 * nt);
                if (close) left = sum_counts(0, r_lo, tag, bad);
                const int x2 = __shfl_down_sync(FULL, x, 2);
                const int ehi = min(min(x + nt, N - 1), x2 - nt - 1);
                const bool mine = lane < near_n && x - nt < hi && ehi >= lo && ehi >= x - nt, odd = (left + lane) & 1;
                const unsigned me = __ballot_sync(FULL, mine && !odd), mo = __ballot_sync(FULL, mine && odd);
                const unsigned below = (1u << lane) - 1u;
                const int dst = odd ? __popc(me) + __popc(mo & below) : __popc(me & below);
                if (mine && dst < a.new_cap) s_new[dst] = make_int4(x, ehi, y, __float_as_int(am));
                n_new = __popc(me | mo);
            } else if (!bad && near_n > 0) {
                left = sum_counts(0, r_lo, tag, bad);
                __syncwarp();
                const int before = left + sum_counts(r_lo, b, tag, bad), tot = left + sum_counts(r_lo, G, tag, bad);
                for (int pass = 0; pass < 2; ++pass)
                    for (int i0 = 0; i0 < near_n; i0 += 30) {
                        int x = INT_MAX / 2, y = 0;
                        float am = 0.f;
                        if (i0 + lane < near_n) entry(i0 + lane, x, y, am);
                        emit(pass, i0, x, y, am);
                        if (pass == 0) {
                            // more than MP_LIST peaks within 2nt of one another are refused, as by
                            // the other rounds kernel (whose lists they would overflow)
                            const int i = i0 + lane;
                            if (lane < 30 && left + i >= before && left + i < before + s_own && i + MP_LIST - 1 < near_n &&
                                left + i + MP_LIST < tot) {
                                int xq = 0, yq = 0;
                                float aq = 0.f;
                                entry(i + MP_LIST - 1, xq, yq, aq);
                                if (xq <= x + 2 * nt) atomicOr(a.status, STATUS_LIST);
                            }
                            __syncwarp();
                        }
                    }
            }
            if (lane == 0) s_nnew = n_new;
        }
        if (__syncthreads_or(bad)) return;
        const int n_new = min(s_nnew, a.new_cap);
        if (s_nnew > a.new_cap && tid == 0) atomicOr(a.status, STATUS_LIST);
        for (int e = tid; e < n_new; e += MPL_THREADS) s_log[nlog + e] = s_new[e];
        // ---- the tiles the spikes reach (a warp per chunk and group of 32
        // blocks, lane = block): a spike that changes the tile, or any spike on
        // a tile that already waits, becomes pending and raises the tile's
        // bound; a tile whose bound reaches the threshold is due
        for (int it = warp; it < nchunk * nbg; it += MPL_WARPS) {
            const int c = it / nbg, blk = (it - c * nbg) * 32 + lane, q = c * nb + blk;
            const int c_lo = lo + c * 32, c_hi = c_lo + 31;
            bool met = false;
            int app = -1;
            float ub = 0.f, thr = 0.f;
            for (int e = 0; e < n_new; ++e) {
                const int4 ev = s_new[e];
                if (ev.x - nt > c_hi || ev.y < c_lo) continue;
                if (blk < nb) {
                    const float2 hg = lag_bounds(ev, c_lo, blk);
                    if (!met) {
                        app = s_app[q];
                        ub = s_ub[q];
                        thr = quarter_ulp(s_tmin[q]);
                    }
                    const float amp = __int_as_float(ev.w);
                    if (app >= 0 || !(fabsf(__fmul_rn(amp, hg.x)) < thr)) {
                        if (app < 0) app = nlog + e;
                        ub = amp > 0.f ? __fmul_ru(__fadd_ru(ub, __fmul_ru(amp, hg.y)), 1.000001f) : INFINITY;
                    }
                    ++n_items;
                }
                met = true;
            }
            if (lane == 0 && blk < 32) s_touch[c] = met;
            if (met) {
                const bool due = blk < nb && app >= 0 && reaches(ub, a.th2);
                // tiles with spikes from earlier rounds take longer: they go to the
                // front of the queue, the others to its back
                const bool old = due && app < nlog;
                const unsigned b_old = __ballot_sync(FULL, old), b_new = __ballot_sync(FULL, due && !old);
                int at_old = 0, at_new = 0;
                if (lane == 0) {
                    if (b_old) at_old = atomicAdd(&s_qold, __popc(b_old));
                    if (b_new) at_new = atomicAdd(&s_qn, __popc(b_new));
                }
                const unsigned below = (1u << lane) - 1u;
                at_old = __shfl_sync(FULL, at_old, 0) + __popc(b_old & below);
                at_new = __shfl_sync(FULL, at_new, 0) + __popc(b_new & below);
                if (due) s_queue[old ? at_old : ntile - 1 - at_new] = q;
                if (blk < nb) {
                    s_app[q] = app;
                    s_ub[q] = ub;
                }
            }
        }
        nlog += n_new;
        // a log that the next round may overflow: every pending spike is applied
        todo_all = nlog + a.new_cap > a.log_cap ? 2 : 0;
        __syncthreads();
    }
    n_items = __reduce_add_sync(FULL, n_items);
    if (lane == 0 && (n_app | n_items)) {
        atomicAdd(a.counters + 2, n_app);
        atomicAdd(a.counters + 3, n_items);
    }
    if (tid == 0) {
        clk.lap(2);
        clk.flush(a.phase);
    }
    if (b == 0 && tid == 0) {
        a.counters[0] = s_base;
        a.counters[1] = r;
        a.round_start[r] = s_base;
    }
}

// ctct[y, b, l, u] = ctcP[y, perm[MPB_ROWS b + u], l] (zero past T) and
// hg[y, g, b] = {max |ctc|, max(0, max -ctc / sqrt(nm)) rounded up} over the
// block's rows and the group's lags, infinite where a value is NaN. CTA = (y,
// b); the block's rows pass through shared memory, so that both sides are read
// and written in whole lines.
__global__ void __launch_bounds__(128) k_tile_ctc(const float* __restrict__ ctcP, const int32_t* __restrict__ perm,
                                                  const float* __restrict__ nm, int T, int L2,
                                                  float* __restrict__ ctct, float2* __restrict__ hg) {
    extern __shared__ float sm[];  // [MPB_ROWS][L2 | 1]
    __shared__ float s_is[MPB_ROWS];
    const int y = blockIdx.x, blk = blockIdx.y, nb = gridDim.y, ldl = L2 | 1;
    const int r0 = blk * MPB_ROWS, nr = min(MPB_ROWS, T - r0), ng = (L2 + MPB_LAGS - 1) / MPB_LAGS;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < nr) s_is[threadIdx.x] = __frcp_ru(__fsqrt_rd(nm[perm[r0 + threadIdx.x]]));
    for (int u = warp; u < MPB_ROWS; u += 4) {
        const float* p = u < nr ? ctcP + ((int64_t)y * T + perm[r0 + u]) * L2 : nullptr;
        for (int l = lane; l < L2; l += 32) sm[u * ldl + l] = p ? p[l] : 0.f;
    }
    __syncthreads();
    const int64_t o = ((int64_t)y * nb + blk) * L2 * MPB_ROWS;
    for (int e = threadIdx.x; e < L2 * MPB_ROWS; e += blockDim.x)
        ctct[o + e] = sm[(e % MPB_ROWS) * ldl + e / MPB_ROWS];
    for (int gr = threadIdx.x; gr < ng; gr += blockDim.x) {
        float h = 0.f, g = 0.f;
        bool nan = false;
        for (int l = gr * MPB_LAGS; l < min(L2, (gr + 1) * MPB_LAGS); ++l)
            for (int u = 0; u < nr; ++u) {
                const float c = sm[u * ldl + l];
                h = fmaxf(h, fabsf(c));
                g = fmaxf(g, __fmul_ru(fmaxf(-c, 0.f), s_is[u]));
                nan |= c != c;
            }
        hg[((int64_t)y * ng + gr) * nb + blk] = nan ? make_float2(INFINITY, INFINITY) : make_float2(h, g);
    }
}

cudaError_t launch_tile_ctc(const float* ctcP, const int32_t* perm, const float* nm, int32_t T, int32_t L2, float* ctct,
                            float2* hg, cudaStream_t s) {
    const size_t smem = sizeof(float) * MPB_ROWS * (size_t)(L2 | 1);  // at most 33 KB (511 lags)
    k_tile_ctc<<<dim3((unsigned)T, (unsigned)((T + MPB_ROWS - 1) / MPB_ROWS)), 128, smem, s>>>(ctcP, perm, nm, T, L2, ctct, hg);
    return cudaGetLastError();
}

// Score rows [T, N] into the rounds' tiles, one tile per CTA of 256 threads
__global__ void __launch_bounds__(256) k_tile_scores(const float* __restrict__ src, int64_t lds,
                                                     const int32_t* __restrict__ perm, int T, int64_t N,
                                                     float* __restrict__ dst) {
    __shared__ float sm[MPB_ROWS][33];
    const int blk = blockIdx.y, nb = gridDim.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t s = (int64_t)blockIdx.x * 32 + lane;
    for (int u = warp; u < MPB_ROWS; u += 8) {
        const int r = blk * MPB_ROWS + u;
        sm[u][lane] = (r < T && s < N) ? src[(int64_t)perm[r] * lds + s] : 0.f;
    }
    __syncthreads();
    float* d = dst + ((int64_t)blockIdx.x * nb + blk) * 32 * MPB_ROWS;
    for (int e = threadIdx.x; e < 32 * MPB_ROWS; e += 256) d[e] = sm[e % MPB_ROWS][e / MPB_ROWS];
}

cudaError_t launch_tile_scores(const float* src, int64_t lds, const int32_t* perm, int32_t T, int64_t N, float* dst,
                               cudaStream_t s) {
    k_tile_scores<<<dim3((unsigned)((N + 31) / 32), (unsigned)((T + MPB_ROWS - 1) / MPB_ROWS)), 256, 0, s>>>(src, lds, perm,
                                                                                                         T, N, dst);
    return cudaGetLastError();
}

// The rounds' tiles to score rows [T, N] in template order: a CTA takes one
// block's tiles of 4 chunks, so that a row is written 512 bytes at a time.
__global__ void __launch_bounds__(256) k_untile_scores(const float* __restrict__ src, const int32_t* __restrict__ perm,
                                                       int T, int64_t N, float* __restrict__ dst, int64_t ldd) {
    __shared__ float sm[4][32 * (MPB_ROWS + 1)];  // a column's rows padded by one: no bank conflicts either way
    const int blk = blockIdx.y, nb = gridDim.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * 4, nchunk = (N + 31) / 32;
    for (int i = threadIdx.x; i < 4 * 32 * MPB_ROWS / 4; i += 256) {
        const int ch = i / (32 * MPB_ROWS / 4), e = i % (32 * MPB_ROWS / 4) * 4;
        if (c0 + ch < nchunk) {
            const float4 v = __ldcs(reinterpret_cast<const float4*>(src + ((c0 + ch) * nb + blk) * 32 * MPB_ROWS + e));
            float* d = sm[ch] + e + e / MPB_ROWS;
            d[0] = v.x;
            d[1] = v.y;
            d[2] = v.z;
            d[3] = v.w;
        }
    }
    __syncthreads();
    for (int u = warp; u < MPB_ROWS; u += 8) {
        const int r = blk * MPB_ROWS + u;
        if (r >= T) break;
        float* d = dst + (int64_t)__ldg(perm + r) * ldd;
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
            const int64_t s = (c0 + ch) * 32 + lane;
            if (s < N) d[s] = sm[ch][lane * (MPB_ROWS + 1) + u];
        }
    }
}

cudaError_t launch_untile_scores(const float* src, const int32_t* perm, int32_t T, int64_t N, float* dst, int64_t ldd,
                                 cudaStream_t s) {
    const int64_t nchunk = (N + 31) / 32;
    k_untile_scores<<<dim3((unsigned)((nchunk + 3) / 4), (unsigned)((T + MPB_ROWS - 1) / MPB_ROWS)), 256, 0, s>>>(
        src, perm, T, N, dst, ldd);
    return cudaGetLastError();
}

// dst row r = src row perm[r] (N columns each)
__global__ void k_gather_rows(const float* __restrict__ src, int64_t lds, const int32_t* __restrict__ perm,
                              int64_t N, float* __restrict__ dst, int64_t ldd) {
    const int r = blockIdx.y;
    const float* sp = src + (int64_t)__ldg(perm + r) * lds;
    float* dp = dst + (int64_t)r * ldd;
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < N; n += (int64_t)gridDim.x * blockDim.x)
        dp[n] = __ldg(sp + n);
}

cudaError_t launch_gather_rows(const float* src, int64_t lds, const int32_t* perm, int32_t rows, int64_t N,
                               float* dst, int64_t ldd, cudaStream_t s) {
    if (rows <= 0 || N <= 0) return cudaSuccess;
    const unsigned gx = (unsigned)std::min<int64_t>((N + 255) / 256, 64);
    k_gather_rows<<<dim3(gx, (unsigned)rows), 256, 0, s>>>(src, lds, perm, N, dst, ldd);
    return cudaGetLastError();
}

// ---- host side: the slices of a batch of N columns and the shared memory of
// a CTA. Slices are whole 32-column chunks.
static int mpl_width(int64_t N, int grid) {
    const int64_t nchunk = (N + 31) / 32;
    return 32 * (int)((nchunk + grid - 1) / grid);
}

int mp_lazy_grid(int64_t N, int max_grid) {
    const int W = mpl_width(N, max_grid);
    return (int)((N + W - 1) / W);
}

// most spikes one round adds to a CTA's log before STATUS_LIST: MP_LIST per
// 2nt+1 columns over its slice and the nt columns on either side, and the last
// MP_LIST of the round, which no limit watches
static int mpl_new_cap(int W, int nt) { return MP_LIST * ((W + 2 * nt) / (2 * nt + 1) + 2) + 2 * MP_LIST; }

static size_t mpl_smem_bytes(int W, int nt, int T, bool ksmem) {
    const size_t nb = (T + MPB_ROWS - 1) / MPB_ROWS, cpc = W / 32, nt_ = nt, w = W;
    const size_t nc = mpl_new_cap(W, nt), lc = std::max<size_t>(MPL_LOG, nc);
    return 16 * (nc + lc) + (ksmem ? 8 * nb * w : 0) +
           4 * (3 * w + 2 * nt_ + 3 * nb * MPB_ROWS + T + nb + 4 * cpc * nb + 2 * cpc);
}

static size_t mpl_room() { return std::min(shared_memory_room<k_mp_lazy<true>>(), shared_memory_room<k_mp_lazy<false>>()); }

bool mp_lazy_fits(int64_t N, int grid, int T, int nt) {
    if (N >= (1 << 28) || T >= (1 << 24) || grid < 1 || grid > MPL_MAX_GRID) return false;
    return mpl_smem_bytes(mpl_width(N, grid), nt, T, false) <= mpl_room();
}

int64_t mp_lazy_words(int64_t N) { return 2 * MPL_MAX_GRID + 5 * (2 * N + 64); }

template <bool KSMEM>
static cudaError_t launch_lazy(const MPArgs& a, int grid, size_t smem, cudaStream_t s) {
    const cudaError_t e = allow_shared_memory<k_mp_lazy<KSMEM>>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(MPL_THREADS);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_mp_lazy<KSMEM>, a);
}

// max_grid: most CTAs that may run together (the batch's slices take no more)
cudaError_t launch_mp_lazy(MPArgs a, int max_grid, cudaStream_t s) {
    if (!a.perm || !a.hg || !a.bkey || !a.xch || a.nb != (a.T + MPB_ROWS - 1) / MPB_ROWS || a.max_rounds >= 4096 ||
        !mp_lazy_fits(a.N, max_grid, a.T, a.nt))
        return cudaErrorInvalidValue;
    const int W = mpl_width(a.N, max_grid);
    const int grid = mp_lazy_grid(a.N, max_grid);
    if ((3 * a.nt + W - 1) / W + (a.nt + W - 1) / W + 1 > MPL_REGIONS) return cudaErrorInvalidValue;
    a.cols_per_blk = W;
    a.new_cap = mpl_new_cap(W, a.nt);
    a.log_cap = std::max(MPL_LOG, a.new_cap);
    const bool ksmem = mpl_smem_bytes(W, a.nt, a.T, true) <= mpl_room();
    cudaError_t e = cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    const size_t smem = mpl_smem_bytes(W, a.nt, a.T, ksmem);
    return ksmem ? launch_lazy<true>(a, grid, smem, s) : launch_lazy<false>(a, grid, smem, s);
}

}  // namespace lss
