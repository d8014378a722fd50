// Temporally blocked drainage step for the DrainageSimulator semantics (drainage.rs:298-503):
// one launch advances the field by K steps of the stencil, the pole-ring means and the
// marginal-regeneration fronts, reading and writing h (and its low words) once.
//
// The interior works like the WGSL-semantics kernel (drainage_wtb.cu): a warp holds a 128-column
// window of a strip of rows (keeping the middle 120) and runs a time-skewed register pipeline,
// computing step l of row t - l once step l - 1 of rows t - l - 1 .. t - l + 1 exists.
//
// What the WGSL kernel does not have are the poles: after every step, row 0 becomes the mean of
// the whole of ring 1 and row N-1 the mean of ring N-2 (update_poles, drainage.rs:480-503), and
// the next step's ring-1 update reads it. A row strip is C blocks of W warps that together cover
// the full ring (block b holds segments b W .. b W + W - 1). When a polar strip has advanced ring 1
// or ring N-2 by a step, every block forms the exact integer sum of its part
// of the ring, publishes it in global memory as 32-bit words that each carry the exchange's tag,
// and its first warp reads the C partials as they arrive, so all blocks hold the same mean after
// one trip through L2. The launch is cooperative (every block resident at once), so nobody waits
// for a block that is not running; the wait is bounded all the same. Interior strips start K + 1
// rows from the poles, so their dependency cones stop short of rows 1 and N-2, and never
// synchronise.
//
// An earlier form made every strip one thread-block cluster and gathered the partials through
// distributed shared memory. Clusters of C = 9 blocks are placed whole on one GPC, which at
// 2048 x 4096 left some SMs without a block and the average SM busy 56 % of the launch (33.5 us
// per step); the plain grid keeps every SM at its four blocks.
//
// What bounds it: instruction issue and the FP32 pipes (145 warp instructions per row of four cells
// a lane and level), and the fetch of the unrolled loop (ncu: a fifth of the stalls), so everything
// that runs once a launch is a loop. 2048 x 4096, compensated K = 3, us per step: 17.9 with the
// polar strips in the same pipeline, 256-bit ring sums by every warp and a barrier of four L2 round
// trips per ring mean; 16.8 with today's polar strips and no code for fronts in launches without
// one; 14.9 with the scalar row update (cell.cuh). 128 x 256: 10.2, then 2.9.
//
// Order within one step is the reference's: stencil (rows 1..N-2), the pole means from the
// stencil's ring values, then the fronts thin their cells.
//
// The per-cell arithmetic is cpu_row() (cell.cuh), which gives the bits of the single-step kernel, and
// the front factor the double-float product of the single-step kernel, so K single steps and one
// launch of this give the same bits (the ring sums are exact, which makes them independent of the
// summation order).
#include <cuda_runtime.h>

#include "cell.cuh"
#include "fixsum.cuh"
#include "sbs_internal.h"

namespace sbs {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kSegStride = 120;  // output columns per warp
// Registers per thread: 128 lets four blocks of four warps share an SM. The pipeline needs more
// warps more than fewer spills (an earlier, cluster-launched form at 2048 x 4096: compensated
// K = 2 32.8 us per step capped at 128 registers against 36-38 us with its own ~138).
constexpr int kMaxRegs = 128;
constexpr int kMaxK = 4;
constexpr int kRingWords = 16;  // 64-bit words per exchange slot (nine used, a 128-byte line)
// Rows in flight per lane. Row t + kDepth is requested while row t is consumed, through a
// per-warp ring of kDepth + 1 row slots (hi and lo words) in shared memory filled by per-thread
// 16-byte cp.async copies: each lane waits only for its own copies (cp.async.wait_group), so no
// handshake between warps is needed and the rows in flight cost no registers. Depths 2 to 6
// measured within 2 % of each other.
constexpr int kDepth = 3;
constexpr int kSlots = kDepth + 1;

// Where a polar strip's blocks exchange their ring partials: one slot of kRingWords 64-bit words per
// block, side, and step of the launch; each word is (tag << 32) | payload.
struct RingX {
    unsigned long long *slots;  // [2][kMaxK][nslots][kRingWords] (top, bottom)
    const unsigned *tags;       // this block's tags of this launch's exchanges, [2][kMaxK] in shared memory
    unsigned *status;           // nonzero: an exchange of the launch timed out
    unsigned *status_host;      // host-mapped copy of the status word
    long long limit;            // wait limit, SM cycles
    unsigned narrive;           // partials an exchange waits for (C, plus one in the timeout test)
    int nslots;                 // C + 1
};

template <bool RAG>
struct Ctx {
    const float *hin, *lin;  // input words
    float *hout, *lout;
    Cols<RAG> cols;          // this lane's columns
    const float4 *sco;       // coefficients of rows [t0, t1) in shared memory
    const unsigned *fsel;    // [K][t1 - t0]: front selection nibbles per step and row
    int t0, span;
    int nt, np, pitch, r0, r1;
    bool keep;               // lane owns kept, valid columns (stores and ring sums)
    float b, DR2, dt, crit;
    const double *vol_w;
    unsigned colbits[kMaxK]; // per step: 4 bits per front, the lane's columns inside it
    const TfeStep *tfe;      // the K steps' front records in shared memory
    bool fronts;             // some cell of the warp's window lies inside a front of some step
    float4 *ring;            // this lane's row slots: ring[(slot * 2 + word) * 32]
};

// Requests row r (hi and lo words) into its ring slot and closes the copy group; rows outside
// [0, nt) and past the strip's span are not fetched (the group is then empty).
template <bool X2, bool RAG>
__device__ __forceinline__ void request_row(const Ctx<RAG> &w, int r) {
    if (r >= 0 && r < w.nt && r < w.t0 + w.span) {
        float4 *slot = w.ring + ((r - w.t0) % kSlots) * 64;
        w.cols.template request<false>(slot, w.hin + (size_t)r * w.pitch);
        if (X2) w.cols.template request<false>(slot + 32, w.lin + (size_t)r * w.pitch);
    }
    cp_async_commit();
}

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long *p, unsigned tag, unsigned payload) {
    const unsigned long long v = ((unsigned long long)tag << 32) | payload;
    asm volatile("st.relaxed.gpu.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

constexpr unsigned kWideTag = 0x80000000u;  // the slot holds a 256-bit partial (nine words), not 128 bits (four)
constexpr unsigned kTagMask = 0x7fffffffu;

// The payloads of N adjacent words once all carry `tag`; *tagbits gets the last one's whole tag. The
// words are read together: one trip to L2 (~700 cycles) where a wait for each in turn was five trips
// for a narrow partial and ten for a wide one, at every level. Gives up (and records it) after the
// wait limit, or when another wait of the launch gave up.
template <int N>
__device__ __forceinline__ void wait_words(const unsigned long long *p, unsigned tag, unsigned *w, unsigned *tagbits,
                                           const RingX &x) {
    long long t0 = 0;
    for (unsigned tries = 0;; ++tries) {
        unsigned long long v[N];
        bool there = true;
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = ld_word(p + k);
#pragma unroll
        for (int k = 0; k < N; ++k) {
            there = there && ((unsigned)(v[k] >> 32) & kTagMask) == tag;
            w[k] = (unsigned)v[k];
        }
        *tagbits = (unsigned)(v[N - 1] >> 32);
        if (there) return;
        if (tries == 0) {
            t0 = clock64();
        } else if (clock64() - t0 > x.limit || (tries % 64 == 0 && *(volatile unsigned *)x.status != 0u)) {
            atomicOr(x.status, 1u);
            *(volatile unsigned *)x.status_host = 1u;
            *tagbits = tag;
#pragma unroll
            for (int k = 0; k < N; ++k) w[k] = 0u;
            return;
        }
    }
}

// Exact sum of the lane's cells v (nv of them its own; hi and lo words in X2) over the block, and what
// becomes of it: published in the exchange slot, or, if the strip is one block, turned into the mean.
// 128 bits wide while the words are in fixsum.cuh's range for it, else 256.
struct RingShared {
    Fix128 part[4];
    FixSum fix[4];
    unsigned wide[4];
    float2 mean;
};

template <bool X2>
__device__ __forceinline__ void ring_publish(const Row4 &oh, const Row4 &ol, int nv, const RingX &x, RingShared &s,
                                             double np, double inv_np, int slot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const float vh[4] = {oh.a.x, oh.b.x, oh.a.y, oh.b.y}, vl[4] = {ol.a.x, ol.b.x, ol.a.y, ol.b.y};
    const bool wide = !__all_sync(kFull, fix128_takes<X2>(vh, vl, nv));
    if (!wide) {
        const Fix128 a = fix128_sum<X2>(vh, vl, nv);
        if (lane == 0) s.part[warp] = a;
    } else {
        FixSum f = fix_zero();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            fix_add_float(f, k < nv ? vh[k] : 0.f);
            if (X2) fix_add_float(f, k < nv ? vl[k] : 0.f);
        }
        fix_warp(f);
        if (lane == 0) s.fix[warp] = f;
    }
    if (lane == 0) s.wide[warp] = wide ? 1u : 0u;
    __syncthreads();
    if (warp != 0) return;
    bool any = false;
    for (int j = 0; j < W; ++j) any = any || s.wide[j] != 0u;
    unsigned long long *own = x.slots + ((size_t)slot * x.nslots + blockIdx.x) * kRingWords;
    if (!any) {
        Fix128 a{0u, 0u, 0u, 0u};
        for (int j = 0; j < W; ++j) {
            const Fix128 p = s.part[j];
            fix128_add_words(a, p.w0, p.w1, p.w2, p.w3);
        }
        if (x.narrive == 1u) {
            if (lane == 0) s.mean = fix_mean<X2>(fix128_to_double(a), np, inv_np);
        } else if (lane < 4) {
            st_word(own + lane, x.tags[slot], lane == 0 ? a.w0 : lane == 1 ? a.w1 : lane == 2 ? a.w2 : a.w3);
        }
    } else {
        FixSum f = fix_zero();
        for (int j = 0; j < W; ++j) fix_add(f, s.wide[j] ? s.fix[j] : fix_widen(s.part[j]));
        if (x.narrive == 1u) {
            if (lane == 0) s.mean = fix_mean<X2>(fix_to_double(f), np, inv_np);
        } else if (lane < 9) {
            const unsigned long long limb = lane < 2 ? f.w0 : lane < 4 ? f.w1 : lane < 6 ? f.w2 : f.w3;
            st_word(own + lane, x.tags[slot] | kWideTag, lane == 8 ? f.bad : (unsigned)(limb >> (32 * (lane & 1))));
        }
    }
}

// The mean of the ring published above as the f32 pair (hi, lo): the first warp reads the strip's
// partials and divides, the others wait for it.
template <bool X2>
__device__ __forceinline__ float2 ring_gather(const RingX &x, RingShared &s, double np, double inv_np, int slot) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32 && x.narrive > 1u) {
        const unsigned tag = x.tags[slot];
        Fix128 a{0u, 0u, 0u, 0u};
        FixSum f = fix_zero();
        bool mine = false;  // one of this lane's partials is wide
        for (unsigned j = lane; j < x.narrive; j += 32) {
            const unsigned long long *p = x.slots + ((size_t)slot * x.nslots + j) * kRingWords;
            unsigned w[9], bits;
            wait_words<4>(p, tag, w, &bits, x);
            fix128_add_words(a, w[0], w[1], w[2], w[3]);
            if (bits & kWideTag) {
                mine = true;
                wait_words<5>(p + 4, tag, w + 4, &bits, x);
                fix_add(f, FixSum{((unsigned long long)w[1] << 32) | w[0], ((unsigned long long)w[3] << 32) | w[2],
                                  ((unsigned long long)w[5] << 32) | w[4], ((unsigned long long)w[7] << 32) | w[6],
                                  w[8], 0u});
            } else {
                fix_add(f, fix_widen(Fix128{w[0], w[1], w[2], w[3]}));
            }
        }
        __syncwarp();
        const bool any = __any_sync(kFull, mine);
        double sum;
        if (any) {
            fix_warp(f);
            sum = fix_to_double(f);
        } else {
            sum = fix128_to_double(fix128_warp(a));
        }
        if (lane == 0) s.mean = fix_mean<X2>(sum, np, inv_np);
    }
    __syncthreads();
    return s.mean;
}

// Thins the cells of one row of step l that lie inside a front of that step (drainage.rs:425-460). In the
// pipeline the product is formed for all cells and selected: a branch there would keep the levels'
// chains of an iteration from overlapping.
template <bool X2, bool SKIP, bool RAG>
__device__ __forceinline__ void apply_fronts(const Ctx<RAG> &w, int l, int i, Row4 &oh, Row4 &ol) {
    if (SKIP && !w.fronts) return;
    unsigned x = w.colbits[0];  // step l's, by selection: an index would move the context to local memory
#pragma unroll
    for (int k = 1; k < kMaxK; ++k) x = l == k + 1 ? w.colbits[k] : x;
    x &= w.fsel[(l - 1) * w.span + (i - w.t0)];
    x |= x >> 16;
    x |= x >> 8;
    x |= x >> 4;
    x &= 0xfu;
    if (SKIP && !x) return;
    const float2 fh = f2(w.tfe[l - 1].factor), fl = f2(w.tfe[l - 1].factor_lo);
    auto thin = [&](float2 &h, float2 &lo, bool first, bool second) {
        if (X2) {
            const float2 p = mul2(h, fh);
            const float2 q = fma2(h, fl, fma2(lo, fh, fma2(h, fh, neg2(p))));
            const float2 s = add2(p, q);
            const float2 e = sub2(q, sub2(s, p));
            lo = make_float2(first ? e.x : lo.x, second ? e.y : lo.y);
            h = make_float2(first ? s.x : h.x, second ? s.y : h.y);
        } else {
            const float2 p = mul2(h, fh);
            h = make_float2(first ? p.x : h.x, second ? p.y : h.y);
        }
    };
    thin(oh.a, ol.a, x & 1u, x & 4u);
    thin(oh.b, ol.b, x & 2u, x & 8u);
}

template <bool VOL, bool RAG>
__device__ __forceinline__ void store_row(const Ctx<RAG> &w, int i, const Row4 &oh, const Row4 &ol, bool x2,
                                          double &vacc) {
    const float4 h = row_to4(oh), l = row_to4(ol);
    w.cols.store(w.hout + (size_t)i * w.pitch, h);
    if (x2) w.cols.store(w.lout + (size_t)i * w.pitch, l);
    if (VOL) {
        const double wi = __ldg(w.vol_w + i);
        auto sum = [&](const float4 &v) {
            const int nv = w.cols.valid();
            double s = (double)v.x;
            if (!RAG || nv > 1) s += (double)v.y;
            if (!RAG || nv > 2) s += (double)v.z;
            if (!RAG || nv > 3) s += (double)v.w;
            return s * wi;
        };
        vacc += sum(h);
        if (x2) vacc += sum(l);
    }
}

// One pipeline iteration of an interior strip: receive level-0 row t from the ring, request row
// t + kDepth, then level l of row t - l for l = 1..K. Slot P holds each level's newest row.
template <int K, int P, bool X2, bool VOL, bool FRONTS, bool RAG>
__device__ __forceinline__ void iter(const Ctx<RAG> &w, int t, Row4 (&wh)[K][3], Row4 (&wl)[K][3], double &vacc) {
    constexpr int CUR = (P + 2) % 3, UP = (P + 1) % 3;
    cp_async_wait<kDepth - 1>();  // the groups of rows <= t have landed
    const float4 *slot = w.ring + ((t - w.t0) % kSlots) * 64;
    wh[0][P] = row_of(slot[0]);
    if (X2) wl[0][P] = row_of(slot[32]);
    // the slot of row t + kDepth last held row t - 1, read one iteration ago
    request_row<X2>(w, t + kDepth);
#pragma unroll
    for (int l = 1; l <= K; ++l) {
        const int i = t - l;
        const bool need = i >= w.r0 - (K - l);  // strip-uniform; i < r1 + (K - l) always
        Row4 oh = row_splat(0.f), ol = oh;
        if (need) {
            const Row4 hc = wh[l - 1][CUR], zero = row_splat(0.f);
            const Row4 lc = X2 ? wl[l - 1][CUR] : zero;
            const float hlft = __shfl_up_sync(kFull, hc.b.y, 1), hrgt = __shfl_down_sync(kFull, hc.a.x, 1);
            float llft = 0.f, lrgt = 0.f;
            if (X2) {
                llft = __shfl_up_sync(kFull, lc.b.y, 1);
                lrgt = __shfl_down_sync(kFull, lc.a.x, 1);
            }
            cpu_row<X2>(hc, wh[l - 1][UP], wh[l - 1][P], hlft, hrgt, lc, X2 ? wl[l - 1][UP] : zero,
                        X2 ? wl[l - 1][P] : zero, llft, lrgt, w.sco[i - w.t0], w.b, w.DR2, w.dt, w.crit,
                        oh, ol);
            if (FRONTS) apply_fronts<X2, false>(w, l, i, oh, ol);
        }
        if (l < K) {
            wh[l][P] = oh;
            if (X2) wl[l][P] = ol;
        } else if (need && w.keep) {
            store_row<VOL>(w, i, oh, ol, X2, vacc);
        }
    }
}

// Rows [r0, r1) of strip `by` of `ns`: the two polar strips have K + 1 rows each, the interior strips
// share the rest evenly.
__host__ __device__ inline void strip_rows(int by, int ns, int nt, int K, int &r0, int &r1) {
    if (by == 0) {
        r0 = 0;
        r1 = K + 1;
    } else if (by == ns - 1) {
        r0 = nt - (K + 1);
        r1 = nt;
    } else {
        const long long rest = nt - 2 * (K + 1);
        r0 = K + 1 + (int)((by - 1) * rest / (ns - 2));
        r1 = K + 1 + (int)(by * rest / (ns - 2));
    }
}

// The pipeline over a whole interior strip: its rows are neither poles nor next to one at any level.
template <int K, bool X2, bool VOL, bool FRONTS, bool ROLL, bool RAG>
__device__ __forceinline__ void interior_strip(const Ctx<RAG> &w, double &vacc) {
    Row4 wh[K][3], wl[K][3];
#pragma unroll
    for (int l = 0; l < K; ++l)
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            wh[l][s] = row_splat(0.f);
            wl[l][s] = wh[l][s];
        }
    const int t0 = w.t0, t1 = w.t0 + w.span;
#pragma unroll
    for (int j = 0; j < kDepth; ++j) request_row<X2>(w, t0 + j);
    if (ROLL) {
        // one copy of the iteration, its rows moved down after it: what bounds a launch with fronts is
        // the fetch of its code (ncu at 1024 x 2048: 60 % of the warps' time), as the warps of an SM are
        // in this loop and in the one without fronts at once
#pragma unroll 1
        for (int t = t0; t < t1; ++t) {
            iter<K, 2, X2, VOL, FRONTS>(w, t, wh, wl, vacc);
#pragma unroll
            for (int l = 0; l < K; ++l)
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    wh[l][s] = wh[l][s + 1];
                    wl[l][s] = wl[l][s + 1];
                }
        }
    } else {
        for (int t = t0; t < t1; t += 3) {
            iter<K, 0, X2, VOL, FRONTS>(w, t, wh, wl, vacc);
            if (t + 1 < t1) iter<K, 1, X2, VOL, FRONTS>(w, t + 1, wh, wl, vacc);
            if (t + 2 < t1) iter<K, 2, X2, VOL, FRONTS>(w, t + 2, wh, wl, vacc);
        }
    }
    cp_async_wait<0>();  // every copy was consumed; nothing may still be landing at exit
}

// A polar strip: rows 0 .. K of the top pole, or the last K + 1 rows of the bottom pole (row index r
// counts from the pole; the bottom's table has E negated, as its rows come in the other order). It is
// a strip of the fewest rows: its 2 K + 1 input rows stay in shared memory, every lane with its own
// cells, and are advanced one level at a time, the ring partial under way while the rows beyond ring
// 1 are computed. The row loop is not unrolled: a launch runs this code once, so what it costs is
// mostly its fetch.
template <int K, bool X2, bool VOL, bool FRONTS, bool RAG>
__device__ __forceinline__ void polar_strip(const Ctx<RAG> &w, Row4 *state, const RingX &x, RingShared &s, bool bottom,
                                            double np, double inv_np, double &vacc) {
    auto row = [&](int r) { return bottom ? w.nt - 1 - r : r; };
    auto cell = [&](int r, int f) -> Row4 & { return state[(size_t)(2 * r + f) * blockDim.x]; };
    for (int r = 0; r <= 2 * K; ++r) {
        cell(r, 0) = row_of(w.cols.load(w.hin + (size_t)row(r) * w.pitch));
        if (X2) cell(r, 1) = row_of(w.cols.load(w.lin + (size_t)row(r) * w.pitch));
    }
    const int nv = w.keep ? w.cols.valid() : 0;
    const Row4 zero = row_splat(0.f);
#pragma unroll 1
    for (int lev = 1; lev <= K; ++lev) {
        const int slot = (bottom ? kMaxK : 0) + lev - 1;
        Row4 hp = cell(0, 0), lp = X2 ? cell(0, 1) : zero;  // the row nearer the pole, before this level
        Row4 hc = cell(1, 0), lc = X2 ? cell(1, 1) : zero;
#pragma unroll 1
        for (int r = 1; r <= 2 * K - lev; ++r) {
            const Row4 hn = cell(r + 1, 0), ln = X2 ? cell(r + 1, 1) : zero;
            const float hl = __shfl_up_sync(kFull, hc.b.y, 1), hr = __shfl_down_sync(kFull, hc.a.x, 1);
            const float ll = X2 ? __shfl_up_sync(kFull, lc.b.y, 1) : 0.f;
            const float lr = X2 ? __shfl_down_sync(kFull, lc.a.x, 1) : 0.f;
            const int at = row(r) - w.t0;
            Row4 oh, ol;
            cpu_row<X2>(hc, hp, hn, hl, hr, lc, lp, ln, ll, lr, w.sco[at], w.b, w.DR2, w.dt, w.crit, oh, ol);
            // the pole's mean is of the stencil's values, before the fronts
            if (r == 1) ring_publish<X2>(oh, ol, nv, x, s, np, inv_np, slot);
            if (FRONTS) apply_fronts<X2, true>(w, lev, row(r), oh, ol);
            cell(r, 0) = oh;
            if (X2) cell(r, 1) = ol;
            hp = hc;
            lp = lc;
            hc = hn;
            lc = ln;
        }
        const float2 m = ring_gather<X2>(x, s, np, inv_np, slot);
        cell(0, 0) = row_splat(m.x);
        if (X2) cell(0, 1) = row_splat(m.y);
    }
    if (!w.keep) return;
    for (int r = 0; r <= K; ++r) store_row<VOL>(w, row(r), cell(r, 0), X2 ? cell(r, 1) : zero, X2, vacc);
}

__device__ __forceinline__ double block_sum(double v, double *smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < nw; ++i) t += smem[i];
    __syncthreads();
    return t;
}

// Rows of shared memory per warp: an interior strip's ring or a polar strip's rows.
__host__ __device__ constexpr int state_rows(int K) { return 2 * K + 1 > kSlots ? 2 * K + 1 : kSlots; }

template <int K, bool X2, bool VOL, bool FRONTS, bool RAG>
__global__ void __maxnreg__(kMaxRegs) wtbc_kernel(const StepArgs a) {
    __shared__ TfeStep s_tfe[kMaxK];
    __shared__ unsigned s_tags[2 * kMaxK];
    __shared__ RingX s_x;
    __shared__ RingShared s_ring;
    __shared__ double s_vred[32];
    __shared__ int s_last;
    extern __shared__ float4 s_dyn[];  // the warps' row rings or polar rows, coefficients of rows [t0, t1), front table

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int np = a.np, nt = a.nt;
    const int segs = (np + kSegStride - 1) / kSegStride;
    const int seg = blockIdx.x * W + warp;
    const int cu = seg * kSegStride - 4 + 4 * lane;  // first column of the lane's window, not wrapped
    const bool bottom = blockIdx.y == gridDim.y - 1, polar = blockIdx.y == 0 || bottom;
    int r0, r1;
    strip_rows(blockIdx.y, gridDim.y, nt, K, r0, r1);

    Ctx<RAG> w{a.hin, a.lin, a.hout, a.lout, Cols<RAG>(cu, np)};
    w.nt = nt;
    w.np = np;
    w.pitch = a.pitch;
    w.r0 = r0;
    w.r1 = r1;
    w.t0 = r0 - K;
    w.span = (r1 + K) - (r0 - K);
    w.keep = seg < segs && lane >= 1 && lane <= 30 && cu < np;
    w.b = a.b;
    w.DR2 = a.DR2;
    w.dt = a.dt;
    w.crit = a.crit;
    w.vol_w = a.vol_w;
    if (threadIdx.x == 0)
        s_x = RingX{a.ring_slots, s_tags, a.ring_status, a.status_host, a.wait_cycles, gridDim.x + a.extra,
                    (int)gridDim.x + 1};
    // an exchange's tag is one more than the last one through the slot: every block of a strip has
    // written its own slots equally often, so all of them expect the same tag
    if (polar && threadIdx.x < 2 * kMaxK)
        s_tags[threadIdx.x] = ((unsigned)(ld_word(a.ring_slots + ((size_t)threadIdx.x * (gridDim.x + 1) + blockIdx.x) *
                                                                     kRingWords) >> 32) + 1u) & kTagMask;
    w.ring = s_dyn + (size_t)warp * kSlots * 64 + lane;
    float4 *sco = s_dyn + (size_t)W * state_rows(K) * 64;
    unsigned *fsel = reinterpret_cast<unsigned *>(sco + w.span);
    w.sco = sco;
    w.fsel = fsel;
    w.tfe = s_tfe;
    w.fronts = false;

    if (FRONTS)  // the K steps' front records
        for (int i = threadIdx.x; i < (int)(K * sizeof(TfeStep) / sizeof(int)); i += blockDim.x)
            reinterpret_cast<int *>(s_tfe)[i] = reinterpret_cast<const int *>(a.tfe)[i];
    for (int i = threadIdx.x; i < w.span; i += blockDim.x) {
        const int r = w.t0 + i;
        const float4 q = (r >= 0 && r < nt) ? __ldg(a.rows + r) : make_float4(0.f, 0.f, 0.f, 0.f);
        sco[i] = make_float4(q.x, bottom ? -q.y : q.y, q.z, q.w);
    }
    __syncthreads();
    if (FRONTS) {
        for (int i = threadIdx.x; i < K * w.span; i += blockDim.x) {
            const int l = i / w.span, r = w.t0 + i % w.span;
            unsigned sel = 0;
            for (int f = 0; f < s_tfe[l].nf; ++f)
                if (r >= s_tfe[l].fr[f].x && r <= s_tfe[l].fr[f].y) sel |= 0xfu << (4 * f);
            fsel[i] = sel;
        }
        bool inside = false;  // one of the lane's cells
#pragma unroll
        for (int l = 0; l < kMaxK; ++l) {
            unsigned bits = 0;
            if (l >= K) {
                w.colbits[l] = 0u;
                continue;
            }
            for (int f = 0; f < s_tfe[l].nf; ++f) {
                const int4 fr = s_tfe[l].fr[f];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    int d = w.cols.at(k) - fr.z;
                    if (d < 0) d += np;
                    if (d < fr.w) bits |= 1u << (4 * f + k);
                }
                inside = inside || (bits >> (4 * f) != 0u && fr.x < w.t0 + w.span && fr.y >= w.t0);
            }
            w.colbits[l] = bits;
        }
        w.fronts = __any_sync(kFull, inside);
        __syncthreads();
    }

    double vacc = 0.0;
    if (polar)
        polar_strip<K, X2, VOL, FRONTS>(w, reinterpret_cast<Row4 *>(s_dyn) + threadIdx.x, s_x, s_ring, bottom,
                                        (double)np, a.inv_np, vacc);
    else if (FRONTS && w.fronts)
        interior_strip<K, X2, VOL, true, true>(w, vacc);
    else  // a front is narrow and starts at the equator: most windows of a launch with fronts meet none.
          // Steps with fronts, us each over 4000 late ones, with one unrolled loop for all, with this one
          // unrolled, rolled: 2048 x 4096 22.7, 19.7, 18.7 (plain f32 11.6, 9.8, 10.0: it stays unrolled);
          // 1024 x 2048 14.7, 9.0, 7.8 (plain f32 6.5, 4.5, 4.4)
        interior_strip<K, X2, VOL, false, FRONTS && X2>(w, vacc);

    if (VOL) {
        const double s = block_sum(vacc, s_vred);
        const unsigned nblocks = gridDim.x * gridDim.y;
        const unsigned bid = blockIdx.y * gridDim.x + blockIdx.x;
        if (threadIdx.x == 0) {
            a.vol_partials[bid] = s;
            __threadfence();
            const unsigned tk = atomicAdd(a.vol_counter, 1u);
            s_last = (tk == nblocks - 1);
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            double tot = 0.0;
            for (unsigned i = threadIdx.x; i < nblocks; i += blockDim.x) tot += __ldcg(a.vol_partials + i);
            tot = block_sum(tot, s_vred);
            if (threadIdx.x == 0) {
                const unsigned idx = *a.vol_index;
                a.vol_out[idx] = tot;
                *a.vol_index = idx + 1;
                *a.vol_counter = 0u;
                __threadfence();
            }
        }
    }
}

template <int K, bool X2, bool FRONTS>
const void *pick_vol(bool vol, bool rag) {
    if (rag)
        return vol ? (const void *)wtbc_kernel<K, X2, true, FRONTS, true>
                   : (const void *)wtbc_kernel<K, X2, false, FRONTS, true>;
    return vol ? (const void *)wtbc_kernel<K, X2, true, FRONTS, false>
               : (const void *)wtbc_kernel<K, X2, false, FRONTS, false>;
}

template <int K>
const void *pick_form(bool x2, bool vol, bool fronts, bool rag) {
    if (fronts) return x2 ? pick_vol<K, true, true>(vol, rag) : pick_vol<K, false, true>(vol, rag);
    return x2 ? pick_vol<K, true, false>(vol, rag) : pick_vol<K, false, false>(vol, rag);
}

const void *wtbc_fn(int K, bool x2, bool vol, bool fronts, bool rag) {
    switch (K) {
        case 2:
            return pick_form<2>(x2, vol, fronts, rag);
        case 3:
            return pick_form<3>(x2, vol, fronts, rag);
        case 4:
            return pick_form<4>(x2, vol, fronts, rag);
        default:
            return nullptr;
    }
}

size_t dyn_smem(int W, int span, int K) {
    return sizeof(float4) * ((size_t)W * state_rows(K) * 64 + span) + sizeof(unsigned) * (size_t)K * span;
}
constexpr int kMaxDynSmem = 220 * 1024;

// The tallest of ns strips.
int tallest_strip(int nt, int K, int ns) {
    int rmax = 0;
    for (int by = 0; by < ns; ++by) {
        int r0, r1;
        strip_rows(by, ns, nt, K, r0, r1);
        rmax = r1 - r0 > rmax ? r1 - r0 : rmax;
    }
    return rmax;
}

}  // namespace

// Geometry of the blocked CPU-semantics step: C = ceil(segments / 4) blocks per strip across the
// ring's 120-column segments, the segments spread evenly over their warps, and no more strips than
// fit one wave (the cooperative launch needs every block resident). The two polar strips have
// K + 1 rows; how many interior strips there are weighs the 2 K rows that each computes twice
// against the warps per scheduler, as in the WGSL pipeline's geometry. nby = 0: unsupported.
StepGeom wtbc_geometry(int nt, int np, int K, int x2) {
    StepGeom g{};
    if (K < 2 || K > kMaxK || np < 8 || nt < 2 * (K + 1)) return g;
    const bool rag = np % 4 != 0;
    const int segs = (np + kSegStride - 1) / kSegStride;
    int dev = 0, sms = 148, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return g;
    for (int v = 0; v < 4; ++v)  // the rows alone take up to 36 KB a block
        if (cudaFuncSetAttribute(wtbc_fn(K, x2 != 0, v & 1, v & 2, rag), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kMaxDynSmem) != cudaSuccess) {
            cudaGetLastError();
            return g;
        }
    const int C = (segs + 3) / 4, W = (segs + C - 1) / C;
    const int rest = nt - 2 * (K + 1), most = 4 * sms / C;  // rows of the interior strips; strips of one wave
    int ns = rest > 0 ? 3 : 2, rmax = 0;
    double best = 0.0;
    for (int n = ns; rest > 0 && n <= rest + 2 && n <= most; ++n) {
        const int rows = (rest + n - 3) / (n - 2);
        const double warps = (double)(((long long)C * n + sms - 1) / sms) * W / 4.0;
        const double cost = (rows + 2 * K) * (warps > 0.9 ? 0.14 + 0.3 * warps : 0.41);
        if (n == 3 || cost < best) {
            best = cost;
            ns = n;
        }
    }
    // strips that fit one wave: shrink until the blocks of the real strip height fit
    for (int it = 0; it < 8 && ns >= (rest > 0 ? 3 : 2); ++it) {
        rmax = tallest_strip(nt, K, ns);
        if (dyn_smem(W, rmax + 2 * K, K) > (size_t)kMaxDynSmem) return g;
        int per_sm = 0;
        for (int v = 0; v < 4; ++v) {
            int n = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wtbc_fn(K, x2 != 0, v & 1, v & 2, rag), 32 * W,
                                                              dyn_smem(W, rmax + 2 * K, K)) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            per_sm = v == 0 || n < per_sm ? n : per_sm;
        }
        const int fit = per_sm * sms / C;
        if (fit >= ns) {
            g.wx = W;
            g.nbx = C;
            g.nby = ns;
            g.rb = rmax;
            g.cap = per_sm * sms;
            return g;
        }
        ns = fit;
    }
    return g;
}

size_t wtbc_ring_bytes(const StepGeom &g) {
    return sizeof(unsigned long long) * 2 * kMaxK * (g.nbx + 1) * kRingWords;
}

cudaError_t launch_wtbc(int K, int x2, const StepArgs &a, const StepGeom &g, cudaStream_t s) {
    const void *fn = wtbc_fn(K, x2 != 0, a.vol_w != nullptr, a.tfe != nullptr, a.np % 4 != 0);
    if (fn == nullptr || g.nby < 1 || a.ring_slots == nullptr || a.ring_status == nullptr) return cudaErrorInvalidValue;
    const int span = g.rb + 2 * K;
    void *args[] = {(void *)&a};
    return cudaLaunchCooperativeKernel(fn, dim3(g.nbx, g.nby), dim3(32 * g.wx), args, dyn_smem(g.wx, span, K), s);
}

}  // namespace sbs
