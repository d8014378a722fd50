// One row of the time-skewed register pipeline that advances a warp's 128-column window of the
// WGSL-semantics fields by K steps (used by the single-bubble and the batched foam kernels, so
// both round identically). See drainage_wtb.cu for the scheme.
#pragma once

#include <cuda_runtime.h>

#include "caustics.cuh"
#include "cell.cuh"

namespace sbs {

template <bool RAG>
struct Wtb {
    const float *hin, *cin;  // input fields
    float *hout, *cout;      // output fields
    Cols<RAG> cols;          // this lane's columns
    float4 *ring;            // this lane's row slots: ring[(slot * 2 + field) * 32]
    const float4 *sco;       // this strip's per-row coefficients in shared memory (two per row), from row sco_base
    int sco_base;
    int nt, pitch, r0, r1;
    bool store;
    WgslK k;
    const double *vol_w;
    // caustic map of the launch's result (CAU launches only)
    float *cau_out;          // map (rows of cau_stride floats)
    int cau_stride;
    int cau_j0, cau_j1;      // map rows this strip writes
    float cau_focal, cau_scale, cau_sharp, cau_branch;
};

// The coefficients of row r, doubled as wgsl_row takes them, into a strip's table (zero outside the grid).
__device__ __forceinline__ void wtb_coefficients(float4 *sco, int i, const float4 *rows, int r, int nt) {
    const float4 q = (r >= 0 && r < nt) ? __ldg(rows + r) : make_float4(0.f, 0.f, 0.f, 0.f);
    sco[2 * i] = make_float4(q.x, q.x, q.y, q.y);
    sco[2 * i + 1] = make_float4(q.z, q.z, q.w, q.w);
}

// Caustic map row j (caustics_compute.wgsl:87-111) from the final rows above (a), at (b) and below
// (c) j; phi neighbours by shuffle (all lanes call; kept lanes store).
template <bool RAG>
__device__ __forceinline__ void wtb_caustic_row(const Wtb<RAG> &w, int j, const Row4 &ra, const Row4 &rb,
                                                const Row4 &rc) {
    const float4 a = row_to4(ra), b = row_to4(rb), c = row_to4(rc);
    const float al = __shfl_up_sync(0xffffffffu, a.w, 1), ar = __shfl_down_sync(0xffffffffu, a.x, 1);
    const float bl = __shfl_up_sync(0xffffffffu, b.w, 1), br = __shfl_down_sync(0xffffffffu, b.x, 1);
    const float cl = __shfl_up_sync(0xffffffffu, c.w, 1), cr = __shfl_down_sync(0xffffffffu, c.x, 1);
    const float av[6] = {al, a.x, a.y, a.z, a.w, ar}, bv[6] = {bl, b.x, b.y, b.z, b.w, br};
    const float cv[6] = {cl, c.x, c.y, c.z, c.w, cr};
    float o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        o[k] = caustic_intensity(w.cau_focal, w.cau_scale, w.cau_sharp, w.cau_branch,
                                 CausticRow{av[k], av[k + 1], av[k + 2]}, CausticRow{bv[k], bv[k + 1], bv[k + 2]},
                                 CausticRow{cv[k], cv[k + 1], cv[k + 2]});
    if (!w.store) return;
    float *row = w.cau_out + (size_t)j * w.cau_stride;
    if (!RAG) {
        w.cols.store(row, make_float4(o[0], o[1], o[2], o[3]));
    } else {  // the map's rows are np floats: not aligned to anything
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < w.cols.valid()) row[w.cols.at(k)] = o[k];
    }
}

// Rows in flight per lane: row t + kWtbDepth is requested while row t is consumed, through a per-warp
// ring of kWtbDepth + 1 row slots (both fields) in shared memory. The rows in flight cost no
// registers; one row ahead in registers left a quarter of the warps' time waiting for memory.
constexpr int kWtbDepth = 3;
constexpr int kWtbSlots = kWtbDepth + 1;
constexpr size_t kWtbRingBytes = sizeof(float4) * kWtbSlots * 2 * 32;  // per warp

// Requests row r and closes the copy group (empty for rows outside the grid or past row `end`).
template <bool CG, bool RAG>
__device__ __forceinline__ void wtb_request(const Wtb<RAG> &w, int r, int t0, int end) {
    if (r >= 0 && r < end) {
        float4 *slot = w.ring + ((r - t0) % kWtbSlots) * 64;
        w.cols.template request<CG>(slot, w.hin + (size_t)r * w.pitch);
        w.cols.template request<CG>(slot + 32, w.cin + (size_t)r * w.pitch);
    }
    cp_async_commit();
}

// One pipeline iteration: take level-0 row t, then compute level l of row t - l for l = 1..K.
// Slot P holds the row most recently written to each level's window.
// CAU: the launch also writes the caustic map of its result. Every level then covers one more row
// on each side (the strip's final rows r0 - 1 and r1 are needed), wk keeps the last three final
// rows, and map row j is written once final row j + 1 exists (theta clamped at the poles).
// STEADY: the caller guarantees that every level's row lies inside the strip's window and the
// grid, none is a pole row, and the final row is one of the strip's own rows; the iteration then
// skips those tests (same arithmetic, same bits).
template <int K, int P, bool VOL, bool MAR, bool CG = false, bool CAU = false, bool STEADY = false, bool RAG = false>
__device__ __forceinline__ void wtb_iter(const Wtb<RAG> &w, int t, int t0, int end, Row4 (&wh)[K][3],
                                         Row4 (&wc)[K][3], double &vacc, Row4 *wk = nullptr) {
    constexpr int CUR = (P + 2) % 3, UP = (P + 1) % 3;
    constexpr int E = CAU ? 1 : 0;
    cp_async_wait<kWtbDepth - 1>();  // the groups of rows <= t have landed
    wh[0][P] = row_splat(0.f);
    wc[0][P] = wh[0][P];
    if (STEADY || (t >= 0 && t < end)) {
        const float4 *slot = w.ring + ((t - t0) % kWtbSlots) * 64;
        wh[0][P] = row_of(slot[0]);
        wc[0][P] = row_of(slot[32]);
    }
    wtb_request<CG>(w, t + kWtbDepth, t0, end);  // into the slot of row t - 1, read one iteration ago
#pragma unroll
    for (int l = 1; l <= K; ++l) {
        const int i = t - l;
        const bool need =
            STEADY || (i >= w.r0 - (K - l) - E && i < w.r1 + (K - l) + E && i >= 0 && i < w.nt);  // warp-uniform
        Row4 oh = row_splat(0.f), oc = oh;
        if (need) {
            const Row4 hc = wh[l - 1][CUR], cc = wc[l - 1][CUR];
            if (!STEADY && (i == 0 || i == w.nt - 1)) {  // pole rows are frozen (drainage.wgsl:85-89)
                oh = hc;
                oc = cc;
            } else {
                const float4 *co = w.sco + 2 * (i - w.sco_base);
                const float hl = __shfl_up_sync(0xffffffffu, hc.b.y, 1), hr = __shfl_down_sync(0xffffffffu, hc.a.x, 1);
                const float cl = __shfl_up_sync(0xffffffffu, cc.b.y, 1), cr = __shfl_down_sync(0xffffffffu, cc.a.x, 1);
                wgsl_row<MAR>(hc, wh[l - 1][UP], wh[l - 1][P], hl, hr, cc, wc[l - 1][UP], wc[l - 1][P], cl, cr, co[0],
                              co[1], w.k, oh, oc);
            }
        }
        if (l < K) {
            wh[l][P] = oh;
            wc[l][P] = oc;
        } else {
            if (STEADY ? w.store : (need && i >= w.r0 && i < w.r1 && w.store)) {
                const float4 o = row_to4(oh);
                w.cols.store(w.hout + (size_t)i * w.pitch, o);
                w.cols.store(w.cout + (size_t)i * w.pitch, row_to4(oc));
                if (VOL) {
                    const int nv = w.cols.valid();
                    double s = (double)o.x;
                    if (!RAG || nv > 1) s += (double)o.y;
                    if (!RAG || nv > 2) s += (double)o.z;
                    if (!RAG || nv > 3) s += (double)o.w;
                    vacc += s * __ldg(w.vol_w + i);
                }
            }
            if (CAU) {
                wk[P] = oh;
                const int j = i - 1;  // warp-uniform
                if (j >= w.cau_j0 && j < w.cau_j1) wtb_caustic_row(w, j, j == 0 ? wk[CUR] : wk[UP], wk[CUR], wk[P]);
                if (i == w.nt - 1 && i >= w.cau_j0 && i < w.cau_j1) wtb_caustic_row(w, i, wk[CUR], wk[P], wk[P]);
            }
        }
    }
}

// A warp's strip from its first level-0 row to its last stored row. Iterations whose rows all lie
// inside the strip and the grid run STEADY. Register slots rotate by three, so the row loop is
// unrolled by three.
template <int K, bool VOL, bool MAR, bool CG, bool CAU, bool RAG>
__device__ __forceinline__ void wtb_strip(const Wtb<RAG> &w, double &vacc) {
    constexpr int E = CAU ? 1 : 0;
    Row4 wh[K][3], wc[K][3], wk[3];  // wk: the last three final rows (CAU)
#pragma unroll
    for (int s = 0; s < 3; ++s) {
#pragma unroll
        for (int l = 0; l < K; ++l) {
            wh[l][s] = row_splat(0.f);
            wc[l][s] = wh[l][s];
        }
        wk[s] = row_splat(0.f);
    }
    const int t0 = w.r0 - K - E, t1 = w.r1 + K + E;  // level-0 rows [t0, t1)
    const int end = min(t1, w.nt);
#pragma unroll
    for (int j = 0; j < kWtbDepth; ++j) wtb_request<CG>(w, t0 + j, t0, end);
    // iterations t in [ts, te) are steady: every level's row t - l inside [r0 - (K - l), r1 + (K - l))
    // and in 1..nt-2, the final row t - K in [r0, r1), row t < nt
    const int ts = w.r0 + K, te = min(w.r1 + K, w.nt);
    for (int t = t0; t < t1; t += 3) {
        if (!CAU && t >= ts && t + 2 < te) {
            wtb_iter<K, 0, VOL, MAR, CG, false, true>(w, t, t0, end, wh, wc, vacc);
            wtb_iter<K, 1, VOL, MAR, CG, false, true>(w, t + 1, t0, end, wh, wc, vacc);
            wtb_iter<K, 2, VOL, MAR, CG, false, true>(w, t + 2, t0, end, wh, wc, vacc);
            continue;
        }
        wtb_iter<K, 0, VOL, MAR, CG, CAU>(w, t, t0, end, wh, wc, vacc, wk);
        if (t + 1 < t1) wtb_iter<K, 1, VOL, MAR, CG, CAU>(w, t + 1, t0, end, wh, wc, vacc, wk);
        if (t + 2 < t1) wtb_iter<K, 2, VOL, MAR, CG, CAU>(w, t + 2, t0, end, wh, wc, vacc, wk);
    }
    cp_async_wait<0>();  // every row was consumed; nothing may still be landing when the ring is used again
}

}  // namespace sbs
