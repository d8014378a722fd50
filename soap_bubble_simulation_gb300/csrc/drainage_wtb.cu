// Temporally blocked drainage step for the GPUDrainageSimulator semantics (drainage.wgsl).
//
// One launch advances the field by K steps with one read and one write of h and Gamma, instead of
// K reads and writes. The pole rows never change in these semantics, so K steps of the 5-point
// stencil only depend on a cone K cells wide around each output cell, which one warp can hold:
//
//  * phi: a warp loads 128 consecutive cells (32 lanes x float4) but keeps only the middle 120.
//    Each level spoils one more cell at each warp edge (the neighbour beyond the warp is not
//    available), so for K <= 4 only lanes 0 and 31 go bad; warps therefore start 120 cells apart
//    and the loads wrap around the row end (Cols: rows whose length is no multiple of 4 gather the
//    four columns at the seam one by one).
//  * theta: a thread sweeps its strip top to bottom as a time-skewed pipeline. After loading row t
//    (level 0) it computes level l of row t - l from a three-row window of level l - 1, for
//    l = 1..K, and stores level K. Each level's windows rotate through three register slots whose
//    index is fixed at compile time (the row loop is unrolled by three), so nothing is copied.
//
// The per-cell arithmetic is wgsl_row(), which gives the bits of the single-step kernel, so K
// launches of one and one launch of this give bit-identical fields.
#include <cuda_runtime.h>

#include <algorithm>

#include "cell.cuh"
#include "sbs_internal.h"
#include "wtb.cuh"

namespace sbs {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerBlock = 4;
constexpr int kSegStride = 120;  // output cells per warp

__device__ __forceinline__ double wtb_block_sum(double v, double *smem) {
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

// At least three blocks per SM: caps the K = 4 pipeline at 168 registers (158-168 used, 12 warps
// per SM). 2048 x 4096, us per pass: 12.0; two blocks (the compiler left to itself) and four (128
// registers, spills) were slower in every form tried (at 14.2 for three: 15.7 and 17.9).
// What bounds it: instruction issue (111 warp instructions per row of four cells a lane and level,
// 54 of them the packed arithmetic) and the FP32 pipes. On the way here from 13.8: the row update's
// cheaper spelling (cell.cuh) 13.05, rows in flight in shared memory 12.4 (ncu: a quarter of the
// warps' time had been waits for the row prefetched into registers), subtractions as FMAs 12.0.
constexpr int kMinBlocksPerSm = 3;

// CAU: the launch also writes the caustic map of its result (wtb_iter); K must be kWtbCausticK.
template <int K, bool VOL, bool MAR, bool RAG, bool CAU = false>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, kMinBlocksPerSm) wtb_wgsl_kernel(const StepArgs a) {
    constexpr int E = CAU ? 1 : 0;  // extra final rows on each side of the strip
    __shared__ double s_red[32];
    __shared__ int s_last;
    extern __shared__ float4 s_dyn[];  // the warps' row rings, coefficients of rows [r0 - K - E, r1 + K + E)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int np = a.np;
    const int seg = blockIdx.x * (blockDim.x >> 5) + warp;
    const int cu = seg * kSegStride - 4 + 4 * lane;  // first column of the lane's window, not wrapped

    Wtb<RAG> w{a.hin, a.cin, a.hout, a.cout, Cols<RAG>(cu, np), s_dyn + warp * (kWtbRingBytes / sizeof(float4)) + lane};
    w.nt = a.nt;
    w.pitch = a.pitch;
    w.r0 = 1 + blockIdx.y * a.rb;
    w.r1 = min(w.r0 + a.rb, a.nt - 1);
    w.store = lane >= 1 && lane <= 30 && cu < np;
    w.k = WgslK{a.b, a.DR2, a.DsR2, a.Gt, a.M, a.dt, a.crit};
    w.vol_w = a.vol_w;
    w.cau_out = a.cau_out;
    w.cau_stride = np;
    w.cau_j0 = w.r0 == 1 ? 0 : w.r0;
    w.cau_j1 = w.r1 == a.nt - 1 ? a.nt : w.r1;
    w.cau_focal = a.cau_focal;
    w.cau_scale = a.cau_scale;
    w.cau_sharp = a.cau_sharp;
    w.cau_branch = a.cau_branch;
    w.sco_base = w.r0 - K - E;
    float4 *s_co = s_dyn + (blockDim.x >> 5) * (kWtbRingBytes / sizeof(float4));
    w.sco = s_co;
    for (int i = threadIdx.x; i < a.rb + 2 * (K + E); i += blockDim.x)
        wtb_coefficients(s_co, i, a.rows, w.sco_base + i, a.nt);
    __syncthreads();

    double vacc = 0.0;
    wtb_strip<K, VOL, MAR, false, CAU, RAG>(w, vacc);

    if (VOL) {
        const double s = wtb_block_sum(vacc, s_red);
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
            double pole = 0.0;  // the frozen pole rows of the input
            for (int j = threadIdx.x; j < np; j += blockDim.x) {
                pole += (double)__ldg(a.hin + j) * __ldg(a.vol_w);
                pole += (double)__ldg(a.hin + (size_t)(a.nt - 1) * a.pitch + j) * __ldg(a.vol_w + a.nt - 1);
            }
            tot = wtb_block_sum(tot, s_red);
            pole = wtb_block_sum(pole, s_red);
            if (threadIdx.x == 0) {
                const unsigned idx = *a.vol_index;
                a.vol_out[idx] = tot + pole;
                *a.vol_index = idx + 1;
                *a.vol_counter = 0u;
                __threadfence();
            }
        }
    }
}

template <int K, bool RAG>
const void *wtb_fn(bool vol, bool mar) {
    if (vol)
        return mar ? (const void *)wtb_wgsl_kernel<K, true, true, RAG>
                   : (const void *)wtb_wgsl_kernel<K, true, false, RAG>;
    return mar ? (const void *)wtb_wgsl_kernel<K, false, true, RAG>
               : (const void *)wtb_wgsl_kernel<K, false, false, RAG>;
}

template <bool RAG>
const void *wtb_pick(int K, bool vol, bool mar, bool cau) {
    if (cau) {
        if (K != kWtbCausticK || vol) return nullptr;
        return mar ? (const void *)wtb_wgsl_kernel<kWtbCausticK, false, true, RAG, true>
                   : (const void *)wtb_wgsl_kernel<kWtbCausticK, false, false, RAG, true>;
    }
    switch (K) {
        case 2:
            return wtb_fn<2, RAG>(vol, mar);
        case 3:
            return wtb_fn<3, RAG>(vol, mar);
        case 4:
            return wtb_fn<4, RAG>(vol, mar);
        default:
            return nullptr;
    }
}

const void *wtb_kernel(int K, bool rag, bool vol, bool mar, bool cau = false) {
    return rag ? wtb_pick<true>(K, vol, mar, cau) : wtb_pick<false>(K, vol, mar, cau);
}

size_t wtb_smem(int warps, int rb, int K, bool cau) {
    return warps * kWtbRingBytes + sizeof(float4) * 2 * (rb + 2 * (K + (cau ? 1 : 0)));
}

// Strips are no taller than this: their coefficients (32 bytes a row) and the rings
// fit the 48 KB that a launch gets without asking. Grids that would need taller ones (over ~3,000
// rows of 64 k columns) run in more than one wave.
constexpr int kMaxStrip = 960;

}  // namespace

bool wtb_supported(int nt, int np) { return np >= 8 && nt >= 3; }

// Segments are spread evenly over blocks of at most kWarpsPerBlock warps. The strip height weighs the
// rows each strip computes twice (2 K of them) against the warps that a grid offers the chip: a
// strip costs rb + 2 K iterations, and an iteration takes 0.41 us on a scheduler with one warp (its
// K levels are a chain) and 0.3 us more for every further one (issue). Measured per pass at
// K = 4, against strips of at least 16 rows that fill three blocks per SM: 64 x 128 3.1 -> 1.5 us (one row),
// 256 x 512 3.3 -> 2.0, 512 x 1024 3.5 -> 2.8, 1024 x 2048 5.8 -> 5.2; 2048 x 4096 keeps its 41 rows.
// Marangoni's chain is longer (its roots): an iteration takes 1.1 us with one warp and with two, 1.45 with
// three. Weighed with the plain times, 500 x 2501 took 8.9 us a pass and 1025 x 2051 13.9 (single steps
// 7.0 and 12.6); with these 5.9 and 8.7 (500 x 2500: 8.2, 5.5).
StepGeom wtb_geometry(int nt, int np, int K, bool mar) {
    StepGeom g{};
    const int segs = (np + kSegStride - 1) / kSegStride;
    g.nbx = (segs + kWarpsPerBlock - 1) / kWarpsPerBlock;
    g.wx = (segs + g.nbx - 1) / g.nbx;
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wtb_kernel(K, np % 4 != 0, false, mar), g.wx * 32,
                                                  wtb_smem(g.wx, 64, K, false));
    if (per_sm < 1) per_sm = 1;
    double best = 0.0;
    for (int rb = 1; rb <= nt - 2 && rb <= kMaxStrip; ++rb) {
        const long long blocks = (long long)g.nbx * ((nt - 2 + rb - 1) / rb);
        const long long each = (blocks + sms - 1) / sms, waves = (each + per_sm - 1) / per_sm;  // per SM
        const double warps = (double)(waves > 1 ? per_sm : each) * g.wx / 4.0;                  // per scheduler
        const double iteration = mar ? std::max(1.1, 0.48 * warps) : warps > 0.9 ? 0.14 + 0.3 * warps : 0.41;
        const double cost = waves * (2.5 + (rb + 2 * K) * iteration);
        if (rb == 1 || cost < best) {
            best = cost;
            g.rb = rb;
        }
    }
    g.nby = (nt - 2 + g.rb - 1) / g.rb;
    g.rb = (nt - 2 + g.nby - 1) / g.nby;  // evened out
    g.cap = per_sm * sms;
    return g;
}

// The same with strips of at least 4 K rows, for a chip that other calls fill too: what counts then is
// the work, and short strips compute 2 K rows beside their own. 16 threads with a handle of 256 x 512
// each, us a run of 256 passes: resident 247, blocked with its own strips 147, with these 101.
StepGeom wtb_crowded(int nt, int K, StepGeom g) {
    const int strips = std::max(g.cap / g.nbx, 1);
    g.rb = std::min(std::max({(nt - 2 + strips - 1) / strips, 4 * K, g.rb}), kMaxStrip);
    g.nby = (nt - 2 + g.rb - 1) / g.rb;
    return g;
}

cudaError_t launch_wtb(int K, const StepArgs &a, const StepGeom &g, cudaStream_t s) {
    const bool cau = a.cau_out != nullptr;
    const void *fn = wtb_kernel(K, a.np % 4 != 0, a.vol_w != nullptr, a.marangoni != 0, cau);
    if (fn == nullptr) return cudaErrorInvalidValue;
    dim3 grid(g.nbx, g.nby), block(g.wx * 32);
    void *args[] = {(void *)&a};
    return cudaLaunchKernel(fn, grid, block, args, wtb_smem(g.wx, g.rb, K, cau), s);
}

}  // namespace sbs
