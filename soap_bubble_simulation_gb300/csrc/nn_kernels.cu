// Training-side kernels of the drainage surrogate (include/sbs_nn.h) and its layered forward
// pass: features, the one-channel output layer and its gradients on the FP32 pipe, loss,
// deterministic gradient reduction, Adam, and weight packing. The 3x3 convolutions, their input
// gradients and their weight gradients run on tcgen05 (nn_conv_tc.cu).
//
// Layouts (channel-last, cells = fields x nt x np):
//   features x        BF16 [cells][16]
//   pre-activations y FP32 [cells][32]       activations a BF16 [cells][32]
//   output y4 / gradient g4 FP32 [cells]     layer gradients g BF16 [cells][32]
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "nn.cuh"
#include "nn_kernels.h"
#include "sbs_internal.h"
#include "tc.cuh"

namespace sbs {
namespace nn {
namespace {

__device__ __forceinline__ int refl_row(int i, int nt) { return i < 0 ? 1 : (i >= nt ? nt - 2 : i); }

// ----------------------------------------------------------------------------------- features
__global__ void features_kernel(Fields fs, GridTab g, uint4 *x) {
    const int b = blockIdx.z, i = blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= g.np) return;
    const Field &f = fs.f[b];
    const int nt = g.nt, np = g.np;
    const float *rc = f.h + (size_t)i * f.pitch;
    const float *rn = f.h + (size_t)refl_row(i - 1, nt) * f.pitch;
    const float *rs = f.h + (size_t)refl_row(i + 1, nt) * f.pitch;
    uint4 p0, p1;
    cell_features(rc[j], rn[j], rs[j], rc[j == 0 ? np - 1 : j - 1], rc[j + 1 == np ? 0 : j + 1],
                  f.c[(size_t)i * f.pitch + j], g.rows[i], g.lip[i], f, g, p0, p1);
    uint4 *o = x + (((size_t)b * nt + i) * np + j) * 2;
    o[0] = p0;
    o[1] = p1;
}

// ------------------------------------------------------------ output layer (one channel, FP32)
// y4 = b4 + sum_{tap, ic} W4[tap][ic] a3[src][ic]; with a target, also the masked loss gradient
// g4 = 2 (y4 - target) / n_mask and per-block partial sums of (y4 - target)^2.
struct OutArgs {
    const bf16 *a3;
    const float *w4;  // [9][32], BF16-rounded values
    const float *b4;
    float *y4;
    const float *target;  // null: forward only
    float *g4;
    double *loss_part;
    float inv_nmask2;  // 2 / n_mask
    GridTab g;
    int nf;
};

// The three layer-4 kernels walk columns: a warp takes a few adjacent columns (its lanes also divide
// the 32 channels) of a strip of rows and goes down it, so the taps' weights or sums stay in
// registers and a row's operands are read and widened once for the three rows they meet. They are
// bound by the FP32 issue of 288 multiply-adds per cell (about 100 instructions per warp and row
// against a row's loads); what ran before took a cell's nine taps from shared memory, 36 to 72 reads
// and up to 288 conversions per cell. Eight 256 x 512 fields, microseconds before and now: output
// layer 75 and 44, weight gradient 84 and 33, input gradient 68 and 57.
//
// Work is dealt as (field, strip, column group) units, groups fastest, to the warps of a grid that
// fits the GPU. A strip's rows minimise the rounds of units times a unit's rows, kWalkExtra of which
// stand for the two rows beyond the strip and the start of the pipeline.
constexpr int kWalkWarps = 8, kWalkExtra = 4;
struct Walk {
    int rows, strips, groups, units, blocks;
};

inline cudaError_t plan_walk(int nf, int nt, int np, int cols, int blocks_per_sm, Walk *w) {
    int dev = 0, sms = 1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const long long groups = (np + cols - 1) / cols, warps = (long long)sms * blocks_per_sm * kWalkWarps;
    long long best = 0;
    for (int rows = 4; rows < nt + 4; rows += 4) {
        const long long units = nf * groups * ((nt + rows - 1) / rows);
        const long long cost = (units + warps - 1) / warps * (rows + kWalkExtra);
        if (best == 0 || cost < best) {
            best = cost;
            w->rows = rows;
        }
    }
    w->strips = (nt + w->rows - 1) / w->rows;
    w->groups = (int)groups;
    w->units = nf * w->strips * w->groups;
    w->blocks = (int)std::min<long long>((long long)sms * blocks_per_sm, (w->units + kWalkWarps - 1) / kWalkWarps);
    return cudaSuccess;
}

// A warp's rows arrive through its own ring in shared memory, kWalkRing - 1 rows ahead by per-lane
// cp.async: one row ahead in registers left the loads' latency uncovered (1,600 cycles a row where
// 600 were issued).
constexpr int kWalkRing = 8;
__device__ __forceinline__ void walk_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kWalkRing - 2) : "memory"); }

// Two BF16 values of a word, widened.
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

// Output layer: eight columns a warp, four lanes (8-channel chunks) a cell. Every source row adds
// its nine taps to the three output rows it belongs to; an output row's chunk sums are complete,
// tap by tap and channel by channel, when the row below it has been added. The lane of chunk k
// finishes the strip's rows k, k + 4, ... (loss, gradient), so that work is done by all lanes.
constexpr int kOutCols = 8, kOutBlocksPerSm = 2;  // two blocks: 72 weights and the rows in flight, 128 registers

__global__ void __launch_bounds__(32 * kWalkWarps, kOutBlocksPerSm) out_kernel(OutArgs a, Walk k) {
    __shared__ __align__(16) uint4 ring[kWalkWarps][kWalkRing][4 * (kOutCols + 2)];
    __shared__ double sred[kWalkWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ch = lane & 3;
    const int nt = a.g.nt, np = a.g.np;
    float w[72];  // [tap][channel of the chunk]
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const float4 *p = reinterpret_cast<const float4 *>(a.w4 + t * 32 + ch * 8);
        const float4 u = p[0], v = p[1];
        w[8 * t] = u.x, w[8 * t + 1] = u.y, w[8 * t + 2] = u.z, w[8 * t + 3] = u.w;
        w[8 * t + 4] = v.x, w[8 * t + 5] = v.y, w[8 * t + 6] = v.z, w[8 * t + 7] = v.w;
    }
    const float b4 = *a.b4;
    double l = 0.0;
    for (int u = blockIdx.x * kWalkWarps + warp; u < k.units; u += gridDim.x * kWalkWarps) {
        const int grp = u % k.groups, v = u / k.groups, f = v / k.strips, r0 = (v - f * k.strips) * k.rows;
        const int r1 = min(nt, r0 + k.rows);
        const int j0 = grp * kOutCols, jt = j0 + (lane >> 2);
        const size_t fb = (size_t)f * nt * np;
        const uint4 *src = reinterpret_cast<const uint4 *>(a.a3 + fb * 32);
        // slot cells 0..9 are columns j0 - 1 .. j0 + 8, wrapped
        const int ca = (j0 - 1 + (lane >> 2) + np) % np * 4 + ch, cb = (j0 + 7 + ((lane & 7) >> 2)) % np * 4 + ch;
        auto fill = [&](int r) {
            if (r <= r1) {
                const uint4 *p = src + (size_t)refl_row(r, nt) * np * 4;
                uint4 *dst = ring[warp][(r + 1) % kWalkRing];
                tc::cp_async16(dst + lane, p + ca);
                if (lane < 8) tc::cp_async16(dst + 32 + lane, p + cb);
            }
            tc::cp_async_commit();
        };
        __syncwarp();  // the previous unit's rows are read
#pragma unroll
        for (int d = 0; d < kWalkRing - 1; ++d) fill(r0 - 1 + d);
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, mine = 0.f;  // rows r + 1, r, r - 1; the lane's finished row
        for (int r = r0 - 1; r <= r1; ++r) {
            walk_wait();
            __syncwarp();  // row r is there, row r - 1 is read
            fill(r + kWalkRing - 1);
            const uint4 *row = ring[warp][(r + 1) % kWalkRing] + lane;
            s2 = s1;
            s1 = s0;
            s0 = 0.f;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                const uint4 now = row[4 * x];
                const uint32_t q[4] = {now.x, now.y, now.z, now.w};
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float v = c & 1 ? bf_hi(q[c >> 1]) : bf_lo(q[c >> 1]);
                    s2 = __fmaf_rn(w[8 * (6 + x) + c], v, s2);
                    s1 = __fmaf_rn(w[8 * (3 + x) + c], v, s1);
                    s0 = __fmaf_rn(w[8 * x + c], v, s0);
                }
            }
            const int i = r - 1 - r0;  // the finished row in the strip
            if (i < 0) continue;
            float y = __fadd_rn(s2, __shfl_xor_sync(0xffffffffu, s2, 1));
            y = __fadd_rn(b4, __fadd_rn(y, __shfl_xor_sync(0xffffffffu, y, 2)));
            if ((i & 3) == ch) mine = y;
            if ((i & 3) != 3 && r < r1) continue;
            const int out = r0 + (i & ~3) + ch;
            if (out >= r1 || jt >= np) continue;
            const size_t c = fb + (size_t)out * np + jt;
            a.y4[c] = mine;
            if (a.target) {
                float gr = 0.f;
                if (a.g.rows[out].w != 0.f) {
                    const float dd = __fsub_rn(mine, a.target[c]);
                    l += (double)dd * (double)dd;
                    gr = __fmul_rn(dd, a.inv_nmask2);
                }
                a.g4[c] = gr;
            }
        }
    }
    if (a.target) {
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) sred[warp] = l;
        __syncthreads();
        if (threadIdx.x == 0) {
            double sum = 0.0;
            for (int q = 0; q < kWalkWarps; ++q) sum += sred[q];
            a.loss_part[blockIdx.x] = sum;
        }
    }
}

// dW4[tap][ic] = sum g4[cell] a3[src(cell,tap)][ic], db4 = sum g4. Lanes as in the output layer; a
// lane holds its chunk's 72 sums, and a source cell's eight channels meet the nine gradients of the
// output cells that read it (three rows and columns, kept as the rows go by; zero outside the
// strip). One partial row [289] per block: lanes, then warps, in a fixed order.
struct Wgrad4Args {
    const float *g4;
    const bf16 *a3;
    float *partial;
    GridTab g;
};

constexpr int kW4BlocksPerSm = 2;

__global__ void __launch_bounds__(32 * kWalkWarps, kW4BlocksPerSm) wgrad4_kernel(Wgrad4Args a, Walk k) {
    __shared__ __align__(16) uint4 ring[kWalkWarps][kWalkRing][4 * kOutCols];
    __shared__ float gring[kWalkWarps][kWalkRing][12];
    __shared__ float sp[kWalkWarps][289];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ch = lane & 3;
    const int nt = a.g.nt, np = a.g.np;
    float acc[72];
#pragma unroll
    for (int t = 0; t < 72; ++t) acc[t] = 0.f;
    float gsum = 0.f;
    for (int u = blockIdx.x * kWalkWarps + warp; u < k.units; u += gridDim.x * kWalkWarps) {
        const int grp = u % k.groups, v = u / k.groups, f = v / k.strips, r0 = (v - f * k.strips) * k.rows;
        const int r1 = min(nt, r0 + k.rows);
        const int j0 = grp * kOutCols, n = min(kOutCols, np - j0), q = lane >> 2;
        const size_t fb = (size_t)f * nt * np;
        const uint4 *src = reinterpret_cast<const uint4 *>(a.a3 + fb * 32) + (size_t)min(j0 + q, np - 1) * 4 + ch;
        // slot cells 0..9 are the gradients of columns j0 - 1 .. j0 + 8, wrapped
        const float *gp = a.g4 + fb + (j0 - 1 + lane + np) % np;
        auto fill = [&](int r) {  // source row r and the gradients of row r + 1 (zero outside the strip)
            if (r <= r1) {
                const int s = (r + 2) % kWalkRing;
                tc::cp_async16_zfill(&ring[warp][s][lane], src + (size_t)refl_row(r, nt) * np * 4, q < n);
                const bool ok = r + 1 >= r0 && r + 1 < r1;
                if (lane < 10) tc::cp_async4_zfill(&gring[warp][s][lane], gp + (ok ? (size_t)(r + 1) * np : 0), ok);
            }
            tc::cp_async_commit();
        };
        __syncwarp();  // the previous unit's rows are read
#pragma unroll
        for (int d = 0; d < kWalkRing - 1; ++d) fill(r0 - 1 + d);
        // tap (d, x) of output cell (i, q) reads source (i + d - 1, q + x - 1): g[d][x] is the gradient
        // of row r - d + 1, column q - x + 1
        float g[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) g[0][x] = g[1][x] = 0.f;
        for (int r = r0 - 1; r <= r1; ++r) {
            walk_wait();
            __syncwarp();  // row r is there, row r - 1 is read
            fill(r + kWalkRing - 1);
            const int s = (r + 2) % kWalkRing;
            const uint4 now = ring[warp][s][lane];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                g[2][x] = g[1][x];
                g[1][x] = g[0][x];
                g[0][x] = gring[warp][s][q + 2 - x];
            }
            if (q < n) gsum = __fadd_rn(gsum, g[1][1]);
            const uint32_t w[4] = {now.x, now.y, now.z, now.w};
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const float v = c & 1 ? bf_hi(w[c >> 1]) : bf_lo(w[c >> 1]);
#pragma unroll
                for (int t = 0; t < 9; ++t) acc[8 * t + c] = __fmaf_rn(g[t / 3][t % 3], v, acc[8 * t + c]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < 72; ++t) {
        float v = acc[t];
        for (int o = 4; o < 32; o <<= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane < 4) sp[warp][(t >> 3) * 32 + ch * 8 + (t & 7)] = v;
    }
    for (int o = 4; o < 32; o <<= 1) gsum = __fadd_rn(gsum, __shfl_xor_sync(0xffffffffu, gsum, o));
    if (lane == 0) sp[warp][288] = gsum;
    __syncthreads();
    for (int e = threadIdx.x; e < 289; e += blockDim.x) {
        float v = 0.f;
        for (int q = 0; q < kWalkWarps; ++q) v = __fadd_rn(v, sp[q][e]);
        a.partial[(size_t)blockIdx.x * 289 + e] = v;
    }
}

// g3[cell][ic] = bf16( (sum over the taps that read `cell` of g4[out] W4[tap][ic]) * act'(y3) ):
// four columns a warp, eight lanes (4 channels) a cell, so that a warp's y3 and g3 accesses are
// whole 128-byte lines (a thread per cell, 128 bytes apart, kept the L1 busy for 40 of 68 us). Taps
// in the order t = 0..8, each tap's pole-reflection source right after its own term.
struct Dgrad4Args {
    const float *g4;
    const float *w4;
    const float *y3;
    bf16 *g3;
    GridTab g;
    int act;  // SBS_NN_ACT_*
};

constexpr int kD4Cols = 4, kD4BlocksPerSm = 3;

__global__ void __launch_bounds__(32 * kWalkWarps, kD4BlocksPerSm) dgrad4_kernel(Dgrad4Args a, Walk k) {
    __shared__ __align__(16) float4 ring[kWalkWarps][kWalkRing][8 * kD4Cols];
    __shared__ float gring[kWalkWarps][kWalkRing][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ch = lane & 7;
    const int nt = a.g.nt, np = a.g.np;
    float2 w[9][2];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const float4 u = *reinterpret_cast<const float4 *>(a.w4 + t * 32 + ch * 4);
        w[t][0] = make_float2(u.x, u.y);
        w[t][1] = make_float2(u.z, u.w);
    }
    for (int u = blockIdx.x * kWalkWarps + warp; u < k.units; u += gridDim.x * kWalkWarps) {
        const int grp = u % k.groups, v = u / k.groups, f = v / k.strips, r0 = (v - f * k.strips) * k.rows;
        const int r1 = min(nt, r0 + k.rows);
        const int j0 = grp * kD4Cols, q = lane >> 3, j = min(j0 + q, np - 1);
        const size_t fb = (size_t)f * nt * np;
        const float4 *yp = reinterpret_cast<const float4 *>(a.y3 + fb * 32) + (size_t)j * 8 + ch;
        uint2 *op = reinterpret_cast<uint2 *>(a.g3 + (fb + (size_t)r0 * np) * 32) + (size_t)j * 8 + ch;
        // slot cells 0..5 are the gradients of columns j0 - 1 .. j0 + 4, wrapped
        const float *gp = a.g4 + fb + (j0 - 1 + lane + np) % np;
        auto fill = [&](int r) {  // row r of y3 (from r0 on) and the gradients of row r + 1
            if (r < r1) {
                const int s = (r + 2) % kWalkRing;
                if (r >= r0) tc::cp_async16(&ring[warp][s][lane], yp + (size_t)r * np * 8);
                if (lane < 6)
                    tc::cp_async4_zfill(&gring[warp][s][lane], gp + (size_t)min(max(r + 1, 0), nt - 1) * np, true);
            }
            tc::cp_async_commit();
        };
        __syncwarp();  // the previous unit's rows are read
#pragma unroll
        for (int d = 0; d < kWalkRing - 1; ++d) fill(r0 - 2 + d);
        // tap (dy, dx) reads the gradient of cell (r - dy, j - dx): g[0] is row r + 1, g[2] row r - 1
        float g[3][3];
#pragma unroll
        for (int x = 0; x < 3; ++x) g[0][x] = g[1][x] = 0.f;
        for (int r = r0 - 2; r < r1; ++r) {
            walk_wait();
            __syncwarp();  // row r is there, row r - 1 is read
            fill(r + kWalkRing - 1);
            const int sl = (r + 2) % kWalkRing;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                g[2][x] = g[1][x];
                g[1][x] = g[0][x];
                g[0][x] = gring[warp][sl][q + 2 - x];
            }
            if (r < r0) continue;
            const float4 y = ring[warp][sl][lane];
            float2 s[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            if (r >= 2 && r + 2 < nt) {
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const float2 m = make_float2(g[t / 3][t % 3], g[t / 3][t % 3]);
                    s[0] = __ffma2_rn(m, w[t][0], s[0]);
                    s[1] = __ffma2_rn(m, w[t][1], s[1]);
                }
            } else {  // the rows next to a pole: no row beyond it, the pole's own row reflected into 1 and nt - 2
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const bool own = t < 3 ? r + 1 < nt : t < 6 || r >= 1;
                    const bool top = r == 1 && t < 3, bottom = r == nt - 2 && t >= 6;
                    const float m = g[t / 3][t % 3], e = g[2 - t / 3][t % 3];
                    if (own) {
                        s[0] = __ffma2_rn(make_float2(m, m), w[t][0], s[0]);
                        s[1] = __ffma2_rn(make_float2(m, m), w[t][1], s[1]);
                    }
                    if (top || bottom) {
                        s[0] = __ffma2_rn(make_float2(e, e), w[t][0], s[0]);
                        s[1] = __ffma2_rn(make_float2(e, e), w[t][1], s[1]);
                    }
                }
            }
            const float2 u0 = __fmul2_rn(s[0], act_grad2(a.act, make_float2(y.x, y.y)));
            const float2 u1 = __fmul2_rn(s[1], act_grad2(a.act, make_float2(y.z, y.w)));
            if (j0 + q < np) *op = make_uint2(pack2(u0.x, u0.y), pack2(u1.x, u1.y));
            op += (size_t)np * 8;
        }
    }
}

// Column sums over the blocks' partial rows, in a fixed order: a block of 32 x ROWS threads takes
// 32 adjacent columns; thread (r, c) sums rows r, r + ROWS, ... of column c (coalesced 128-byte
// rows), then the ROWS partial sums are added in order r = 0, 1, ... Returns the sum in the threads
// with r = 0.
constexpr int kRedCols = 32, kRedRows = 8, kRed4Rows = 32;
template <int ROWS>
__device__ __forceinline__ float column_sum(const float *partial, int nblocks, int ncol, int col) {
    __shared__ float s_part[ROWS][kRedCols];
    const int c = threadIdx.x % kRedCols, r = threadIdx.x / kRedCols;
    float s = 0.f;
    if (col < ncol)
        for (int k = r; k < nblocks; k += ROWS) s = __fadd_rn(s, partial[(size_t)k * ncol + col]);
    s_part[r][c] = s;
    __syncthreads();
    float t = 0.f;
    if (r == 0)
        for (int q = 0; q < ROWS; ++q) t = __fadd_rn(t, s_part[q][c]);
    return t;
}

// sum of partial rows scattered into the canonical parameter layout W[tap][oc][ic] (partial column
// oc * 9 * CIN + tap * CIN + ic) and b[oc].
__global__ void __launch_bounds__(kRedCols *kRedRows) reduce_partials_kernel(const float *partial, int nblocks,
                                                                               int ci, int co, float *grad_w,
                                                                               float *grad_b) {
    const int ncol = co * 9 * ci + co;
    const int e = blockIdx.x * kRedCols + threadIdx.x % kRedCols;
    const float s = column_sum<kRedRows>(partial, nblocks, ncol, e);
    if (threadIdx.x >= kRedCols || e >= ncol) return;
    if (e < co * 9 * ci) {
        const int oc = e / (9 * ci), r = e % (9 * ci), t = r / ci, ic = r % ci;
        grad_w[((size_t)t * co + oc) * ci + ic] = s;
    } else {
        grad_b[e - co * 9 * ci] = s;
    }
}

// layer-4 partial rows are [block][tap*32 + ic] then db4
__global__ void __launch_bounds__(kRedCols *kRed4Rows) reduce4_kernel(const float *partial, int nblocks,
                                                                        float *grad_w4, float *grad_b4) {
    const int e = blockIdx.x * kRedCols + threadIdx.x % kRedCols;
    const float s = column_sum<kRed4Rows>(partial, nblocks, 289, e);
    if (threadIdx.x >= kRedCols || e >= 289) return;
    if (e < 288)
        grad_w4[e] = s;
    else
        *grad_b4 = s;
}

// A step that may not be taken (a non-finite loss, a timed-out wait, a step before it that failed) is
// decided here, so that the host need not read the loss before it enqueues the update and what
// follows: every block sums the loss partials, in one fixed order, and comes to the same answer.
// The first block records it for the host and for the steps behind it.
__global__ void __launch_bounds__(256) adam_kernel(float *theta, float *m, float *v, const float *grad, int n, float lr,
                                                   float b1, float b2, float eps, float c1, float c2, StepGate gate) {
    __shared__ double part[256];
    double sum = 0.0;
    for (int k = threadIdx.x; k < gate.nparts; k += 256) sum += gate.parts[k];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    const double loss = part[0] / gate.nmask;
    const unsigned code = gate.prev && gate.prev->code ? gate.prev->code : *gate.err ? 2u : isfinite(loss) ? 0u : 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) *gate.log = StepLog{loss, code, 0u};
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n || code) return;
    const float g = grad[e];
    const float mm = b1 * m[e] + (1.f - b1) * g;
    const float vv = b2 * v[e] + (1.f - b2) * g * g;
    m[e] = mm;
    v[e] = vv;
    theta[e] -= lr * (mm * c1) / (sqrtf(vv * c2) + eps);
}

// BF16 weight layouts for the layered kernels from the FP32 parameter vector.
__global__ void pack_kernel(const float *theta, Packed p) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    // forward layouts [oc][tap*CIN+ic]
    if (e < 32 * 144) {
        const int oc = e / 144, k = e % 144;
        p.wf1[e] = __float2bfloat16_rn(theta[SBS_NN_W1 + ((k / 16) * 32 + oc) * 16 + (k % 16)]);
    }
    if (e < 32 * 288) {
        const int n = e / 288, k = e % 288, t = k / 32, r = k % 32;
        // forward: n = oc, r = ic;  transpose: n = ic, r = oc
        p.wf2[e] = __float2bfloat16_rn(theta[SBS_NN_W2 + (t * 32 + n) * 32 + r]);
        p.wf3[e] = __float2bfloat16_rn(theta[SBS_NN_W3 + (t * 32 + n) * 32 + r]);
        p.wb2[e] = __float2bfloat16_rn(theta[SBS_NN_W2 + (t * 32 + r) * 32 + n]);
        p.wb3[e] = __float2bfloat16_rn(theta[SBS_NN_W3 + (t * 32 + r) * 32 + n]);
    }
    if (e < 288) p.w4[e] = __bfloat162float(__float2bfloat16_rn(theta[SBS_NN_W4 + e]));
    if (e < 32) {
        p.b[e] = theta[SBS_NN_B1 + e];
        p.b[32 + e] = theta[SBS_NN_B2 + e];
        p.b[64 + e] = theta[SBS_NN_B3 + e];
    }
    if (e == 0) p.b[96] = theta[SBS_NN_B4];
}

// h' = max(h + kout y, 0) on rows 1..nt-2, rows 0 and nt-1 copied (one field).
__global__ void apply_kernel(const float *h, size_t pitch_in, const float *y, float kout, int nt, int np, float *out,
                             size_t pitch_out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= np) return;
    const float hc = h[(size_t)i * pitch_in + j];
    float r = hc;
    if (i > 0 && i + 1 < nt) r = fmaxf(__fadd_rn(hc, __fmul_rn(kout, y[(size_t)i * np + j])), 0.f);
    out[(size_t)i * pitch_out + j] = r;
}

// target[b][cell] = (h_next - h) / kout for a batch of snapshot pairs
struct TargetArgs {
    const float *h0[kMaxFields];
    const float *h1[kMaxFields];
    float kout[kMaxFields];
};

__global__ void target_kernel(TargetArgs t, int nt, int np, float *target) {
    const int b = blockIdx.z, i = blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= np) return;
    const size_t k = (size_t)i * np + j;
    target[((size_t)b * nt) * np + k] = __fdiv_rn(__fsub_rn(t.h1[b][k], t.h0[b][k]), t.kout[b]);
}

// max |a - b| and max |b| over the masked rows (rows[i].w != 0) as float bit patterns (both are
// non-negative, so unsigned order is float order); a NaN difference counts as +inf.
// Bound by the reads, which the cache mostly serves. A block walks (row, 1024 columns) pieces and adds
// one pair of atomics at its end; with a pair from every warp of a block per row, 131072 updates of the
// same two words took 173 us of a 2048 x 2048 check, the pieces take 19.
__global__ void __launch_bounds__(256) masked_err_kernel(const float *__restrict__ a, size_t pa,
                                                         const float *__restrict__ b, size_t pb,
                                                         const float4 *__restrict__ rows, int nt, int np,
                                                         unsigned *out) {
    const int segs = (np + 1023) / 1024, units = nt * segs;
    float d = 0.f, m = 0.f;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
        const int i = u / segs, j0 = (u - i * segs) * 1024 + threadIdx.x;
        if (rows[i].w == 0.f) continue;
        float va[4], vb[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int j = j0 + 256 * k;
            va[k] = j < np ? a[(size_t)i * pa + j] : 0.f;
            vb[k] = j < np ? b[(size_t)i * pb + j] : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float e = fabsf(__fsub_rn(va[k], vb[k]));
            if (e != e) e = __int_as_float(0x7f800000);
            d = fmaxf(d, e);
            m = fmaxf(m, fabsf(vb[k]));
        }
    }
    __shared__ unsigned best[2];
    if (threadIdx.x < 2) best[threadIdx.x] = 0u;
    __syncthreads();
    // neither is negative or NaN, so the bits are ordered like the values
    const unsigned wd = __reduce_max_sync(0xffffffffu, __float_as_uint(d));
    const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&best[0], wd);
        atomicMax(&best[1], wm);
    }
    __syncthreads();
    if (threadIdx.x < 2) atomicMax(out + threadIdx.x, best[threadIdx.x]);
}

}  // namespace

// ------------------------------------------------------------------------------ host wrappers
cudaError_t features(const Fields &fs, int nf, const GridTab &g, bf16 *x, cudaStream_t st) {
    dim3 grid((g.np + 127) / 128, g.nt, nf);
    features_kernel<<<grid, 128, 0, st>>>(fs, g, (uint4 *)x);
    return cudaGetLastError();
}


cudaError_t conv_backward_weight(int layer, const bf16 *g, const bf16 *x, float *partial, int nblocks, float *grad,
                                 unsigned *err, int nf, int nt, int np, cudaStream_t st) {
    const int ci = layer == 1 ? 16 : 32;
    const int ow = layer == 1 ? SBS_NN_W1 : (layer == 2 ? SBS_NN_W2 : SBS_NN_W3);
    const int ob = layer == 1 ? SBS_NN_B1 : (layer == 2 ? SBS_NN_B2 : SBS_NN_B3);
    cudaError_t e = wgrad_tc(ci, g, x, partial, &nblocks, err, nf, nt, np, st);
    if (e != cudaSuccess) return e;
    const int ncol = 32 * 9 * ci + 32;
    reduce_partials_kernel<<<(ncol + kRedCols - 1) / kRedCols, kRedCols * kRedRows, 0, st>>>(partial, nblocks, ci, 32,
                                                                                         grad + ow, grad + ob);
    return cudaGetLastError();
}

cudaError_t output_layer(const bf16 *a3, const Packed &p, float *y4, const float *target, float *g4,
                         double *loss_part, float inv_nmask2, const GridTab &g, int nf, cudaStream_t st,
                         int *nblocks_out) {
    OutArgs o{};
    o.a3 = a3;
    o.w4 = p.w4;
    o.y4 = y4;
    o.target = target;
    o.g4 = g4;
    o.loss_part = loss_part;
    o.inv_nmask2 = inv_nmask2;
    o.g = g;
    o.nf = nf;
    o.b4 = p.b + 96;
    Walk k{};
    const cudaError_t e = plan_walk(nf, g.nt, g.np, kOutCols, kOutBlocksPerSm, &k);
    if (e != cudaSuccess) return e;
    out_kernel<<<k.blocks, 32 * kWalkWarps, 0, st>>>(o, k);
    if (nblocks_out) *nblocks_out = k.blocks;
    return cudaGetLastError();
}

cudaError_t output_backward(const float *g4, const bf16 *a3, const float *y3, const Packed &p, bf16 *g3,
                            float *partial, float *grad, const GridTab &g, int nf, cudaStream_t st) {
    Wgrad4Args w{};
    w.g4 = g4;
    w.a3 = a3;
    w.partial = partial;
    w.g = g;
    Walk k{};
    cudaError_t e = plan_walk(nf, g.nt, g.np, kOutCols, kW4BlocksPerSm, &k);
    if (e != cudaSuccess) return e;
    // partial rows of 289 floats in a buffer of nblocks (two per SM) x (32 x 9 x 32 + 32) floats
    static_assert(kW4BlocksPerSm * 289 <= 2 * (32 * 9 * 32 + 32), "layer-4 partial rows fit the buffer");
    wgrad4_kernel<<<k.blocks, 32 * kWalkWarps, 0, st>>>(w, k);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    reduce4_kernel<<<(289 + kRedCols - 1) / kRedCols, kRedCols * kRed4Rows, 0, st>>>(
        partial, k.blocks, grad + SBS_NN_W4, grad + SBS_NN_B4);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    Dgrad4Args d{};
    d.g4 = g4;
    d.w4 = p.w4;
    d.y3 = y3;
    d.g3 = g3;
    d.g = g;
    d.act = p.act;
    if ((e = plan_walk(nf, g.nt, g.np, kD4Cols, kD4BlocksPerSm, &k)) != cudaSuccess) return e;
    dgrad4_kernel<<<k.blocks, 32 * kWalkWarps, 0, st>>>(d, k);
    return cudaGetLastError();
}

cudaError_t adam(float *theta, float *m, float *v, const float *grad, float lr, float b1, float b2, float eps,
                 int step, const StepGate &gate, cudaStream_t st) {
    const float c1 = (float)(1.0 / (1.0 - std::pow((double)b1, step)));
    const float c2 = (float)(1.0 / (1.0 - std::pow((double)b2, step)));
    adam_kernel<<<(SBS_NN_PARAMS + 255) / 256, 256, 0, st>>>(theta, m, v, grad, SBS_NN_PARAMS, lr, b1, b2, eps, c1,
                                                             c2, gate);
    return cudaGetLastError();
}

cudaError_t pack(const float *theta, const Packed &p, cudaStream_t st) {
    pack_kernel<<<(32 * 288 + 255) / 256, 256, 0, st>>>(theta, p);
    return cudaGetLastError();
}

cudaError_t apply(const float *h, size_t pitch_in, const float *y, float kout, int nt, int np, float *out,
                  size_t pitch_out, cudaStream_t st) {
    dim3 grid((np + 127) / 128, nt);
    apply_kernel<<<grid, 128, 0, st>>>(h, pitch_in, y, kout, nt, np, out, pitch_out);
    return cudaGetLastError();
}

cudaError_t targets(const float *const *h0, const float *const *h1, const float *kout, int nf, int nt, int np,
                    float *target, cudaStream_t st) {
    TargetArgs t{};
    for (int b = 0; b < nf; ++b) {
        t.h0[b] = h0[b];
        t.h1[b] = h1[b];
        t.kout[b] = kout[b];
    }
    dim3 grid((np + 127) / 128, nt, nf);
    target_kernel<<<grid, 128, 0, st>>>(t, nt, np, target);
    return cudaGetLastError();
}

cudaError_t masked_error(const float *a, size_t pa, const float *b, size_t pb, const GridTab &g, unsigned *out2,
                         cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(out2, 0, 2 * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 1;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const size_t units = (size_t)g.nt * ((g.np + 1023) / 1024);
    masked_err_kernel<<<(unsigned)std::min(units, (size_t)sms * 4), 256, 0, st>>>(a, pa, b, pb, g.rows, g.nt, g.np, out2);
    return cudaGetLastError();
}

}  // namespace nn
}  // namespace sbs
