// Drainage steps of a grid that fits the chip's shared memory: one launch advances the field by a
// whole chunk of steps, for both semantics (drainage.rs:298-503 and drainage.wgsl:72-202).
//
// A block owns a few theta rows over the whole ring (a warp 128 columns of them, four per lane) and
// keeps them in shared memory from the first step to the last; every lane reads and writes only its
// own cells there. Per step it needs from outside
//  * the columns next to its warps' edges: through shared memory, one __syncthreads a step;
//  * the row above its first and below its last one: from the neighbouring blocks, through global
//    memory (L2). Every 32-bit value travels in a 64-bit word with the number of its step, so a
//    reader polls the data itself: one trip through L2 instead of data, fence, flag and data again.
//    Two buffers by step parity are enough: a block writes step s + 2 only after it has read its
//    neighbours' s + 1, which they wrote after reading its s;
//  * CPU semantics: the pole value, the mean of ring 1 (or N - 2): the block that owns the ring sums
//    it exactly (fixsum.cuh), its first warp divides.
// The launch is cooperative (every block is resident), and every wait is bounded.
//
// What bounds it: on small grids the chain of one step (a row's update, ~300 cycles, and the trip
// through L2, ~900; with poles also the ring's sum and division), on large ones instruction issue:
// nothing is computed twice, whereas the temporally blocked kernels recompute their strips' 2 K
// edge rows and pay, at every launch, the fetch of ~50 KB of unrolled code (ncu: 80 % of the
// warps' time at 128 x 256). The rows of a block are a loop here, not unrolled, for the same
// reason. Us per step, at the start (blocked or single steps), with the blocked kernels of today, and
// here: CPU semantics 128 x 256 10.2, 2.9, 2.0; 512 x 1024 9.9, 4.6, 3.5; WGSL semantics 64 x 128
// 3.4, 1.34, 0.92; 512 x 1024 3.9, 2.8, 2.6; 1024 x 2048 6.5, 5.2, 4.1; with Marangoni 517 x 1037
// 6.2, 4.6, 3.5.
//
// The arithmetic is wgsl_row() / cpu_row() (cell.cuh), the blocked kernels' own: the same bits.
#include <cuda_runtime.h>

#include "cell.cuh"
#include "fixsum.cuh"
#include "sbs_internal.h"

namespace sbs {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxWarps = 16;  // 512 threads: rows of up to 2048 columns, 128 registers a thread
constexpr size_t kMaxSmem = 220 * 1024;

__device__ __forceinline__ void st_pair(unsigned long long *p, unsigned tag, float u, float v) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(u)),
                 "l"(t | __float_as_uint(v))
                 : "memory");
}
// The payloads of two words; false unless both carry `tag`.
__device__ __forceinline__ bool ld_pair(const unsigned long long *p, unsigned tag, float &u, float &v) {
    unsigned long long x, y;
    asm volatile("ld.relaxed.gpu.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
    u = __uint_as_float((unsigned)x);
    v = __uint_as_float((unsigned)y);
    return (unsigned)(x >> 32) == tag && (unsigned)(y >> 32) == tag;
}

// Rows [r0, r1) of block b of nb (rows 1 .. nt - 2, shared evenly).
__device__ __forceinline__ void block_rows(int b, int nb, int nt, int &r0, int &r1) {
    const long long rows = nt - 2;
    r0 = 1 + (int)(b * rows / nb);
    r1 = 1 + (int)((b + 1) * rows / nb);
}

struct Ring {  // the sums of the rings that a block owns: [0] row 1, [1] row nt - 2
    Fix128 part[2][kMaxWarps];
    FixSum fix[2][kMaxWarps];
    unsigned wide[2][kMaxWarps];
    float2 mean[2];
};

// The warp's exact sum of a ring row (nv of the lane's cells are its own).
template <bool X2>
__device__ __forceinline__ void ring_sum(const Row4 &h, const Row4 &l, int nv, Ring &s, int side) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float vh[4] = {h.a.x, h.b.x, h.a.y, h.b.y}, vl[4] = {l.a.x, l.b.x, l.a.y, l.b.y};
    const bool wide = !__all_sync(kFull, fix128_takes<X2>(vh, vl, nv));
    if (!wide) {
        const Fix128 a = fix128_sum<X2>(vh, vl, nv);
        if (lane == 0) s.part[side][warp] = a;
    } else {
        FixSum f = fix_zero();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            fix_add_float(f, k < nv ? vh[k] : 0.f);
            if (X2) fix_add_float(f, k < nv ? vl[k] : 0.f);
        }
        fix_warp(f);
        if (lane == 0) s.fix[side][warp] = f;
    }
    if (lane == 0) s.wide[side][warp] = wide ? 1u : 0u;
}

// The ring's mean from the warps' sums, by one warp.
template <bool X2>
__device__ __forceinline__ void ring_mean(Ring &s, int side, int W, double np, double inv_np) {
    const int lane = threadIdx.x & 31;
    const bool wide = __any_sync(kFull, lane < W && s.wide[side][lane] != 0u);
    double sum;
    if (!wide) {
        Fix128 a{0u, 0u, 0u, 0u};
        if (lane < W) a = s.part[side][lane];
        sum = fix128_to_double(fix128_warp(a));
    } else {
        FixSum f = fix_zero();
        if (lane < W) f = s.wide[side][lane] ? s.fix[side][lane] : fix_widen(s.part[side][lane]);
        fix_warp(f);
        sum = fix_to_double(f);
    }
    if (lane == 0) s.mean[side] = fix_mean<X2>(sum, np, inv_np);
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

// Which of the lane's cells (first column col) lie inside a front (drainage.rs:425-460): four bits for
// each of the rows [r0, r1), at most kFrontRows of them. It does not depend on the field, so it is
// formed while the neighbours' rows are on their way.
constexpr int kFrontRows = 8;
__device__ __forceinline__ unsigned front_cells(const TfeStep &t, int r0, int r1, int col, int np) {
    unsigned in = 0u;
    for (int f = 0; f < t.nf; ++f) {
        const int4 fr = t.fr[f];
        const int first = max(fr.x, r0) - r0, rows = min(fr.y + 1, r1) - r0 - first;
        if (rows <= 0) continue;
        int d = col - fr.z;
        if (d < 0) d += np;
        unsigned cells = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int e = d + k;
            cells |= (e >= np ? e - np : e) < fr.w ? 1u << k : 0u;
        }
        in |= cells * ((0x11111111u >> (4 * (kFrontRows - rows))) << (4 * first));
    }
    return in;
}

// Thins the cells marked in the low four bits.
template <bool X2>
__device__ __forceinline__ void apply_fronts(const TfeStep &t, unsigned in, Row4 &h, Row4 &l) {
    const float2 fh = f2(t.factor), fl = f2(t.factor_lo);
    auto thin = [&](float2 &h, float2 &l, bool x, bool y) {
        const float2 p = mul2(h, fh);
        if (X2) {
            const float2 q = fma2(h, fl, fma2(l, fh, fma2(h, fh, neg2(p))));
            const float2 s = add2(p, q);
            const float2 e = sub2(q, sub2(s, p));
            l = make_float2(x ? e.x : l.x, y ? e.y : l.y);
            h = make_float2(x ? s.x : h.x, y ? s.y : h.y);
        } else {
            h = make_float2(x ? p.x : h.x, y ? p.y : h.y);
        }
    };
    thin(h.a, l.a, in & 1u, in & 4u);
    thin(h.b, l.b, in & 2u, in & 8u);
}

// Dynamic shared memory of a block of W warps and at most rb rows.
struct Layout {
    size_t edges, coefs, bytes;  // offsets behind the state: [rb + 1][2 fields][threads] Row4
    __host__ __device__ Layout(int W, int rb) {
        edges = sizeof(Row4) * 2 * (rb + 1) * (size_t)(32 * W);
        coefs = edges + sizeof(float4) * 2 * (size_t)rb * W;
        bytes = coefs + sizeof(float4) * 2 * (size_t)rb;
    }
};

// RAG: rows of a number of cells that is no multiple of four.
template <int SEM, bool X2, bool MAR, bool RAG>
__global__ void __launch_bounds__(kMaxWarps * 32, 1) resident_kernel(const StepArgs a, const ResidentArgs ra) {
    constexpr bool CPU = SEM == SBS_CPU_SEMANTICS;
    constexpr bool TWO = !CPU || X2;  // a second field: the surfactant, or the low words
    extern __shared__ float4 s_dyn[];
    __shared__ alignas(16) TfeStep s_tfe[2];
    __shared__ Ring s_ring;
    __shared__ double s_red[kMaxWarps];
    __shared__ int s_last;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int np = a.np, nt = a.nt, nb = gridDim.x, b = blockIdx.x;
    const int col = warp * 128 + lane * 4;
    const int nv = min(max(np - col, 0), 4);                           // the lane's cells in the row
    const bool last = lane == min(32, (np - warp * 128 + 3) / 4) - 1;  // holds the warp's rightmost cell
    const int wl = warp == 0 ? W - 1 : warp - 1, wr = warp + 1 == W ? 0 : warp + 1;
    int r0, r1;
    block_rows(b, nb, nt, r0, r1);
    const int rb = r1 - r0;
    const bool top = b == 0, bottom = b == nb - 1;

    const Layout lay(W, a.rb);
    Row4 *state = reinterpret_cast<Row4 *>(s_dyn) + threadIdx.x;
    float4 *s_co = reinterpret_cast<float4 *>(reinterpret_cast<char *>(s_dyn) + lay.coefs);
    // the warps' edge cells, [parity][row][warp] float4: leftmost cell of both fields, then rightmost
    float2 *s_edge = reinterpret_cast<float2 *>(reinterpret_cast<char *>(s_dyn) + lay.edges);
    const int edges = 2 * W;  // float2 per row
    // this lane's cells of row r (r = rb: the neighbour's row below), field f
    auto cell = [&](int r, int f) -> Row4 & { return state[(2 * r + f) * (int)blockDim.x]; };

    const float *sin = CPU ? a.lin : a.cin;
    float *sout = CPU ? a.lout : a.cout;
    // cells past the row's end take the values of the columns they wrap to: they are computed along
    // with the others and never looked at
    auto load = [&](const float *f, int r) {
        const float *p = f + (size_t)r * a.pitch;
        if (nv == 4) return row_of(__ldg(reinterpret_cast<const float4 *>(p + col)));
        return row_of(make_float4(__ldg(p + col % np), __ldg(p + (col + 1) % np), __ldg(p + (col + 2) % np),
                                  __ldg(p + (col + 3) % np)));
    };
    auto store = [&](float *f, int r, const Row4 &x) {
        if (nv > 0) *reinterpret_cast<float4 *>(f + (size_t)r * a.pitch + col) = row_to4(x);  // rows are padded
    };

    Row4 uh = load(a.hin, r0 - 1), us = row_splat(0.f), dh = load(a.hin, r1), ds = us;
    if (TWO) {
        us = load(sin, r0 - 1);
        ds = load(sin, r1);
    }
    for (int r = 0; r < rb; ++r) {
        cell(r, 0) = load(a.hin, r0 + r);
        if (TWO) cell(r, 1) = load(sin, r0 + r);
    }
    for (int r = threadIdx.x; r < rb; r += blockDim.x) {
        const float4 q = __ldg(a.rows + r0 + r);
        s_co[2 * r] = CPU ? q : make_float4(q.x, q.x, q.y, q.y);
        s_co[2 * r + 1] = make_float4(q.z, q.z, q.w, q.w);
    }
    auto load_tfe = [&](int step) {  // a step ahead
        if (CPU && a.tfe != nullptr && step < ra.steps && threadIdx.x < sizeof(TfeStep) / 16)
            cp_async16(reinterpret_cast<float4 *>(&s_tfe[step & 1]) + threadIdx.x,
                       reinterpret_cast<const float *>(a.tfe + step) + 4 * threadIdx.x);
        if (CPU) cp_async_commit();
    };
    auto put_edges = [&](float2 *row, const Row4 &x, const Row4 &y) {
        if (lane == 0) row[2 * warp] = make_float2(x.a.x, y.a.x);
        if (last) {
            if (!RAG || nv == 4)
                row[2 * warp + 1] = make_float2(x.b.y, y.b.y);
            else
                row[2 * warp + 1] = nv == 3   ? make_float2(x.a.y, y.a.y)
                                    : nv == 2 ? make_float2(x.b.x, y.b.x)
                                              : make_float2(x.a.x, y.a.x);
        }
    };
    load_tfe(0);
    for (int r = 0; r < rb; ++r) put_edges(s_edge + r * edges, cell(r, 0), TWO ? cell(r, 1) : row_splat(0.f));
    if (CPU) cp_async_wait<0>();
    __syncthreads();

    // this lane's words of the row that block `of` publishes upwards (dir 0) or downwards (1) after a
    // step of parity `par`; a block of one row publishes it once
    auto slot = [&](int par, int of, int dir, int f) {
        return ra.halo + ((((size_t)par * nb + of) * 2 + dir) * 2 + f) * (size_t)(W * 128) + col;
    };
    int up_dir = 0;
    if (!top) {
        int q0, q1;
        block_rows(b - 1, nb, nt, q0, q1);
        up_dir = q1 - q0 > 1 ? 1 : 0;
    }
    bool dead = false;  // a wait ran out: no further ones
    auto take = [&](const unsigned long long *p, unsigned tag, Row4 &x) {
        const bool u = ld_pair(p, tag, x.a.x, x.b.x);
        return ld_pair(p + 2, tag, x.a.y, x.b.y) && u;
    };

    double vacc = 0.0;
    const WgslK k{a.b, a.DR2, a.DsR2, a.Gt, a.M, a.dt, a.crit};
    for (int step = 0; step < ra.steps; ++step) {
        const int par = step & 1;
        const float2 *edge_in = s_edge + par * a.rb * edges;
        float2 *edge_out = s_edge + (par ^ 1) * a.rb * edges;
        const unsigned thinned = CPU && a.tfe != nullptr ? front_cells(s_tfe[par], r0, r1, col, np) : 0u;
        if (step > 0) {
            // the neighbours' rows after `step` steps (the poles come below)
            const unsigned tag = ra.tag0 + (unsigned)step + ra.stall;
            const long long t0 = clock64();
            for (unsigned tries = 1; !dead; ++tries) {
                bool ok = true;
                if (!top) {
                    ok = take(slot(par, b - 1, up_dir, 0), tag, uh);
                    if (TWO) ok = take(slot(par, b - 1, up_dir, 1), tag, us) && ok;
                }
                if (!bottom) {
                    ok = take(slot(par, b + 1, 0, 0), tag, dh) && ok;
                    if (TWO) ok = take(slot(par, b + 1, 0, 1), tag, ds) && ok;
                }
                if (__all_sync(kFull, ok)) break;
                const bool late =
                    clock64() - t0 > a.wait_cycles || (tries % 64 == 0 && *(volatile unsigned *)a.ring_status != 0u);
                if (__any_sync(kFull, late)) {
                    dead = true;
                    if (lane == 0) {
                        atomicOr(a.ring_status, 1u);
                        *(volatile unsigned *)a.status_host = 1u;
                    }
                }
            }
            if (CPU && top) {
                uh = row_splat(s_ring.mean[0].x);
                us = row_splat(s_ring.mean[0].y);
            }
            if (CPU && bottom) {
                dh = row_splat(s_ring.mean[1].x);
                ds = row_splat(s_ring.mean[1].y);
            }
        }
        if (!CPU) {  // the pole rows are frozen
            if (top && step > 0) {
                uh = load(a.hin, 0);
                us = load(sin, 0);
            }
            if (bottom && step > 0) {
                dh = load(a.hin, nt - 1);
                ds = load(sin, nt - 1);
            }
            // the field one pass behind the newest, over the input (which everybody has read by now:
            // the neighbours have published a step)
            if (step + 1 == ra.steps && step > 0)
                for (int r = 0; r < rb; ++r) {
                    store(ra.hprev, r0 + r, cell(r, 0));
                    store(ra.cprev, r0 + r, cell(r, 1));
                }
        }
        cell(rb, 0) = dh;
        if (TWO) cell(rb, 1) = ds;
        load_tfe(step + 1);
        const unsigned tag = ra.tag0 + (unsigned)step + 1u;
        const bool more = step + 1 < ra.steps;
        auto publish = [&](int dir, const Row4 &x, const Row4 &y) {
            unsigned long long *p = slot(par ^ 1, b, dir, 0);
            st_pair(p, tag, x.a.x, x.b.x);
            st_pair(p + 2, tag, x.a.y, x.b.y);
            if (TWO) {
                p = slot(par ^ 1, b, dir, 1);
                st_pair(p, tag, y.a.x, y.b.x);
                st_pair(p + 2, tag, y.a.y, y.b.y);
            }
        };
        // row r from the old rows above (u), at (c) and below it; the row below, loaded here, is the next
        // row's c. Three calls rotate the three windows' names, so no row is moved.
        auto advance = [&](int r, const Row4 &hu, const Row4 &su, Row4 &hc, Row4 &sc, Row4 &hn, Row4 &sn) {
            hn = cell(r + 1, 0);
            if (TWO) sn = cell(r + 1, 1);
            float hl = __shfl_up_sync(kFull, hc.b.y, 1), hr = __shfl_down_sync(kFull, hc.a.x, 1), sl = 0.f, sr = 0.f;
            if (TWO) {
                sl = __shfl_up_sync(kFull, sc.b.y, 1);
                sr = __shfl_down_sync(kFull, sc.a.x, 1);
            }
            if (lane == 0) {
                const float2 e = edge_in[r * edges + 2 * wl + 1];
                hl = e.x;
                sl = e.y;
            }
            if (last) {
                const float2 e = edge_in[r * edges + 2 * wr];
                if (!RAG || nv == 4) {
                    hr = e.x;
                    sr = e.y;
                } else {  // the seam is inside the lane's window: its next cell is column 0
                    (nv == 3 ? hc.b.y : nv == 2 ? hc.a.y : hc.b.x) = e.x;
                    (nv == 3 ? sc.b.y : nv == 2 ? sc.a.y : sc.b.x) = e.y;
                }
            }
            const int i = r0 + r;
            Row4 oh, os = row_splat(0.f);
            if (CPU) {
                cpu_row<X2>(hc, hu, hn, hl, hr, sc, su, sn, sl, sr, s_co[2 * r], a.b, a.DR2, a.dt, a.crit, oh, os);
                // the pole's mean is of the stencil's values, before the fronts
                if (i == 1) ring_sum<X2>(oh, os, nv, s_ring, 0);
                if (i == nt - 2) ring_sum<X2>(oh, os, nv, s_ring, 1);
                const unsigned in = thinned >> (4 * (r & (kFrontRows - 1))) & 0xfu;
                if (in) apply_fronts<X2>(s_tfe[par], in, oh, os);
            } else {
                wgsl_row<MAR>(hc, hu, hn, hl, hr, sc, su, sn, sl, sr, s_co[2 * r], s_co[2 * r + 1], k, oh,
                              os);
            }
            if (more && ((r == 0 && !(top && rb > 1)) || (r == rb - 1 && !bottom))) publish(r == 0 ? 0 : 1, oh, os);
            cell(r, 0) = oh;
            if (TWO) cell(r, 1) = os;
            put_edges(edge_out + r * edges, oh, os);
        };
        Row4 hc = cell(0, 0), sc = TWO ? cell(0, 1) : row_splat(0.f), hn, sn = row_splat(0.f);
#pragma unroll 1
        for (int r = 0; r < rb; r += 3) {
            advance(r, uh, us, hc, sc, hn, sn);
            if (r + 1 < rb) advance(r + 1, hc, sc, hn, sn, uh, us);
            if (r + 2 < rb) advance(r + 2, hn, sn, uh, us, hc, sc);
        }
        if (CPU) cp_async_wait<0>();
        __syncthreads();
        if (CPU && (top || bottom)) {
            if (top && warp == 0) ring_mean<X2>(s_ring, 0, W, (double)np, a.inv_np);
            if (bottom && warp == W - 1) ring_mean<X2>(s_ring, 1, W, (double)np, a.inv_np);
            __syncthreads();
        }
    }

    auto finish = [&](int i, const Row4 &x, const Row4 &y) {
        store(a.hout, i, x);
        if (TWO) store(sout, i, y);
        if (a.vol_w != nullptr) {
            const double wi = __ldg(a.vol_w + i);
            auto sum = [&](const Row4 &v) {
                double t = nv > 0 ? (double)v.a.x : 0.0;
                if (nv > 1) t += (double)v.b.x;
                if (nv > 2) t += (double)v.a.y;
                if (nv > 3) t += (double)v.b.y;
                return t * wi;
            };
            vacc += sum(x);
            if (CPU && X2) vacc += sum(y);
        }
    };
    for (int r = 0; r < rb; ++r) finish(r0 + r, cell(r, 0), TWO ? cell(r, 1) : row_splat(0.f));
    if (CPU && top) finish(0, row_splat(s_ring.mean[0].x), row_splat(s_ring.mean[0].y));
    if (CPU && bottom) finish(nt - 1, row_splat(s_ring.mean[1].x), row_splat(s_ring.mean[1].y));

    if (a.vol_w != nullptr) {
        const double v = block_sum(vacc, s_red);
        if (threadIdx.x == 0) {
            a.vol_partials[b] = v;
            __threadfence();
            s_last = atomicAdd(a.vol_counter, 1u) == (unsigned)nb - 1u;
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            double tot = 0.0;
            for (int i = threadIdx.x; i < nb; i += blockDim.x) tot += __ldcg(a.vol_partials + i);
            if (!CPU)  // the frozen pole rows of the input
                for (int j = threadIdx.x; j < np; j += blockDim.x) {
                    tot += (double)__ldg(a.hin + j) * __ldg(a.vol_w);
                    tot += (double)__ldg(a.hin + (size_t)(nt - 1) * a.pitch + j) * __ldg(a.vol_w + nt - 1);
                }
            tot = block_sum(tot, s_red);
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

template <bool RAG>
const void *pick(int sem, bool x2, bool mar) {
    if (sem == SBS_CPU_SEMANTICS)
        return x2 ? (const void *)resident_kernel<SBS_CPU_SEMANTICS, true, false, RAG>
                  : (const void *)resident_kernel<SBS_CPU_SEMANTICS, false, false, RAG>;
    return mar ? (const void *)resident_kernel<SBS_WGSL_SEMANTICS, false, true, RAG>
               : (const void *)resident_kernel<SBS_WGSL_SEMANTICS, false, false, RAG>;
}

const void *resident_fn(int sem, bool x2, bool mar, bool rag) {
    return rag ? pick<true>(sem, x2, mar) : pick<false>(sem, x2, mar);
}

}  // namespace

// As few rows a block as make all blocks resident at once. nby = 0: rows of more than 2048 columns,
// or more rows than the chip holds, or, in CPU semantics, more than kCpuRows a block: from there on
// issue decides, and the blocked step spends fewer instructions a row (640 x 1280, five rows: 4.3 us
// here, 4.7 blocked; 768 x 1536, six: 5.1 and 4.6). Which WGSL runs of a grid that fits are left to the
// other kernels all the same, resident_from() in drainage.cu says. Both Marangoni forms of the kernel have
// to fit, as the choice is made per run.
constexpr int kCpuRows = 5;
static_assert(kCpuRows <= kFrontRows, "the fronts' cells of a block's rows are one word");
StepGeom resident_geometry(int nt, int np, int semantics, int x2) {
    StepGeom g{};
    const int W = (np + 127) / 128;
    if (W > kMaxWarps || nt < 3 || np < 3) return g;
    int dev = 0, sms = 148, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return g;
    const int forms = semantics == SBS_WGSL_SEMANTICS ? 2 : 1;
    for (int mar = 0; mar < forms; ++mar)
        if (cudaFuncSetAttribute(resident_fn(semantics, x2 != 0, mar != 0, np % 4 != 0),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess) {
            cudaGetLastError();
            return g;
        }
    const int most = semantics == SBS_CPU_SEMANTICS ? kCpuRows : 1 << 20;
    for (int rb = 1; rb <= most && Layout(W, rb).bytes <= kMaxSmem; ++rb) {
        int fit = 0;
        for (int mar = 0; mar < forms; ++mar) {
            int n = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                    &n, resident_fn(semantics, x2 != 0, mar != 0, np % 4 != 0), 32 * W, Layout(W, rb).bytes) !=
                cudaSuccess) {
                cudaGetLastError();
                return g;
            }
            fit = mar == 0 || n < fit ? n : fit;
        }
        const int blocks = (nt - 2 + rb - 1) / rb;
        if (blocks > fit * sms) continue;
        g.wx = W;
        g.nbx = 1;
        g.nby = blocks;
        g.rb = rb;
        g.cap = fit * sms;
        return g;
    }
    return g;
}

size_t resident_halo_bytes(const StepGeom &g) {
    return sizeof(unsigned long long) * 2 * g.nby * 2 * 2 * (size_t)(g.wx * 128);
}

cudaError_t launch_resident(int semantics, int x2, const StepArgs &a, const ResidentArgs &ra, const StepGeom &g,
                            cudaStream_t s) {
    if (g.nby < 1) return cudaErrorInvalidValue;
    void *args[] = {(void *)&a, (void *)&ra};
    return cudaLaunchCooperativeKernel(resident_fn(semantics, x2 != 0, a.marangoni != 0, a.np % 4 != 0), dim3(g.nby),
                                       dim3(32 * g.wx), args, Layout(g.wx, a.rb).bytes, s);
}

}  // namespace sbs
