// Per-cell update of the drainage step, shared by every step kernel so that all of them round
// identically (and the oracle's kernel-order mode can repeat them).
//
// The update runs on pairs of neighbouring cells with Blackwell's packed FP32 instructions
// (__fadd2_rn / __fmul2_rn / __ffma2_rn: two IEEE round-to-nearest f32 operations per
// instruction). Each half rounds exactly like the scalar operation, and a - b is written as
// a + (-b) (negation is exact), so results are bit-identical to the scalar formula while the
// floating-point instruction count halves.
#pragma once

#include <cuda_runtime.h>

namespace sbs {

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// GPUDrainageSimulator semantics (drainage.wgsl:104-201) for two cells of h and surfactant Gamma.
//   co = per-row (A, E, F, G); neighbours theta-1 (tm), theta+1 (tp), phi-1 (pm), phi+1 (pp).
//   lt = (tp-h)+(tm-h), d1 = tp-tm, lp = (pp-h)+(pm-h), L = F*lp + E*d1 + b*lt
//   h' = max(h + dt*(D/R^2*L + A*h^3 [+ M*|grad Gamma|*h^2]), 0)
//   Gamma' = clamp(Gamma + dt*(Ds/R^2*L_Gamma [+ 0.001*L*Gamma]), 0, 1)
// Branch-free: the update is always evaluated and cells below the critical thickness keep their
// values by selection (drainage.wgsl:108-112), which gives the same bits as skipping them.
template <bool MAR>
__device__ __forceinline__ void wgsl_cell2(float2 h, float2 tm, float2 tp, float2 pm, float2 pp, float2 cv, float2 ctm,
                                           float2 ctp, float2 cpm, float2 cpp, const float4 &co, float b, float DR2,
                                           float DsR2, float Gt, float M, float dt, float crit, float2 &vh,
                                           float2 &vc) {
    const float2 lt = add2(sub2(tp, h), sub2(tm, h));
    const float2 d1 = sub2(tp, tm);
    const float2 lp = add2(sub2(pp, h), sub2(pm, h));
    const float2 L = fma2(f2(co.z), lp, fma2(f2(co.y), d1, mul2(f2(b), lt)));
    const float2 h3 = mul2(mul2(h, h), h);
    float2 inc = fma2(f2(DR2), L, mul2(f2(co.x), h3));
    if (MAR) {
        const float2 gt = mul2(f2(Gt), sub2(ctp, ctm));
        const float2 gp = mul2(f2(co.w), sub2(cpp, cpm));
        const float2 sq = fma2(gt, gt, mul2(gp, gp));
        const float2 mag = make_float2(sqrtf(sq.x), sqrtf(sq.y));
        inc = add2(inc, mul2(mul2(f2(M), mag), mul2(h, h)));
    }
    const float2 lc = add2(sub2(ctp, cv), sub2(ctm, cv));
    const float2 d1c = sub2(ctp, ctm);
    const float2 lpc = add2(sub2(cpp, cv), sub2(cpm, cv));
    const float2 Lc = fma2(f2(co.z), lpc, fma2(f2(co.y), d1c, mul2(f2(b), lc)));
    float2 dc = mul2(f2(DsR2), Lc);
    if (MAR) dc = fma2(mul2(f2(0.001f), L), cv, dc);
    const float2 y = fma2(f2(dt), dc, cv);
    const float2 x = fma2(f2(dt), inc, h);
    float y0 = y.x > 0.f ? y.x : 0.f, y1 = y.y > 0.f ? y.y : 0.f;
    y0 = y0 < 1.f ? y0 : 1.f;
    y1 = y1 < 1.f ? y1 : 1.f;
    const float x0 = x.x > 0.f ? x.x : 0.f, x1 = x.y > 0.f ? x.y : 0.f;
    vh.x = h.x < crit ? h.x : x0;
    vh.y = h.y < crit ? h.y : x1;
    vc.x = h.x < crit ? cv.x : y0;
    vc.y = h.y < crit ? cv.y : y1;
}

// The same update for the four cells of a float4 (two pairs).
template <bool MAR>
__device__ __forceinline__ void wgsl_cell4(const float4 &h, const float4 &tm, const float4 &tp, const float4 &pm,
                                           const float4 &pp, const float4 &cv, const float4 &ctm, const float4 &ctp,
                                           const float4 &cpm, const float4 &cpp, const float4 &co, float b, float DR2,
                                           float DsR2, float Gt, float M, float dt, float crit, float4 &vh,
                                           float4 &vc) {
    float2 a, c, e, g;
    wgsl_cell2<MAR>(make_float2(h.x, h.y), make_float2(tm.x, tm.y), make_float2(tp.x, tp.y), make_float2(pm.x, pm.y),
                    make_float2(pp.x, pp.y), make_float2(cv.x, cv.y), make_float2(ctm.x, ctm.y),
                    make_float2(ctp.x, ctp.y), make_float2(cpm.x, cpm.y), make_float2(cpp.x, cpp.y), co, b, DR2, DsR2,
                    Gt, M, dt, crit, a, c);
    wgsl_cell2<MAR>(make_float2(h.z, h.w), make_float2(tm.z, tm.w), make_float2(tp.z, tp.w), make_float2(pm.z, pm.w),
                    make_float2(pp.z, pp.w), make_float2(cv.z, cv.w), make_float2(ctm.z, ctm.w),
                    make_float2(ctp.z, ctp.w), make_float2(cpm.z, cpm.w), make_float2(cpp.z, cpp.w), co, b, DR2, DsR2,
                    Gt, M, dt, crit, e, g);
    vh = make_float4(a.x, a.y, e.x, e.y);
    vc = make_float4(c.x, c.y, g.x, g.y);
}

}  // namespace sbs

namespace sbs {

// DrainageSimulator semantics (drainage.rs:326-379) for two cells, plain f32 (X2 = false) or
// compensated hi + lo words (X2 = true: differences include the lo words and h + dt*inc is an
// error-free TwoSum). Cells below the critical thickness keep their words (drainage.rs:331).
template <bool X2>
__device__ __forceinline__ void cpu_cell2(float2 h, float2 tm, float2 tp, float2 pm, float2 pp, float2 l, float2 tml,
                                          float2 tpl, float2 pml, float2 ppl, const float4 &co, float b, float DR2,
                                          float dt, float crit, float2 &vh, float2 &vl) {
    float2 lt = add2(sub2(tp, h), sub2(tm, h));
    float2 d1 = sub2(tp, tm);
    float2 lp = add2(sub2(pp, h), sub2(pm, h));
    if (X2) {
        lt = add2(lt, add2(sub2(tpl, l), sub2(tml, l)));
        d1 = add2(d1, sub2(tpl, tml));
        lp = add2(lp, add2(sub2(ppl, l), sub2(pml, l)));
    }
    const float2 L = fma2(f2(co.z), lp, fma2(f2(co.y), d1, mul2(f2(b), lt)));
    const float2 h3 = mul2(mul2(h, h), h);
    const float2 inc = fma2(f2(DR2), L, mul2(f2(co.x), h3));
    if (X2) {
        const float2 t = fma2(f2(dt), inc, l);
        const float2 s = add2(h, t);
        const float2 bb = sub2(s, h);
        const float2 e = add2(sub2(h, sub2(s, bb)), sub2(t, bb));
        vh.x = h.x < crit ? h.x : (s.x < 0.f ? 0.f : s.x);
        vh.y = h.y < crit ? h.y : (s.y < 0.f ? 0.f : s.y);
        vl.x = h.x < crit ? l.x : (s.x < 0.f ? 0.f : e.x);
        vl.y = h.y < crit ? l.y : (s.y < 0.f ? 0.f : e.y);
    } else {
        const float2 x = fma2(f2(dt), inc, h);
        vh.x = h.x < crit ? h.x : (x.x > 0.f ? x.x : 0.f);
        vh.y = h.y < crit ? h.y : (x.y > 0.f ? x.y : 0.f);
        vl = make_float2(0.f, 0.f);
    }
}

template <bool X2>
__device__ __forceinline__ void cpu_cell4(const float4 &h, const float4 &tm, const float4 &tp, const float4 &pm,
                                          const float4 &pp, const float4 &l, const float4 &tml, const float4 &tpl,
                                          const float4 &pml, const float4 &ppl, const float4 &co, float b, float DR2,
                                          float dt, float crit, float4 &vh, float4 &vl) {
    float2 a, c, e, g;
    cpu_cell2<X2>(make_float2(h.x, h.y), make_float2(tm.x, tm.y), make_float2(tp.x, tp.y), make_float2(pm.x, pm.y),
                  make_float2(pp.x, pp.y), make_float2(l.x, l.y), make_float2(tml.x, tml.y), make_float2(tpl.x, tpl.y),
                  make_float2(pml.x, pml.y), make_float2(ppl.x, ppl.y), co, b, DR2, dt, crit, a, c);
    cpu_cell2<X2>(make_float2(h.z, h.w), make_float2(tm.z, tm.w), make_float2(tp.z, tp.w), make_float2(pm.z, pm.w),
                  make_float2(pp.z, pp.w), make_float2(l.z, l.w), make_float2(tml.z, tml.w), make_float2(tpl.z, tpl.w),
                  make_float2(pml.z, pml.w), make_float2(ppl.z, ppl.w), co, b, DR2, dt, crit, e, g);
    vh = make_float4(a.x, a.y, e.x, e.y);
    vl = make_float4(c.x, c.y, g.x, g.y);
}


// ---------------------------------------------------------------------------
// The same two updates for the blocked and the resident pipelines, on a row of four cells held as the
// pairs of columns (0, 2) and (1, 3). With that split one pair's phi neighbour is the other pair as it
// stands, and only the neighbours beyond the four cells are put together from a shuffle; adjacent
// columns (0, 1), (2, 3) need every shifted pair assembled from moves. The kernels are bound by
// instruction issue, so the rest is spelled to cost few instructions too: the phi difference of
// columns (0, 1) and (2, 3) is formed once and used with both signs (a - b = -(b - a) exactly), the
// clamps are FMNMX and the FMA's own saturation, and cells below the critical thickness are looked
// for with one three-input minimum and a warp vote: the per-cell selects run only in warps that
// hold such a cell. Results are those of wgsl_cell2 / cpu_cell2 bit for bit (a zero may differ in
// its sign, which no later operation or comparison sees).
//
// Packed or scalar: a packed instruction takes both FP32 pipes for a cycle, as two scalar ones do,
// and saves an issue slot, but its operands must be register pairs and cannot be negated in place.
// At 2048 x 4096, us per step: the compensated update (K = 3) 16.8 packed, 15.5 with scalar
// subtractions, 14.9 all scalar; the WGSL update (K = 4) 12.4 packed with negated operands, 12.0
// with a - b as fma(b, -1, a) and scalar phi differences, 13.3 all scalar.
struct alignas(16) Row4 {
    float2 a, b;  // columns (0, 2) and (1, 3)
};
__device__ __forceinline__ Row4 row_of(const float4 &v) { return Row4{make_float2(v.x, v.z), make_float2(v.y, v.w)}; }
__device__ __forceinline__ float4 row_to4(const Row4 &r) { return make_float4(r.a.x, r.b.x, r.a.y, r.b.y); }
__device__ __forceinline__ Row4 row_splat(float v) { return Row4{f2(v), f2(v)}; }
__device__ __forceinline__ float row_min(const Row4 &r) { return fminf(fminf(fminf(r.a.x, r.a.y), r.b.x), r.b.y); }
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
    float d;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// a - b as one packed operation, and the scalar forms.
__device__ __forceinline__ float2 psub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }
__device__ __forceinline__ float2 sadd2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 ssub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 smul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 sfma2(float2 a, float2 b, float2 c) {
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
}

// Second difference in phi, (pp - x) + (pm - x); xl, xr = columns -1 and 4.
__device__ __forceinline__ void row_phi2(const Row4 &x, float xl, float xr, float2 &la, float2 &lb) {
    const float2 d = ssub2(x.b, x.a);
    la = make_float2(d.x + (xl - x.a.x), d.y + (x.b.x - x.a.y));
    lb = make_float2((x.a.y - x.b.x) - d.x, (xr - x.b.y) - d.y);
}

// Correctly rounded square roots of a pair, as sqrtf gives them: from r = rsqrt(x) (the hardware's
// approximation), g = x r is improved by its exact residual, g + (x - g g) r / 2 (Markstein, IA-64
// and Elementary Functions, 2000, ch. 9). For one step from this approximation that is the rounded
// root of every x in [1, 4), which a test goes through (the exponent only scales it), as long as
// nothing underflows or overflows on the way: x = 0 or in [2^-96, 2^126); `odd` is set for others.
// sqrtf itself is ~10 instructions with a branch of its own per cell, which kept the Marangoni step
// at twice the time of the plain one.
__device__ __forceinline__ float2 sqrt2(float2 x, bool &odd) {
    const unsigned lo = 0x0f800000u, hi = 0x7e800000u;  // 2^-96, 2^126
    const unsigned u = __float_as_uint(x.x), v = __float_as_uint(x.y);
    odd = odd || min(u - 1u, v - 1u) < lo - 1u || max(u, v) >= hi;  // negative and NaN are the largest
    float2 r;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r.x) : "f"(fmaxf(x.x, __uint_as_float(lo))));
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(r.y) : "f"(fmaxf(x.y, __uint_as_float(lo))));
    const float2 g = mul2(x, r);
    return fma2(fma2(neg2(g), g, x), mul2(f2(0.5f), r), g);
}

struct WgslK {
    float b, DR2, DsR2, Gt, M, dt, crit;
};

// Row coefficients (A, E, F, G) of the theta row, each doubled: c0 = (A, A, E, E), c1 = (F, F, G, G).
template <bool MAR>
__device__ __forceinline__ void wgsl_row(const Row4 &h, const Row4 &hu, const Row4 &hd, float hl, float hr,
                                         const Row4 &c, const Row4 &cu, const Row4 &cd, float cl, float cr,
                                         const float4 &c0, const float4 &c1, const WgslK &k, Row4 &oh, Row4 &oc) {
    const float2 A = make_float2(c0.x, c0.y), E = make_float2(c0.z, c0.w), F = make_float2(c1.x, c1.y);
    float2 lpa, lpb, lpca, lpcb;
    row_phi2(h, hl, hr, lpa, lpb);
    row_phi2(c, cl, cr, lpca, lpcb);
    float2 maga = f2(0.f), magb = maga;
    if (MAR) {
        const float2 G = make_float2(c1.z, c1.w);
        auto square = [&](float2 ctm, float2 ctp, float2 cpm, float2 cpp) {
            const float2 gt = mul2(f2(k.Gt), psub2(ctp, ctm)), gp = mul2(G, psub2(cpp, cpm));
            return fma2(gt, gt, mul2(gp, gp));
        };
        const float2 sa = square(cu.a, cd.a, make_float2(cl, c.b.x), c.b);
        const float2 sb = square(cu.b, cd.b, c.a, make_float2(c.a.y, cr));
        bool odd = false;
        maga = sqrt2(sa, odd);
        magb = sqrt2(sb, odd);
        if (__any_sync(0xffffffffu, odd)) {
            maga = make_float2(sqrtf(sa.x), sqrtf(sa.y));
            magb = make_float2(sqrtf(sb.x), sqrtf(sb.y));
        }
    }
    auto pair = [&](float2 h, float2 tm, float2 tp, float2 lp, float2 cv, float2 ctm, float2 ctp, float2 lpc,
                    float2 mag, float2 &vh, float2 &vc) {
        const float2 lt = add2(psub2(tp, h), psub2(tm, h));
        const float2 L = fma2(F, lp, fma2(E, psub2(tp, tm), mul2(f2(k.b), lt)));
        float2 inc = fma2(f2(k.DR2), L, mul2(A, mul2(mul2(h, h), h)));
        if (MAR) inc = add2(inc, mul2(mul2(f2(k.M), mag), mul2(h, h)));
        const float2 lc = add2(psub2(ctp, cv), psub2(ctm, cv));
        float2 dc = mul2(f2(k.DsR2), fma2(F, lpc, fma2(E, psub2(ctp, ctm), mul2(f2(k.b), lc))));
        if (MAR) dc = fma2(mul2(f2(0.001f), L), cv, dc);
        const float2 x = fma2(f2(k.dt), inc, h);
        vh = make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
        vc = make_float2(fma_sat(k.dt, dc.x, cv.x), fma_sat(k.dt, dc.y, cv.y));
    };
    pair(h.a, hu.a, hd.a, lpa, c.a, cu.a, cd.a, lpca, maga, oh.a, oc.a);
    pair(h.b, hu.b, hd.b, lpb, c.b, cu.b, cd.b, lpcb, magb, oh.b, oc.b);
    if (__any_sync(0xffffffffu, row_min(h) < k.crit)) {  // cells below the critical thickness keep their values
        auto keep = [&](float h, float cv, float &vh, float &vc) {
            vh = h < k.crit ? h : vh;
            vc = h < k.crit ? cv : vc;
        };
        keep(h.a.x, c.a.x, oh.a.x, oc.a.x);
        keep(h.a.y, c.a.y, oh.a.y, oc.a.y);
        keep(h.b.x, c.b.x, oh.b.x, oc.b.x);
        keep(h.b.y, c.b.y, oh.b.y, oc.b.y);
    }
}

// c = the row's A, E, F.
template <bool X2>
__device__ __forceinline__ void cpu_row(const Row4 &h, const Row4 &hu, const Row4 &hd, float hl, float hr,
                                        const Row4 &l, const Row4 &lu, const Row4 &ld, float ll, float lr,
                                        const float4 &c, float b, float DR2, float dt, float crit,
                                        Row4 &oh, Row4 &ol) {
    const float2 A = f2(c.x), E = f2(c.y), F = f2(c.z), b2 = f2(b), D2 = f2(DR2), dt2 = f2(dt);
    float2 lpa, lpb, lpla = f2(0.f), lplb = f2(0.f);
    row_phi2(h, hl, hr, lpa, lpb);
    if (X2) row_phi2(l, ll, lr, lpla, lplb);
    auto pair = [&](float2 h, float2 tm, float2 tp, float2 lp, float2 l, float2 tml, float2 tpl, float2 lpl, float2 &vh,
                    float2 &vl) {
        float2 lt = sadd2(ssub2(tp, h), ssub2(tm, h));
        float2 d1 = ssub2(tp, tm);
        if (X2) {
            lt = sadd2(lt, sadd2(ssub2(tpl, l), ssub2(tml, l)));
            d1 = sadd2(d1, ssub2(tpl, tml));
            lp = sadd2(lp, lpl);
        }
        const float2 L = sfma2(F, lp, sfma2(E, d1, smul2(b2, lt)));
        const float2 inc = sfma2(D2, L, smul2(A, smul2(smul2(h, h), h)));
        if (X2) {
            const float2 t = sfma2(dt2, inc, l);
            const float2 s = sadd2(h, t);
            const float2 bb = ssub2(s, h);
            vl = sadd2(ssub2(h, ssub2(s, bb)), ssub2(t, bb));
            vh = s;
        } else {
            const float2 x = sfma2(dt2, inc, h);
            vh = make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
            vl = f2(0.f);
        }
    };
    pair(h.a, hu.a, hd.a, lpa, l.a, lu.a, ld.a, lpla, oh.a, ol.a);
    pair(h.b, hu.b, hd.b, lpb, l.b, lu.b, ld.b, lplb, oh.b, ol.b);
    const bool thin = row_min(h) < crit || (X2 && row_min(oh) < 0.f);
    if (__any_sync(0xffffffffu, thin)) {
        auto keep = [&](float h, float l, float &vh, float &vl) {
            if (X2) {
                vl = h < crit ? l : (vh < 0.f ? 0.f : vl);
                vh = h < crit ? h : (vh < 0.f ? 0.f : vh);
            } else {
                vh = h < crit ? h : vh;
            }
        };
        keep(h.a.x, l.a.x, oh.a.x, ol.a.x);
        keep(h.a.y, l.a.y, oh.a.y, ol.a.y);
        keep(h.b.x, l.b.x, oh.b.x, ol.b.x);
        keep(h.b.y, l.b.y, oh.b.y, ol.b.y);
    }
}

// Per-thread copies into shared memory: each lane waits for its own, so the warps need no handshake.
__device__ __forceinline__ void cp_async16(float4 *smem, const float *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(float *smem, const float *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The columns a lane's four-cell window reads and writes: cells cu .. cu + 3 of a row of np cells,
// wrapped at the row end. With rows of a multiple of four cells (RAG false) the window is always four
// aligned cells. Else the window that holds the seam is put together cell by cell: lanes whose cells
// all lie in the row (or in the aligned copy of it that starts at column 0) still move 16 bytes.
template <bool RAG>
struct Cols;
template <>
struct Cols<false> {
    int col;
    __device__ __forceinline__ Cols(int cu, int np) : col(((cu % np) + np) % np) {}
    __device__ __forceinline__ int valid() const { return 4; }
    // The offset of cell k of the window.
    __device__ __forceinline__ int at(int k) const { return col + k; }
    __device__ __forceinline__ float4 load(const float *row) const {
        return __ldg(reinterpret_cast<const float4 *>(row + col));
    }
    // Requests the window into shared memory (cp.async; the caller closes the group).
    template <bool CG>
    __device__ __forceinline__ void request(float4 *slot, const float *row) const {
        cp_async16(slot, row + col);
    }
    __device__ __forceinline__ void store(float *row, const float4 &v) const {
        *reinterpret_cast<float4 *>(row + col) = v;
    }
};
template <>
struct Cols<true> {
    int c[4];
    int nv;  // cells cu + k < np (of a kept lane: the ones it writes)
    __device__ __forceinline__ Cols(int cu, int np) {
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = (((cu + k) % np) + np) % np;
        nv = min(max(np - cu, 0), 4);
    }
    __device__ __forceinline__ int valid() const { return nv; }
    __device__ __forceinline__ int at(int k) const { return c[k]; }
    __device__ __forceinline__ bool vec() const { return c[3] == c[0] + 3 && (c[0] & 3) == 0; }
    __device__ __forceinline__ float4 load(const float *row) const {
        if (vec()) return __ldg(reinterpret_cast<const float4 *>(row + c[0]));
        return make_float4(__ldg(row + c[0]), __ldg(row + c[1]), __ldg(row + c[2]), __ldg(row + c[3]));
    }
    template <bool CG>
    __device__ __forceinline__ void request(float4 *slot, const float *row) const {
        if (vec()) {
            cp_async16(slot, row + c[0]);
        } else if (CG) {  // 4-byte copies go through L1, which may hold what another block has since written
            *slot = make_float4(__ldcg(row + c[0]), __ldcg(row + c[1]), __ldcg(row + c[2]), __ldcg(row + c[3]));
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) cp_async4(reinterpret_cast<float *>(slot) + k, row + c[k]);
        }
    }
    __device__ __forceinline__ void store(float *row, const float4 &v) const {
        if (nv == 4) {
            *reinterpret_cast<float4 *>(row + c[0]) = v;
        } else {
            row[c[0]] = v.x;
            if (nv > 1) row[c[1]] = v.y;
            if (nv > 2) row[c[2]] = v.z;
        }
    }
};

}  // namespace sbs
