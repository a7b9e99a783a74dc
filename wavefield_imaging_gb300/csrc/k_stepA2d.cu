// One time step of the 2D GPU-program scheme (cartesian and polar) in one
// launch: injection, update, one-way boundary, free-surface mask, sponge of
// both levels, and the receiver gather of the level the step reads.
//
// The level is small (317 k cells: 1.3 MB, resident in L2), so a step is bound
// by launches and their latency.  Five launches a step (one-thread injection,
// update, two boundary passes over every cell, gather) took 24 us at 483 x
// 657 cells; one launch takes 3.6 us (300 steps, replayed graph).  What makes one launch possible:
//  * the new level goes to a third buffer, so every thread may read any cell
//    of the current and previous levels;
//  * a boundary row's value needs the new level only at one cell of the last
//    line (row +- 1 there), which has no stencil: each thread of the eight rows
//    forms it again from the two old levels;
//  * levels are stored without their injection and the few source cells add
//    it when read (as the current level for step it, as the previous one for
//    step it - 1): the same float additions, in the same order;
//  * the traces of step it - 1 are gathered from the level step it reads.
#include <cuda_runtime.h>

#include "awe_internal.h"
#include "fp_exact.cuh"

namespace awe {

namespace {

// sponge factor by index and its product with a value (the reference's FP64
// factor in AWE_EXACT)
template <bool EXACT>
struct Damp2 {
    double f64;
    float f32;
    __device__ __forceinline__ Damp2() {}
    __device__ __forceinline__ Damp2(int i, const StepAParams &p) {
        if constexpr (EXACT) f64 = i ? __ldg(p.dtab + i) : 1.0;
        else f32 = i ? __ldg(p.ftab + i) : 1.f;
    }
    __device__ __forceinline__ float operator()(float v) const {
        if constexpr (EXACT) return (float)((double)v * f64);
        else return __fmul_rn(v, f32);
    }
};

// sponge index of spongeKernel_2D: the priority axis first (cartesian: axis 2,
// polar: axis 1), low faces before high ones
template <int GEOM>
__device__ __forceinline__ int sponge2(int i1, int i2, const Grid &g, int nb) {
    const int a = GEOM == 0 ? i2 : i1, na = GEOM == 0 ? g.n2 : g.n1;
    const int b = GEOM == 0 ? i1 : i2, nbx = GEOM == 0 ? g.n1 : g.n2;
    if (a < nb) return nb - a;
    if (b < nb) return nb - b;
    if (a > na - nb) return a - (na - nb);
    if (b > nbx - nb) return b - (nbx - nb);
    return 0;
}

// corner e's injection of step `it` added to v (k_injectA's operations)
template <bool EXACT>
__device__ __forceinline__ float inj2(float v, int e, int it, const StepA2Fused &f) {
    float a = __ldg(f.wav + (long long)it * f.ncs + (f.ncs == 1 ? 0 : f.inj_src[e] >> 3)), w = f.inj_w[e];
    if (f.scaled) {
        a = __fmul_rn(a, w);
        w = __ldg(f.scale + f.inj_src[e]);
    }
    return EXACT ? __fadd_rn(v, __fmul_rn(a, w)) : fmaf(a, w, v);
}

// 64 x 8 cells per block, two per thread (rows 4 apart): 483 x 657 cells are
// one wave of blocks.  What no earlier launch writes (velocity, tables) is
// loaded before the wait for the previous step, the levels after it, all of
// them unconditionally (clamped), so their latencies overlap.
// Idx: int up to 2^31 - 1 cells (64-bit indices cost 6 % of a step)
template <int GEOM, bool EXACT, typename Idx>
__global__ void __launch_bounds__(256) k_stepA2(const float *__restrict__ cur, const float *__restrict__ prv,
                                                float *__restrict__ nxt, const float *__restrict__ vel,
                                                const StepAParams p, const StepA2Fused f) {
    const Grid g = p.g;
    const Idx s2 = g.n1, last = s2 * g.n2 - 1;
    const int rows = (g.n2 + 7) / 8;  // blocks of cells
    if ((int)blockIdx.y >= rows) {    // receiver gather of cur, extract_2D's order
        const int r = (((int)blockIdx.y - rows) * (int)gridDim.x + (int)blockIdx.x) * 256 +
                      (int)(threadIdx.y * 64 + threadIdx.x);
        GeoPoint pt{};
        if (r < f.nr) pt = f.rec[r];
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;");
        if (r >= f.nr) return;
        const long long sz = GEOM == 0 ? 1 : s2, sx = GEOM == 0 ? s2 : 1;
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const float v = cur[pt.base + ((c & 1) ? sz : 0) + ((c & 2) ? sx : 0)];
            acc = (c == 0) ? __fmul_rn(v, pt.w[c]) : EXACT ? __fadd_rn(acc, __fmul_rn(v, pt.w[c])) : fmaf(v, pt.w[c], acc);
        }
        f.rec_row[r] = acc;
        return;
    }
    const int b1 = blockIdx.x * 64, b2 = blockIdx.y * 8;
    const int i1 = b1 + threadIdx.x, j1 = min(i1, g.n1 - 1);
    // source corners on this block's cells or their neighbours
    unsigned near = 0;
    for (int e = 0; e < f.inj_n; e++)
        if (f.inj_i1[e] >= b1 - 1 && f.inj_i1[e] <= b1 + 64 && f.inj_i2[e] >= b2 - 1 && f.inj_i2[e] <= b2 + 8)
            near |= 1u << e;
    float am = 0.f, ap = 0.f, b = 0.f, b0 = 0.f;
    if constexpr (GEOM == 2) {
        am = __ldg(p.tr0 + j1), ap = __ldg(p.tr1 + j1), b = __ldg(p.tr2 + j1), b0 = __ldg(p.tr3 + j1);
    }
    Idx i[2];
    Damp2<EXACT> damp[2];
    float v[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int j2 = min(b2 + (int)threadIdx.y + 4 * r, g.n2 - 1);
        i[r] = j2 * s2 + j1;
        v[r] = __ldg(vel + i[r]);
        damp[r] = Damp2<EXACT>(sponge2<GEOM>(j1, j2, g, p.nb), p);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    float q[2], u[2], zm[2], zp[2], xm[2], xp[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        u[r] = cur[i[r]];
        q[r] = prv[i[r]];
        zm[r] = cur[max(i[r] - 1, (Idx)0)];
        zp[r] = cur[min(i[r] + 1, last)];
        xm[r] = cur[max(i[r] - s2, (Idx)0)];
        xp[r] = cur[min(i[r] + s2, last)];
    }
    for (; near; near &= near - 1) {  // in (source, corner) order
        const int e = __ffs(near) - 1;
        const Idx c = f.inj_i2[e] * s2 + f.inj_i1[e];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const Idx d = c - i[r];
            if (d == 0) {
                u[r] = inj2<EXACT>(u[r], e, f.it, f);
                if (f.it > 0) q[r] = inj2<EXACT>(q[r], e, f.it - 1, f);
            } else if (d == 1) {
                zp[r] = inj2<EXACT>(zp[r], e, f.it, f);
            } else if (d == -1) {
                zm[r] = inj2<EXACT>(zm[r], e, f.it, f);
            } else if (d == s2) {
                xp[r] = inj2<EXACT>(xp[r], e, f.it, f);
            } else if (d == -s2) {
                xm[r] = inj2<EXACT>(xm[r], e, f.it, f);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int i2 = b2 + threadIdx.y + 4 * r;
        if (i1 >= g.n1 || i2 >= g.n2) continue;
        const float qd = damp[r](q[r]);
        const float u2 = __fadd_rn(u[r], u[r]);
        const bool in = i1 >= 4 && i1 < g.n1 - 4 && i2 >= 4 && i2 < g.n2 - 4;
        const float vv = __fmul_rn(v[r], v[r]);
        // AWE_EXACT: the reference's operations, each rounded; AWE_FAST: products
        // fused into the sums that take them
        float lap = 0.f, o;
        if constexpr (GEOM == 0) {
            const float dx = __fadd_rn(__fsub_rn(xp[r], u2), xm[r]), dz = __fadd_rn(__fsub_rn(zp[r], u2), zm[r]);
            if constexpr (EXACT) {
                if (in) lap = __fadd_rn(__fdiv_rn(dx, p.dd2), __fdiv_rn(dz, p.dd1));
                o = __fadd_rn(__fmul_rn(p.dt2, __fmul_rn(vv, lap)), u2);
            } else {
                if (in) lap = fmaf(dx, p.rd[1], __fmul_rn(dz, p.rd[0]));
                o = fmaf(p.dt2, __fmul_rn(vv, lap), u2);
            }
        } else if constexpr (EXACT) {
            if (in)
                lap = __fadd_rn(
                    __fadd_rn(__fadd_rn(__fmul_rn(am, zm[r]), __fmul_rn(p.a0, u[r])), __fmul_rn(ap, zp[r])),
                    __fadd_rn(__fadd_rn(__fmul_rn(b, xm[r]), __fmul_rn(b0, u[r])), __fmul_rn(b, xp[r])));
            o = __fadd_rn(__fmul_rn(__fmul_rn(p.dt2, vv), lap), u2);
        } else {
            if (in)
                lap = __fadd_rn(fmaf(ap, zp[r], fmaf(am, zm[r], __fmul_rn(p.a0, u[r]))),
                                fmaf(b, xp[r], fmaf(b0, u[r], __fmul_rn(b, xm[r]))));
            o = fmaf(__fmul_rn(p.dt2, vv), lap, u2);
        }
        o = __fsub_rn(o, qd);
        // one-way boundary: rows 1..4 and n-5..n-2 of the swept axis
        const int row = GEOM == 0 ? i1 : i2, nsw = GEOM == 0 ? g.n1 : g.n2;
        const bool lo = row >= 1 && row <= 4, hi = row >= nsw - 5 && row <= nsw - 2;
        if ((lo || hi) && (GEOM != 0 || row < g.n2)) {
            const int nbr = lo ? row + 1 : row - 1;
            const int l1 = GEOM == 0 ? nbr : g.n1 - 1, l2 = GEOM == 0 ? g.n2 - 1 : nbr;
            const Idx l = l2 * s2 + l1;
            const float um = cur[l];
            const float ql = Damp2<EXACT>(sponge2<GEOM>(l1, l2, g, p.nb), p)(prv[l]);
            const float d = __fsub_rn(u[r], __fsub_rn(__fadd_rn(um, um), ql)), c = lo ? p.b2lo : p.b2hi;
            o = EXACT ? __fadd_rn(um, __fmul_rn(d, c)) : fmaf(d, c, um);
        }
        o = damp[r](o);
        if (p.mask == 1 && (i2 > g.n2 - p.nb || (i2 < p.spill && i1 >= 1))) o = 0.f;
        if (p.mask == 3 && (i1 > g.n1 - p.nb || (i1 < p.spill && i2 >= 1))) o = 0.f;
        nxt[i[r]] = o;
    }
}

}  // namespace

template <typename Idx>
static void launch_a2(int geom, bool exact, const float *cur, const float *prv, float *nxt, const float *vel,
                      const StepAParams &p, const StepA2Fused &f, cudaStream_t s) {
    dim3 grid((p.g.n1 + 63) / 64, (p.g.n2 + 7) / 8);
    if (f.nr > 0) grid.y += (unsigned)((f.nr + grid.x * 256 - 1) / (grid.x * 256));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(64, 4);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (geom == 0) {
        if (exact) cudaLaunchKernelEx(&cfg, k_stepA2<0, true, Idx>, cur, prv, nxt, vel, p, f);
        else cudaLaunchKernelEx(&cfg, k_stepA2<0, false, Idx>, cur, prv, nxt, vel, p, f);
    } else {
        if (exact) cudaLaunchKernelEx(&cfg, k_stepA2<2, true, Idx>, cur, prv, nxt, vel, p, f);
        else cudaLaunchKernelEx(&cfg, k_stepA2<2, false, Idx>, cur, prv, nxt, vel, p, f);
    }
}

void launch_stepA2(int geom, bool exact, const float *cur, const float *prv, float *nxt, const float *vel,
                   const StepAParams &p, const StepA2Fused &f, cudaStream_t s) {
    if (p.g.cells() + p.g.n1 < (1ll << 31)) launch_a2<int>(geom, exact, cur, prv, nxt, vel, p, f, s);
    else launch_a2<long long>(geom, exact, cur, prv, nxt, vel, p, f, s);
}

}  // namespace awe
