// One time step of the cartesian 3D GPU-program scheme in one launch:
// injection, update, free surface, one-way boundary (onewayBC_3D), sponge of
// both levels, and the receiver gather of the level the step reads.
//
// 16 bytes a cell have to move (two levels and the velocity read, one level
// written); what bounds the kernel is instruction issue (about 150 a cell at
// 0.65 of the issue slots).  At 210 x 210 x 193 cells the update with its
// coordinates in indexed arrays took 94 us and two boundary passes over every
// cell 44 and 45 us more; this kernel takes 48 us and the step, with injection
// and gather, 196 us before and 48 now.
//  * The new level goes to a third buffer, so any cell of the old ones may be read.
//  * A boundary cell's value needs the new level, before the boundary, at one
//    inward neighbour: um[n] + (um[c] - new[n]) b.  Its thread computes new[n]
//    from the old levels in place of new[c], which nobody needs: the same work
//    at a shifted cell, no second pass.
//  * Injection on read and the traces of the previous step as in k_stepA2d.cu.
#include <cuda_runtime.h>

#include <type_traits>

#include "awe_internal.h"
#include "fp_exact.cuh"

namespace awe {

namespace {

// Sponge factor of a line (z, x) on a plane y, spongeKernel_3D: the first low
// face of (x, y, z), else the first high face.  On planes off the axis-3 bands
// it is the line's own; on them it is the plane's unless a face that comes
// first holds the line, so a plane costs one selection.
template <bool EXACT>
struct Line3 {
    using F = typename std::conditional<EXACT, double, float>::type;
    F f;
    bool low, high;  // the line's factor also holds on planes of the low / high axis-3 band
    __device__ __forceinline__ Line3(int z, int x, const Grid &g, int nb, const StepAParams &p) {
        const int lx = max(nb - x, 0), lz = max(nb - z, 0), hx = max(x - (g.n2 - nb), 0), hz = max(z - (g.n1 - nb), 0);
        f = tab(lx ? lx : lz ? lz : hx ? hx : hz, p);
        low = lx > 0;
        high = lx > 0 || lz > 0 || hx > 0;
    }
    // entry 0 is 1
    __device__ static __forceinline__ F tab(int i, const StepAParams &p) {
        if constexpr (EXACT) return __ldg(p.dtab + i);
        else return __ldg(p.ftab + i);
    }
    // (FP64 is slow on this GPU: the product only where it changes the value, a
    // factor being 1 exactly when its high word is 1's)
    __device__ static __forceinline__ float times(float v, F w) {
        if constexpr (EXACT) return __double2hiint(w) >= 0x3ff00000 ? v : (float)((double)v * w);
        else return __fmul_rn(v, w);
    }
};

// corner e's injection of step `it` added to v (k_injectA's operations)
template <bool EXACT>
__device__ __forceinline__ float inj3(float v, int e, int it, const StepA3Fused &f) {
    float a = __ldg(f.wav + (long long)it * f.ncs + (f.ncs == 1 ? 0 : f.inj_src[e] >> 3)), w = f.inj_w[e];
    if (f.scaled) {
        a = __fmul_rn(a, w);
        w = __ldg(f.scale + f.inj_src[e]);
    }
    return EXACT ? __fadd_rn(v, __fmul_rn(a, w)) : fmaf(a, w, v);
}

constexpr int TZ = 32, TX = 8, UY = 2;  // threads along axes 1 and 2, planes in flight

// the new level before the boundary at a cell (v its velocity, q the previous
// level, sponged; in: it has a stencil).  AWE_EXACT: the reference's
// operations, each rounded; AWE_FAST: products fused into the sums that take them
template <bool EXACT>
__device__ __forceinline__ float update3(bool in, float u, float q, float v, float zm, float zp, float xm, float xp,
                                         float ym, float yp, const StepAParams &p) {
    const float u2 = __fadd_rn(u, u), vv = __fmul_rn(v, v);
    const float dx = __fadd_rn(__fsub_rn(xp, u2), xm), dy = __fadd_rn(__fsub_rn(yp, u2), ym);
    const float dz = __fadd_rn(__fsub_rn(zp, u2), zm);
    float lap = 0.f, o;
    if constexpr (EXACT) {
        if (in) lap = __fadd_rn(__fadd_rn(__fdiv_rn(dx, p.dd2), __fdiv_rn(dy, p.dd3)), __fdiv_rn(dz, p.dd1));
        o = __fadd_rn(__fmul_rn(p.dt2, __fmul_rn(vv, lap)), u2);
    } else {
        if (in) lap = fmaf(dz, p.rd[0], fmaf(dx, p.rd[1], __fmul_rn(dy, p.rd[2])));
        o = fmaf(p.dt2, __fmul_rn(vv, lap), u2);
    }
    return __fsub_rn(o, q);
}

// um[n] + (um[c] - new[n]) b
template <bool EXACT>
__device__ __forceinline__ float oneway3(float un, float uc, float on, float b) {
    const float d = __fsub_rn(uc, on);
    return EXACT ? __fadd_rn(un, __fmul_rn(d, b)) : fmaf(d, b, un);
}

// A block owns 32 x 8 lines and some planes of them: the five planes of an
// axis-3 face, or up to L planes between the faces.  Over those planes a
// thread's shift (to the inward neighbour along the last axis, z, x, y, whose
// face is within 5 cells) is the same, so boundary and interior cells run one
// loop: two planes at a time, their loads all issued before the first is used.
// One cell per thread spent most of its instructions on the set-up of a line
// (157 us at 210 x 210 x 193 cells); 16 planes share it.
template <bool EXACT>
__global__ void __launch_bounds__(TZ *TX, 4) k_stepA3(const float *__restrict__ cur, const float *__restrict__ prv,
                                                      float *__restrict__ nxt, const float *__restrict__ vel,
                                                      const StepAParams p, const StepA3Fused f, int L, int segs) {
    const Grid g = p.g;
    const long long s2 = g.n1, s3 = (long long)g.n1 * g.n2;
    const int seg = blockIdx.z;
    if (seg >= segs) {  // receiver gather of cur, extract_3D's order
        const int r = (((seg - segs) * (int)gridDim.y + (int)blockIdx.y) * (int)gridDim.x + (int)blockIdx.x) *
                          (TZ * TX) + (int)(threadIdx.y * TZ + threadIdx.x);
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;");
        if (r >= f.nr) return;
        const GeoPoint pt = f.rec[r];
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float v = cur[pt.base + ((c & 1) ? 1 : 0) + ((c & 2) ? s2 : 0) + ((c & 4) ? s3 : 0)];
            acc = (c == 0) ? __fmul_rn(v, pt.w[c])
                           : EXACT ? __fadd_rn(acc, __fmul_rn(v, pt.w[c])) : fmaf(v, pt.w[c], acc);
        }
        f.rec_row[r] = acc;
        return;
    }
    const int b1 = blockIdx.x * TZ, b2 = blockIdx.y * TX;
    const int z = b1 + threadIdx.x, x = b2 + threadIdx.y;
    int y0 = 5 + (seg - 2) * L, y1 = min(y0 + L, g.n3 - 5), sh = 0, tz = z, tx = x;
    const float *btab = nullptr;  // this thread's one-way coefficients (null: not a boundary cell)
    int bst = 0;
    if (seg < 2) {  // axis-3 faces
        y0 = seg == 0 ? 0 : g.n3 - 5;
        y1 = y0 + 5;
        sh = seg == 0 ? 1 : -1;
        btab = (seg == 0 ? p.tb[4] : p.tb[5]) + (long long)z * g.n2 + x;
    } else if (x <= 4 || x >= g.n2 - 5) {
        tx += x >= g.n2 - 5 ? -1 : 1;
        btab = (x >= g.n2 - 5 ? p.tb[1] : p.tb[2]) + z;  // high: the z-high table, as the reference
        bst = g.n1;
    } else if (z <= 4 || z >= g.n1 - 5) {
        tz += z >= g.n1 - 5 ? -1 : 1;
        btab = (z >= g.n1 - 5 ? p.tb[1] : p.tb[0]) + x;
        bst = g.n2;
    }
    // source corners this thread reads: at its update's line or one next to it,
    // or at its own cell's line; worked out before the wait, only in blocks that
    // hold such lines, and looked at again only on the planes [ylo, yhi] they
    // touch (testing them on every plane made the blocks around one source the
    // last of the launch)
    unsigned long long mine = 0;
    int ylo = g.n3, yhi = -1;
    for (int e = 0; e < f.inj_n; e++) {
        const int c1 = f.inj_i1[e], c2 = f.inj_i2[e], c3 = f.inj_i3[e];
        if (c1 < b1 - 2 || c1 > b1 + TZ + 1 || c2 < b2 - 2 || c2 > b2 + TX + 1 || c3 < y0 - 2 || c3 > y1 + 1) continue;
        if (abs(c1 - tz) + abs(c2 - tx) <= 1 || (c1 == z && c2 == x)) {
            mine |= 1ull << e;
            ylo = min(ylo, c3 - 2);
            yhi = max(yhi, c3 + 2);
        }
    }
    const bool in = tz >= 4 && tz < g.n1 - 4 && tx >= 4 && tx < g.n2 - 4;
    const bool zero = tz < p.nb;  // freeSurf_3D, before the boundary
    const bool ok = z < g.n1 && x < g.n2, edge = __any_sync(0xffffffffu, ok && btab);
    if (!ok) tz = tx = 0;
    const Line3<EXACT> lc(ok ? z : 0, ok ? x : 0, g, p.nb, p), lt(tz, tx, g, p.nb, p);
    const long long t = (y0 + sh) * s3 + tx * s2 + tz;
    const float *pc = cur + t, *pq = prv + t, *pv = vel + t;
    const float *po = cur + y0 * s3 + x * s2 + z;  // the own cell (read by boundary lines only)
    float *pn = nxt + y0 * s3 + x * s2 + z;
    if (btab) btab += (long long)y0 * bst;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    if (!ok) return;
    // every address below lies inside the level: boundary lines are shifted
    // inward, and an axis-3 face's updates are on planes 1 .. n3 - 2
    float um = pc[-s3], uc = pc[0];
    int y = y0;
    auto planes = [&](auto count) {
        constexpr int N = decltype(count)::value;
        float u[N + 2], q[N], v[N], zm[N], zp[N], xm[N], xp[N], own[N], b[N];
        u[0] = um;
        u[1] = uc;
#pragma unroll
        for (int k = 0; k < N; k++) {
            u[k + 2] = pc[s3];
            zm[k] = pc[-1], zp[k] = pc[1];
            xm[k] = pc[-s2], xp[k] = pc[s2];
            q[k] = *pq;
            v[k] = __ldg(pv);
            own[k] = b[k] = 0.f;
            if (edge) {
                if (btab) {
                    own[k] = *po;
                    b[k] = __ldg(btab);
                    btab += bst;
                }
                po += s3;
            }
            pc += s3, pq += s3, pv += s3;
        }
        um = u[N];
        uc = u[N + 1];
        for (unsigned long long m = y <= yhi && y + N > ylo ? mine : 0; m; m &= m - 1) {  // (source, corner) order
            const int e = __ffsll((long long)m) - 1;
            const int dz = f.inj_i1[e] - tz, dx = f.inj_i2[e] - tx, yy = f.inj_i3[e] - y;
#pragma unroll
            for (int k = 0; k < N + 2; k++)
                if (dz == 0 && dx == 0 && yy == k - 1 + sh) u[k] = inj3<EXACT>(u[k], e, f.it, f);
#pragma unroll
            for (int k = 0; k < N; k++) {
                if (f.inj_i1[e] == z && f.inj_i2[e] == x && yy == k) own[k] = inj3<EXACT>(own[k], e, f.it, f);
                if (yy != k + sh) continue;
                if (dz == 0 && dx == 0 && f.it > 0) q[k] = inj3<EXACT>(q[k], e, f.it - 1, f);
                if (dz == 1 && dx == 0) zp[k] = inj3<EXACT>(zp[k], e, f.it, f);
                if (dz == -1 && dx == 0) zm[k] = inj3<EXACT>(zm[k], e, f.it, f);
                if (dz == 0 && dx == 1) xp[k] = inj3<EXACT>(xp[k], e, f.it, f);
                if (dz == 0 && dx == -1) xm[k] = inj3<EXACT>(xm[k], e, f.it, f);
            }
        }
#pragma unroll
        for (int k = 0; k < N; k++) {
            // the two lines' factors on this plane (the same plane but for an axis-3 face)
            typename Line3<EXACT>::F wt = lt.f, wc = lc.f;
            const int ty = y + k + sh;
            if (ty < p.nb) wt = lt.low ? lt.f : Line3<EXACT>::tab(p.nb - ty, p);
            else if (ty > g.n3 - p.nb) wt = lt.high ? lt.f : Line3<EXACT>::tab(ty - (g.n3 - p.nb), p);
            if (y + k < p.nb) wc = lc.low ? lc.f : Line3<EXACT>::tab(p.nb - (y + k), p);
            else if (y + k > g.n3 - p.nb) wc = lc.high ? lc.f : Line3<EXACT>::tab(y + k - (g.n3 - p.nb), p);
            const float qd = Line3<EXACT>::times(q[k], wt);
            const bool stencil = in && (sh == 0 || (ty >= 4 && ty < g.n3 - 4));
            float o = update3<EXACT>(stencil, u[k + 1], qd, v[k], zm[k], zp[k], xm[k], xp[k], u[k], u[k + 2], p);
            if (zero) o = 0.f;
            if (edge && btab) o = oneway3<EXACT>(u[k + 1], own[k], o, b[k]);
            *pn = Line3<EXACT>::times(o, wc);
            pn += s3;
        }
        y += N;
    };
    while (y + UY <= y1) planes(std::integral_constant<int, UY>());
    while (y < y1) planes(std::integral_constant<int, 1>());
}

}  // namespace

void launch_stepA3(bool exact, const float *cur, const float *prv, float *nxt, const float *vel, const StepAParams &p,
                   const StepA3Fused &f, cudaStream_t s) {
    dim3 grid((p.g.n1 + TZ - 1) / TZ, (p.g.n2 + TX - 1) / TX, 1);
    // Planes per block: a block's set-up costs about as much as 10 planes of
    // one line, and 16 blocks per SM keep the last wave short.  56 x 56 x 60
    // cells: 5.4 us a step with one plane, 13.7 with 16; 100^3: 12.4 with two,
    // 16.6 with 16; 290^3: 228 with two, 132 with 16.
    int L = 16;
    while (L > 1 && (long long)grid.x * grid.y * (2 + (p.g.n3 - 10 + L - 1) / L) < 16LL * p.sms) L /= 2;
    const int segs = 2 + (p.g.n3 - 10 + L - 1) / L;
    grid.z = (unsigned)segs;
    const unsigned per = grid.x * grid.y * TZ * TX;
    if (f.nr > 0) grid.z += ((unsigned)f.nr + per - 1) / per;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(TZ, TX);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (exact) cudaLaunchKernelEx(&cfg, k_stepA3<true>, cur, prv, nxt, vel, p, f, L, segs);
    else cudaLaunchKernelEx(&cfg, k_stepA3<false>, cur, prv, nxt, vel, p, f, L, segs);
}

}  // namespace awe
