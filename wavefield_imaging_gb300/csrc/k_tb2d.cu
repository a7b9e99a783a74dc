// Several 2D time steps of the CPU-program scheme in one launch (temporal
// blocking over overlapping tiles).
//
// A single shot's levels (592 x 592 cells: 1.4 MB each) live in L2, and a step
// of its own is launch and latency: 4.35 us for 0.5 us of work.  Here a block
// loads its tile of both levels and of v^2 dt^2 with a halo of k * nop cells
// once, steps k times in shared memory, and stores the tile of the last two
// levels; halo cells are computed by every tile that needs them.  A thread owns
// 4 (axis 1) x 1, 2 or 4 (axis 2) cells: their two levels and v^2 dt^2 stay in
// registers, the current level also in one of two shared-memory buffers that
// the neighbours read.  Sources, the receivers of every step's level and the
// sponge are inside.  The operations of a cell are k_stepB's in the same order
// (with the products that its compiled form fuses), so the result is the same
// bits.  Measured, us a step, one-step kernel and this one (replayed graphs):
// 592 x 592 8th order 4.35, 1.91; 141 x 183 4th order 2.45, 0.79; 1480 x 1480
// 8th order 16.4, 8.6.  What bounds it now is the latency of a step in one
// block per SM (0.4 of the issue slots), then shared-memory reads.
//
// A batch of shots takes its windows' tiles in one launch, two smaller blocks
// per SM: 12 windows of 592 x 580 at 8th order 17.8 us a step with the one-step
// kernels, 14.3 so; their gradient (recompute and adjoint sweep of a segment,
// then its imaging condition at once) 102 us a step, 68 so.  48 such windows
// stream from HBM, where the column march (52 us) is ahead of this (60).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "awe_internal.h"
#include "fp_exact.cuh"
#include "gsum.cuh"

namespace awe {

namespace {

// MODE 0: AWE_FAST, 1: AWE_EXACT, 3: AWE_FAST storing slots (the gradient's recompute),
// 2 (ADJ): the adjoint step (k_adjB): cur = nu_k, prv = nu_{k+1}, shared memory holds
// I vel2 nu; step j is time step it - j; the cells' entries are receiver residuals
// BATCH: tiles of many shots' windows (p.tiles), with the operations of k_batch2d and
// k_batch2d_adj, whose Laplacian is one chain of fused multiply-adds
template <int NOP, int MODE, int CX, bool BATCH>
__global__ void __launch_bounds__(BATCH ? kTb2BatchThreads : kTb2Threads, BATCH ? 2 : 1) k_tb2(const Tb2Params p) {
    constexpr bool EXACT = MODE == 1, ADJ = MODE == 2, SLOTS = MODE >= 2;
    extern __shared__ float smem[];
    const int zt = p.rz / 4, rz = p.rz, tid = threadIdx.x;
    const int xg = tid / zt, zs = tid - xg * zt;
    // four columns of padding on either side: outer halo strips read past the region
    const int plane = (p.rx + 8) * rz;
    float *S0 = smem + 4 * rz, *S1 = S0 + plane;
    int tz0 = blockIdx.x * p.tz, tx0 = blockIdx.y * p.tx, tile = blockIdx.y * gridDim.x + blockIdx.x;
    int n2 = p.n2, nr = p.nr, ncs = p.ncs, ihi2 = p.ihi2;
    int rec0, nrec, cell0, ncell, ent0, nent;  // the tile's points in the lists
    long long off = 0;
    const float *w2 = p.w2, *wav = p.wav;
    float *dat = p.dat;
    if constexpr (BATCH) {
        tile = blockIdx.x;
        const Tb2Tile t = p.tiles[tile];
        tz0 = t.z0, tx0 = t.x0;
        n2 = t.n2, nr = t.nr, ihi2 = n2 - p.ilo2;
        off = t.off;
        w2 += t.wx_off, dat += t.dat_off;
        if (ADJ) ncs = nr, wav += t.dat_off;
        rec0 = t.rec0, nrec = p.rec_start ? t.nrec : 0, cell0 = t.cell0, ncell = t.ncell, ent0 = t.ent0, nent = t.nent;
    } else {
        rec0 = p.rec_start ? p.rec_start[tile] : 0, nrec = p.rec_start ? p.rec_start[tile + 1] - rec0 : 0;
        cell0 = p.inj_start ? p.inj_start[tile] : 0, ncell = p.inj_start ? p.inj_start[tile + 1] - cell0 : 0;
        ent0 = p.inj_start ? p.ent_start[tile] : 0, nent = p.inj_start ? p.ent_start[tile + 1] - ent0 : 0;
    }
    const int z0 = tz0 - p.hz + 4 * zs, x0 = tx0 - p.hx + CX * xg;  // the thread's first cell
    const int n1 = p.n1, tz1 = min(tz0 + p.tz, n1), tx1 = min(tx0 + p.tx, n2);
    const int own = CX * xg * rz + 4 * zs;
    const bool vec = BATCH || (n1 & 3) == 0;

    // cells outside the grid take the nearest one's values: nothing a step keeps depends on them
    const int zc[4] = {min(max(z0, 0), vec ? n1 - 4 : n1 - 1), min(max(z0 + 1, 0), n1 - 1), min(max(z0 + 2, 0), n1 - 1),
                       min(max(z0 + 3, 0), n1 - 1)};
    auto load = [&](const float *src, int c) {
        const float *q = src + off + (long long)min(max(x0 + c, 0), n2 - 1) * n1;
        return vec ? *reinterpret_cast<const float4 *>(q + zc[0]) : make_float4(q[zc[0]], q[zc[1]], q[zc[2]], q[zc[3]]);
    };
    float4 cur[CX], prv[CX], vel[CX];
    float wz[4], wx[CX];
    // a batch has rounds of tiles: all loads of a tile go out first
    if constexpr (BATCH) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
        for (int c = 0; c < CX; c++) {
            cur[c] = load(p.cur, c);
            prv[c] = load(p.prv, c);
        }
    }
    // what no step writes, before the wait for the previous launch
#pragma unroll
    for (int c = 0; c < CX; c++) {
        vel[c] = load(p.vel, c);
        wx[c] = w2 ? __ldg(w2 + min(max(x0 + c, 0), n2 - 1)) : 1.f;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) wz[i] = p.w1 ? __ldg(p.w1 + min(max(z0 + i, 0), n1 - 1)) : 1.f;
    // The tile's receivers and sources, with the wavelet samples of the launch's
    // steps, go to shared memory here: read from global memory in every step,
    // the chain of their loads made the tiles that hold them twice as slow.
    float4 *rec_w = reinterpret_cast<float4 *>(smem + 2 * plane), *rec_d = rec_w + p.max_rec;
    int4 *cells = reinterpret_cast<int4 *>(rec_d + p.max_rec);  // cell, first and last entry, v^2 dt^2 (ADJ: sponge)
    int2 *rec_l = reinterpret_cast<int2 *>(cells + p.max_cell);  // cell, receiver
    int *mine = reinterpret_cast<int *>(rec_l + p.max_rec);      // per thread: first cell * 65536 + cells
    float *ent_w = reinterpret_cast<float *>(mine + kTb2Threads), *ent_d = ent_w + p.max_ent;
    for (int r = tid; r < nrec; r += blockDim.x) {
        const int4 q = p.rec_pt[rec0 + r];  // z, x, receiver
        rec_l[r] = make_int2((q.y - tx0 + p.hx) * rz + q.x - tz0 + p.hz, q.z);
        rec_w[r] = *reinterpret_cast<const float4 *>(p.rec_wt + 4 * (rec0 + r));
        if (p.w1) rec_d[r] = make_float4(p.w1[q.x], p.w1[q.x + 1], w2[q.y], w2[q.y + 1]);
    }
    if (ADJ) mine[tid] = 0;
    if (ncell > 0) {
        if (ADJ) __syncthreads();
        auto owner = [&](const int4 &q) { return (q.y - tx0 + p.hx) / CX * zt + (q.x - tz0 + p.hz) / 4; };
        for (int s = tid; s < ncell; s += blockDim.x) {
            const int4 q = p.inj_cell[cell0 + s];  // z, x, first and last entry, a thread's cells one after the other
            float f = ADJ ? 1.f : p.vel[off + (long long)q.y * n1 + q.x];
            if (ADJ && p.w1) f = __fmul_rn(p.w1[q.x], w2[q.y]);
            cells[s] = make_int4((q.y - tx0 + p.hx) * rz + q.x - tz0 + p.hz, q.z - ent0, q.w - ent0, __float_as_int(f));
            const int o = owner(q);
            if (ADJ && (s == 0 || owner(p.inj_cell[cell0 + s - 1]) != o)) {
                int n = 1;
                while (s + n < ncell && owner(p.inj_cell[cell0 + s + n]) == o) n++;
                mine[o] = s * 65536 + n;
            }
        }
        for (int e = tid; e < nent; e += blockDim.x) {
            const int2 en = p.inj_ent[ent0 + e];
            ent_w[e] = __int_as_float(en.y);
            for (int j = 0; j < p.k; j++) {
                const int it = ADJ ? p.it - j : p.it + j;
                float d = 0.f;
                if (!ADJ) d = wav[(long long)it * ncs + (ncs == 1 ? 0 : en.x >> 3)];
                else if (it % p.jdata == 0) d = wav[(long long)(it / p.jdata) * ncs + (en.x >> 3)];
                ent_d[j * p.max_ent + e] = d;
            }
        }
    }
    // I vel2 nu of a strip
    auto weighted = [&](const float4 &v, int c) {
        const bool xin = x0 + c >= NOP && x0 + c < n2 - NOP;
        return make_float4(xin && z0 >= NOP && z0 < n1 - NOP ? __fmul_rn(vel[c].x, v.x) : 0.f,
                           xin && z0 + 1 >= NOP && z0 + 1 < n1 - NOP ? __fmul_rn(vel[c].y, v.y) : 0.f,
                           xin && z0 + 2 >= NOP && z0 + 2 < n1 - NOP ? __fmul_rn(vel[c].z, v.z) : 0.f,
                           xin && z0 + 3 >= NOP && z0 + 3 < n1 - NOP ? __fmul_rn(vel[c].w, v.w) : 0.f);
    };
    // a strip of the tile to global memory
    auto store = [&](float *dst, int c, const float4 &v) {
        const int x = x0 + c;
        if (z0 < tz0 || z0 >= tz1 || x < tx0 || x >= tx1) return;
        float *d = dst + off + (long long)x * n1 + z0;
        if (vec) {
            *reinterpret_cast<float4 *>(d) = v;
        } else {
            d[0] = v.x;
            if (z0 + 1 < tz1) d[1] = v.y;
            if (z0 + 2 < tz1) d[2] = v.z;
            if (z0 + 3 < tz1) d[3] = v.w;
        }
    };
    if constexpr (!BATCH) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;");
#pragma unroll
        for (int c = 0; c < CX; c++) {
            cur[c] = load(p.cur, c);
            prv[c] = load(p.prv, c);
        }
    }
#pragma unroll
    for (int c = 0; c < CX; c++) {
        *reinterpret_cast<float4 *>(S0 + own + c * rz) = ADJ ? weighted(cur[c], c) : cur[c];
    }
    __syncthreads();
    // (ADJ) the thread's cells with entries
    const int my0 = ADJ ? mine[tid] >> 16 : 0, my1 = ADJ ? my0 + (mine[tid] & 65535) : 0;

    // uniform: every cell the steps compute is interior / keeps its value under the sponge
    const int e0 = NOP * (p.k - 1);
    const bool inner = tz0 - e0 - 3 >= NOP && tz1 + e0 + 3 <= n1 - NOP && tx0 - e0 - 3 >= NOP && tx1 + e0 + 3 <= n2 - NOP;
    const bool damp = p.w1 && !(tz0 - e0 >= p.ilo1 && tz1 + e0 <= p.ihi1 && tx0 - e0 >= p.ilo2 && tx1 + e0 <= ihi2);

    // the thread's cells are within `need` of the tile: computed while the later
    // steps of the launch still need them
    int need = max(max(max(tz0 - (z0 + 3), z0 - (tz1 - 1)), max(tx0 - (x0 + CX - 1), x0 - (tx1 - 1))), 0);
    if (z0 + 3 < 0 || z0 >= n1 || x0 + CX - 1 < 0 || x0 >= n2) {
        need = 1 << 30;
        // I vel2 nu outside the grid in the second buffer too: no step stores it there, and the cells within NOP
        // of an edge, whose nu the sources' term of the gradient takes, read it
        if constexpr (ADJ) {
#pragma unroll
            for (int c = 0; c < CX; c++)
                *reinterpret_cast<float4 *>(S1 + own + c * rz) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    // v with its cell's entries of step j added, in (point, corner) order
    auto with_entries = [&](float v, const int4 &q, int j) {
        const float f = __int_as_float(q.w), *dd = ent_d + j * p.max_ent;
#pragma unroll 1
        for (int e = q.y; e < q.z; e++) {
            if constexpr (ADJ) {
                const float r = __fmul_rn(f, __fmul_rn(ent_w[e], dd[e]));
                v = BATCH ? fmaf(f, r, v) : __fadd_rn(v, __fmul_rn(f, r));
            } else {
                const float a = __fmul_rn(dd[e], ent_w[e]);
                v = EXACT ? __fadd_rn(v, __fmul_rn(a, f)) : fmaf(a, f, v);
            }
        }
        return v;
    };
    // GEN: cells that are not interior, or change under the sponge (a factor of 1 changes nothing)
    auto steps = [&](auto gen_) {
        constexpr bool GEN = decltype(gen_)::value;
        for (int j = 0; j < p.k; j++) {
            const int it = p.it + j;
            float *slot = SLOTS ? p.slots + j * p.slot_stride : nullptr;
            if (need <= NOP * (p.k - 1 - j)) {
                float4 W[CX + 2 * NOP];  // columns x0 - NOP .. x0 + CX - 1 + NOP of the strip
#pragma unroll
                for (int k = 0; k < CX + 2 * NOP; k++)
                    W[k] = !ADJ && k >= NOP && k < NOP + CX ? cur[k - NOP < CX ? k - NOP : 0]
                                                    : *reinterpret_cast<const float4 *>(S0 + own + (k - NOP) * rz);
#pragma unroll
                for (int c = 0; c < CX; c++) {
                    const float4 a = *reinterpret_cast<const float4 *>(S0 + own + c * rz - 4);
                    const float4 b = *reinterpret_cast<const float4 *>(S0 + own + c * rz + 4);
                    const float4 m = W[NOP + c];
                    const float zw[12] = {a.x, a.y, a.z, a.w, m.x, m.y, m.z, m.w, b.x, b.y, b.z, b.w};
                    float4 pr = prv[c], o;
                    if (!ADJ && GEN) {
                        pr.x = __fmul_rn(__fmul_rn(pr.x, wz[0]), wx[c]);
                        pr.y = __fmul_rn(__fmul_rn(pr.y, wz[1]), wx[c]);
                        pr.z = __fmul_rn(__fmul_rn(pr.z, wz[2]), wx[c]);
                        pr.w = __fmul_rn(__fmul_rn(pr.w, wz[3]), wx[c]);
                    }
                    float4 lp = make_float4(0.f, 0.f, 0.f, 0.f);  // L(V) of the strip
                    // ts_kernel.c:140-144: lap = u*c0 + sum_k [(z pair)*cz + (x pair)*cx]
                    if constexpr (EXACT) {
                        float *ov = &o.x;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const float u = zw[4 + i];
                            float lap = __fmul_rn(u, p.c0);
#pragma unroll
                            for (int k = 1; k <= NOP; k++) {
                                const float zp = __fadd_rn(zw[4 + i - k], zw[4 + i + k]);
                                const float xp = __fadd_rn((&W[NOP + c - k].x)[i], (&W[NOP + c + k].x)[i]);
                                lap = __fadd_rn(lap, __fadd_rn(__fmul_rn(zp, p.cz[k]), __fmul_rn(xp, p.cx[k])));
                            }
                            ov[i] = sum3_rn(__fmul_rn((&vel[c].x)[i], lap), __fadd_rn(u, u), -(&pr.x)[i]);
                        }
                    } else if constexpr (ADJ) {
                        // lambda = 2 I nu + L(I vel2 nu) + W (1 - 2 I) nu_{k+1}, mu = W lambda
                        const float2 c0 = make_float2(p.c0, p.c0);
                        float2 l0 = __fmul2_rn(c0, make_float2(m.x, m.y)), l1 = __fmul2_rn(c0, make_float2(m.z, m.w));
#pragma unroll
                        for (int k = 1; k <= NOP; k++) {
                            const float4 xm = W[NOP + c - k], xp = W[NOP + c + k];
                            const float2 cz = make_float2(p.cz[k], p.cz[k]), cx = make_float2(p.cx[k], p.cx[k]);
                            float2 z0p, z1p;
                            if (k % 2 == 0) {
                                z0p = __fadd2_rn(make_float2(zw[4 - k], zw[5 - k]), make_float2(zw[4 + k], zw[5 + k]));
                                z1p = __fadd2_rn(make_float2(zw[6 - k], zw[7 - k]), make_float2(zw[6 + k], zw[7 + k]));
                            } else {
                                z0p = make_float2(__fadd_rn(zw[4 - k], zw[4 + k]), __fadd_rn(zw[5 - k], zw[5 + k]));
                                z1p = make_float2(__fadd_rn(zw[6 - k], zw[6 + k]), __fadd_rn(zw[7 - k], zw[7 + k]));
                            }
                            l0 = __ffma2_rn(z0p, cz, l0);
                            l1 = __ffma2_rn(z1p, cz, l1);
                            l0 = __ffma2_rn(__fadd2_rn(make_float2(xm.x, xm.y), make_float2(xp.x, xp.y)), cx, l0);
                            l1 = __ffma2_rn(__fadd2_rn(make_float2(xm.z, xm.w), make_float2(xp.z, xp.w)), cx, l1);
                        }
                        const float4 u = cur[c];
                        const float lt[4] = {l0.x, l0.y, l1.x, l1.y}, uv[4] = {u.x, u.y, u.z, u.w};
                        const float yv[4] = {pr.x, pr.y, pr.z, pr.w};
                        float ov[4];
                        const bool xin = x0 + c >= NOP && x0 + c < n2 - NOP;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const bool in = !GEN || (xin && z0 + i >= NOP && z0 + i < n1 - NOP);
                            const float w = GEN ? __fmul_rn(wz[i], wx[c]) : 1.f;
                            const float t = __fadd_rn(in ? __fadd_rn(uv[i], uv[i]) : 0.f, lt[i]);
                            const float lam = fmaf(in ? -w : w, yv[i], t);
                            ov[i] = GEN ? __fmul_rn(w, lam) : lam;
                        }
                        o = make_float4(ov[0], ov[1], ov[2], ov[3]);
                    } else {
                        // two cells per instruction, with the products that k_stepB's compiled form fuses
                        const float2 u0 = make_float2(m.x, m.y), u1 = make_float2(m.z, m.w);
                        float2 l0, l1;
#pragma unroll
                        for (int k = 1; k <= NOP; k++) {
                            const float4 xm = W[NOP + c - k], xp = W[NOP + c + k];
                            const float2 cz = make_float2(p.cz[k], p.cz[k]), cx = make_float2(p.cx[k], p.cx[k]);
                            float2 z0p, z1p;
                            if (k % 2 == 0) {  // pairs aligned with the 16-byte loads
                                z0p = __fadd2_rn(make_float2(zw[4 - k], zw[5 - k]), make_float2(zw[4 + k], zw[5 + k]));
                                z1p = __fadd2_rn(make_float2(zw[6 - k], zw[7 - k]), make_float2(zw[6 + k], zw[7 + k]));
                            } else {
                                z0p = make_float2(__fadd_rn(zw[4 - k], zw[4 + k]), __fadd_rn(zw[5 - k], zw[5 + k]));
                                z1p = make_float2(__fadd_rn(zw[6 - k], zw[6 + k]), __fadd_rn(zw[7 - k], zw[7 + k]));
                            }
                            const float2 x0p = __fadd2_rn(make_float2(xm.x, xm.y), make_float2(xp.x, xp.y));
                            const float2 x1p = __fadd2_rn(make_float2(xm.z, xm.w), make_float2(xp.z, xp.w));
                            const float2 c0 = make_float2(p.c0, p.c0);
                            if constexpr (BATCH) {
                                l0 = __ffma2_rn(x0p, cx, __ffma2_rn(z0p, cz, k == 1 ? __fmul2_rn(u0, c0) : l0));
                                l1 = __ffma2_rn(x1p, cx, __ffma2_rn(z1p, cz, k == 1 ? __fmul2_rn(u1, c0) : l1));
                                continue;
                            }
                            const float2 t0 = __ffma2_rn(z0p, cz, __fmul2_rn(x0p, cx));
                            const float2 t1 = __ffma2_rn(z1p, cz, __fmul2_rn(x1p, cx));
                            l0 = k == 1 ? __ffma2_rn(u0, c0, t0) : __fadd2_rn(l0, t0);
                            l1 = k == 1 ? __ffma2_rn(u1, c0, t1) : __fadd2_rn(l1, t1);
                        }
                        const float2 m1 = make_float2(-1.f, -1.f);
                        const float2 d0 = __ffma2_rn(make_float2(pr.x, pr.y), m1, __fadd2_rn(u0, u0));  // 2 u - pr
                        const float2 d1 = __ffma2_rn(make_float2(pr.z, pr.w), m1, __fadd2_rn(u1, u1));
                        const float2 o0 = __ffma2_rn(make_float2(vel[c].x, vel[c].y), l0, d0);
                        const float2 o1 = __ffma2_rn(make_float2(vel[c].z, vel[c].w), l1, d1);
                        o = make_float4(o0.x, o0.y, o1.x, o1.y);
                        lp = make_float4(l0.x, l0.y, l1.x, l1.y);
                    }
                    if (!ADJ && GEN) {
                        const bool xin = x0 + c >= NOP && x0 + c < n2 - NOP;
                        if (!(xin && z0 >= NOP && z0 < n1 - NOP)) o.x = pr.x;
                        if (!(xin && z0 + 1 >= NOP && z0 + 1 < n1 - NOP)) o.y = pr.y;
                        if (!(xin && z0 + 2 >= NOP && z0 + 2 < n1 - NOP)) o.z = pr.z;
                        if (!(xin && z0 + 3 >= NOP && z0 + 3 < n1 - NOP)) o.w = pr.w;
                        o.x = __fmul_rn(__fmul_rn(o.x, wz[0]), wx[c]);
                        o.y = __fmul_rn(__fmul_rn(o.y, wz[1]), wx[c]);
                        o.z = __fmul_rn(__fmul_rn(o.z, wz[2]), wx[c]);
                        o.w = __fmul_rn(__fmul_rn(o.w, wz[3]), wx[c]);
                    }
                    if (SLOTS) store(slot, c, ADJ || p.slot_level ? cur[c] : lp);
                    prv[c] = cur[c];
                    cur[c] = o;
                }
                // residuals of the thread's own cells: on mu, before it is weighted
                if (ADJ && my1 > my0) {
#pragma unroll
                    for (int c = 0; c < CX; c++) *reinterpret_cast<float4 *>(S1 + own + c * rz) = cur[c];
#pragma unroll 1
                    for (int s = my0; s < my1; s++) S1[cells[s].x] = with_entries(S1[cells[s].x], cells[s], j);
#pragma unroll
                    for (int c = 0; c < CX; c++) cur[c] = *reinterpret_cast<const float4 *>(S1 + own + c * rz);
                }
#pragma unroll
                for (int c = 0; c < CX; c++)
                    *reinterpret_cast<float4 *>(S1 + own + c * rz) = ADJ ? weighted(cur[c], c) : cur[c];
            }
            // receivers of the level this step reads, pending sponge applied (lint2d_extract)
            if (!ADJ && nrec > 0 && (p.jdata == 1 || it % p.jdata == 0)) {
                float *row = dat + (long long)(it / p.jdata) * nr;
                for (int r = tid; r < nrec; r += blockDim.x) {
                    const int2 li = rec_l[r];
                    const float4 w = rec_w[r], d = rec_d[r];
                    float v0 = S0[li.x], v1 = S0[li.x + 1], v2 = S0[li.x + rz], v3 = S0[li.x + rz + 1];
                    if (p.w1) {
                        v0 = __fmul_rn(__fmul_rn(v0, d.x), d.z), v1 = __fmul_rn(__fmul_rn(v1, d.y), d.z);
                        v2 = __fmul_rn(__fmul_rn(v2, d.x), d.w), v3 = __fmul_rn(__fmul_rn(v3, d.y), d.w);
                    }
                    float acc = __fmul_rn(v0, w.x);
                    if constexpr (EXACT) {
                        acc = __fadd_rn(acc, __fmul_rn(v1, w.y));
                        acc = __fadd_rn(acc, __fmul_rn(v2, w.z));
                        acc = __fadd_rn(acc, __fmul_rn(v3, w.w));
                    } else {
                        acc = fmaf(v3, w.w, fmaf(v2, w.z, fmaf(v1, w.y, acc)));
                    }
                    row[li.y] = acc;
                }
            }
            __syncthreads();
            if (!ADJ && ncell > 0) {  // sources on the new level, one thread per cell
                for (int s = tid; s < ncell; s += blockDim.x)
                    S1[cells[s].x] = with_entries(S1[cells[s].x], cells[s], j);
                __syncthreads();
#pragma unroll
                for (int c = 0; c < CX; c++) cur[c] = *reinterpret_cast<const float4 *>(S1 + own + c * rz);
            }
            float *t = S0;
            S0 = S1;
            S1 = t;
        }
    };
    if (inner && !damp) steps(std::false_type());
    else steps(std::true_type());
#pragma unroll
    for (int c = 0; c < CX; c++) {  // the last two levels
        store(p.ocur, c, cur[c]);
        store(p.oprv, c, prv[c]);
    }
}

template <int NOP, int MODE, int CX, bool BATCH = false>
static void launch_cx(const Tb2Params &p, const Tb2Shape &sh, size_t smem, cudaStream_t s, int ntile = 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = BATCH ? dim3(ntile) : dim3(sh.ntz, sh.ntx);
    cfg.blockDim = dim3((sh.rz / 4) * (sh.rx / CX));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaFuncSetAttribute(k_tb2<NOP, MODE, CX, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTb2SmemMax);
    cudaLaunchKernelEx(&cfg, k_tb2<NOP, MODE, CX, BATCH>, p);
}

template <int NOP, int CX>
static void launch_mode(int mode, const Tb2Params &p, const Tb2Shape &sh, size_t smem, cudaStream_t s) {
    switch (mode) {
        case 0: launch_cx<NOP, 0, CX>(p, sh, smem, s); break;
        case 1: launch_cx<NOP, 1, CX>(p, sh, smem, s); break;
        case 2: launch_cx<NOP, 2, CX>(p, sh, smem, s); break;
        default: launch_cx<NOP, 3, CX>(p, sh, smem, s); break;
    }
}

template <int NOP>
static void launch_nop(int mode, const Tb2Params &p, const Tb2Shape &sh, size_t smem, cudaStream_t s) {
    if (sh.cx == 1) launch_mode<NOP, 1>(mode, p, sh, smem, s);
    else if (sh.cx == 2) launch_mode<NOP, 2>(mode, p, sh, smem, s);
    else launch_mode<NOP, 4>(mode, p, sh, smem, s);
}

template <int NOP>
static void launch_batch(int mode, const Tb2Params &p, const Tb2Shape &sh, int ntile, size_t smem, cudaStream_t s) {
    if (mode == 0) launch_cx<NOP, 0, 4, true>(p, sh, smem, s, ntile);
    else if (mode == 2) launch_cx<NOP, 2, 4, true>(p, sh, smem, s, ntile);
    else launch_cx<NOP, 3, 4, true>(p, sh, smem, s, ntile);
}

}  // namespace

void launch_tb2_batch(int nop, int mode, const Tb2Params &p, const Tb2Shape &sh, int ntile, size_t smem,
                      cudaStream_t s) {
    switch (nop) {
        case 1: launch_batch<1>(mode, p, sh, ntile, smem, s); break;
        case 2: launch_batch<2>(mode, p, sh, ntile, smem, s); break;
        case 3: launch_batch<3>(mode, p, sh, ntile, smem, s); break;
        default: launch_batch<4>(mode, p, sh, ntile, smem, s); break;
    }
}

void launch_tb2(int nop, int mode, const Tb2Params &p, const Tb2Shape &sh, size_t smem, cudaStream_t s) {
    switch (nop) {
        case 1: launch_nop<1>(mode, p, sh, smem, s); break;
        case 2: launch_nop<2>(mode, p, sh, smem, s); break;
        case 3: launch_nop<3>(mode, p, sh, smem, s); break;
        default: launch_nop<4>(mode, p, sh, smem, s); break;
    }
}

// The imaging condition of a segment: G += I nu_k L(V_k) (or I nu_k V_k, the
// cross-correlation) and, at source cells, nu_k wav w, k from k1 - 1 down to
// k0.  One thread per cell keeps its compensated sum in registers over the
// segment; the levels come from the slots that the recompute (lap) and the
// adjoint sweep (nu) wrote, both read once.
__global__ void __launch_bounds__(256) k_tb2_image(float2 *__restrict__ G, const float *__restrict__ lap,
                                                   const float *__restrict__ nu, long long stride, const AdjParams p,
                                                   int k0, int k1) {
    const Grid g = p.g;
    const int i1 = blockIdx.x * 64 + threadIdx.x, i2 = blockIdx.y * 4 + threadIdx.y;
    if (i1 >= g.n1 || i2 >= g.n2) return;
    const long long i = (long long)i2 * g.n1 + i1;
    const bool in = i1 >= p.nop && i1 < g.n1 - p.nop && i2 >= p.nop && i2 < g.n2 - p.nop;
    const int e0 = p.wav && !p.xcorr ? p.sc_start[i] : 0, e1 = p.wav && !p.xcorr ? p.sc_start[i + 1] : 0;
    if (!in && e1 == e0) return;
    float2 a = G[i];
    const float *l = lap + i + (k1 - k0) * stride;  // slot k - k0: L(V_k)
    const float *n = nu + i;                        // slot k1 - 1 - k: nu_k
#pragma unroll 4
    for (int k = k1 - 1; k >= k0; k--) {
        l -= stride;
        const float x = *n;
        n += stride;
        if (in) a = gsum_add(a, __fmul_rn(x, *l));
        for (int e = e0; e < e1; e++) {
            const int2 en = p.sc_ent[e];
            const float dd = p.one_wavelet ? p.wav[(long long)k * p.ncs] : p.wav[(long long)k * p.ncs + en.x];
            a = gsum_add_prod(a, x, dd * __int_as_float(en.y));
        }
    }
    G[i] = a;
}

void launch_tb2_image(float2 *G, const float *lap, const float *nu, long long stride, const AdjParams &p, int k0,
                      int k1, cudaStream_t s) {
    k_tb2_image<<<dim3((p.g.n1 + 63) / 64, (p.g.n2 + 3) / 4), dim3(64, 4), 0, s>>>(G, lap, nu, stride, p, k0, k1);
}

// The same for a batch: four cells of axis 1 per thread; a shot's few sources
// are matched to the thread's cells once.
__global__ void __launch_bounds__(128) k_batch_image(float2 *__restrict__ G, const float *__restrict__ lap,
                                                     const float *__restrict__ nu, long long stride,
                                                     const BatchShot *__restrict__ shots,
                                                     const int2 *__restrict__ cols, int n1, int nop,
                                                     const GeoPoint *__restrict__ src, const float *__restrict__ wav,
                                                     int k0, int k1) {
    const int2 item = cols[blockIdx.x];
    const BatchShot sh = shots[item.x];
    const int z = 4 * (blockIdx.y * 32 + threadIdx.x), x = item.y + threadIdx.y;
    if (z >= n1 || x >= sh.n2) return;
    const long long cell = (long long)x * n1 + z, i = sh.off + cell;
    bool in[4], src_here = false;
#pragma unroll
    for (int c = 0; c < 4; c++) in[c] = x >= nop && x < sh.n2 - nop && z + c >= nop && z + c < n1 - nop;
    for (int q = 0; q < sh.ns; q++) {  // corners lie within n1 + 1 of the base index
        const long long b = src[sh.src0 + q].base - cell;
        src_here = src_here || (b >= -(long long)n1 - 1 && b <= 3);
    }
    float4 *g = reinterpret_cast<float4 *>(G + i);
    const float4 g0 = g[0], g1 = g[1];
    float2 a[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
    const float *l = lap + i + (k1 - k0) * stride;  // slot k - k0: L(V_k)
    const float *n = nu + i;                        // slot k1 - 1 - k: nu_k
#pragma unroll 4
    for (int k = k1 - 1; k >= k0; k--) {
        l -= stride;
        const float4 lv = __ldcs(reinterpret_cast<const float4 *>(l)), nv = __ldcs(reinterpret_cast<const float4 *>(n));
        n += stride;
        const float lf[4] = {lv.x, lv.y, lv.z, lv.w}, nf[4] = {nv.x, nv.y, nv.z, nv.w};
#pragma unroll
        for (int c = 0; c < 4; c++)
            if (in[c]) a[c] = gsum_add(a[c], __fmul_rn(nf[c], lf[c]));
        if (src_here) {
            const float dd = wav[k];
#pragma unroll 1
            for (int q = 0; q < sh.ns; q++) {
                const GeoPoint gp = src[sh.src0 + q];
#pragma unroll
                for (int cc = 0; cc < 4; cc++) {
                    const long long d = gp.base + (cc & 1) + (cc >> 1) * (long long)n1 - cell;
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (d == c) a[c] = gsum_add_prod(a[c], nf[c], __fmul_rn(dd, gp.w[cc]));
                }
            }
        }
    }
    g[0] = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
    g[1] = make_float4(a[2].x, a[2].y, a[3].x, a[3].y);
}

void launch_batch_image(float2 *G, const float *lap, const float *nu, long long stride, const BatchShot *shots,
                        const int2 *cols, int ncols, int n1, int nop, const GeoPoint *src, const float *wav, int k0,
                        int k1, cudaStream_t s) {
    k_batch_image<<<dim3(ncols, (n1 / 4 + 31) / 32), dim3(32, 4), 0, s>>>(G, lap, nu, stride, shots, cols, n1, nop, src,
                                                                         wav, k0, k1);
}

}  // namespace awe
