// The boundary work of one 3D step of the CPU-program scheme in one launch:
// the one-way ABC of the six faces (abcone3d_apply, fdutil.c:2085-2177), the
// sponge of the shell the step kernel left unsponged (sponge3d_apply,
// fdutil.c:2248-2310), the receiver gather of the level the step read
// (lint3d_extract, fdutil.c:1653-1670) and, when no source touches a cell that
// another role stores, the injection (lint3d_inject1_with_vv,
// fdutil.c:1723-1740).
//
// The reference applies the ABC as three passes over the whole grid (axis-1
// lines, then axis-2 lines, then axis-3 lines, each an outward recurrence over
// the nop outer cells from cell nop + 1), then the sponge.  The passes only
// meet in the shell (cells within nop + 2 of a face), so the work splits into
// roles, longest chain first, that each own whole chains of dependencies:
//  * a plane y in [nop+2, n3-nop-2) (no axis-3 face cell), its axis-2 shell
//    lines: their axis-1 ends, then (after a barrier) the axis-2 pass with the
//    sponge, four z cells per thread;
//  * a face block (the nop + 2 planes of a y face) x about 16 columns x about
//    32 cells of axis 1: the axis-1 pass of its line ends, the axis-2 pass
//    (x-ranges holding a face), then the axis-3 pass and the sponge of its
//    columns together, four z cells per thread;
//  * the axis-1 ends of every other line, one thread per end, sponged;
//  * receiver blocks (256 receivers each) and the injection, which read or
//    write cells no pass touches.
// Latency bounds it but on the largest grids: every role is two or three
// dependent rounds of loads, so they are kept short and the blocks many.  (A
// block per plane for both its passes, and face blocks of up to 31 x 124
// columns one cell at a time: 22.5 us for 251 x 223 x 199 cells at 4th order,
// 52 us for 576^3 at 8th; so 11.8 us and 51 us, the scattered sectors of the
// line ends.)
// Every cell is written by one block only, so the result does not depend on
// the order in which blocks run.
//
// The axis-1 ends (8 cells at each end of every line, 32 bytes of every
// p1*4-byte line) are the scattered part of the work.  Within a forward run
// each launch also writes the final ends of the new level to a compact
// [n3][n2][16] copy, and the next step's launch reads the ends of the level
// its step read (the same values) from that copy with coalesced loads
// instead of one scattered sector per line end.
#include <cuda_runtime.h>

#include "awe_internal.h"
#include "fp_exact.cuh"

namespace awe {

namespace b3 {
constexpr int SHELL = 6;  // the adjoint's nop + 2 (nop = 4): cells the ABC writes (1..4) or reads (5), and the face cell 0
constexpr int XR = 16, ZQ = 8;  // face blocks: least columns and 4-cell groups of axis 1
constexpr int NT = 256;
static_assert(kBndEnd == 8, "b3_ld8, b3_st8: the cells of a line end");
}  // namespace b3

template <bool EXACT>
__device__ __forceinline__ float b3_abc(float um_in, float um_c, float uo_in, float b) {
    // uo = um[inner] + (um[c] - uo[inner]) * b
    return fadd<EXACT>(um_in, fmul<EXACT>(fsub<EXACT>(um_c, uo_in), b));
}

template <bool EXACT>
__device__ __forceinline__ float b3_damp(float v, float wz, float wx, float wy) {
    return fmul<EXACT>(fmul<EXACT>(fmul<EXACT>(v, wz), wx), wy);
}

// Axis-1 line ends: cells 0..7 and n1-8..n1-1 in registers.  Lines start on
// 16-byte boundaries (the pitch p1), so the low end is two 16-byte accesses;
// the high end is too where n1 % 4 == 0 (AL), else 8 scalar ones in the same
// two sectors.
template <bool AL>
__device__ __forceinline__ void b3_ld8(float (&v)[8], const float *a) {
    if constexpr (AL) {
        const float4 x = *reinterpret_cast<const float4 *>(a), y = *reinterpret_cast<const float4 *>(a + 4);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = a[k];
    }
}

template <bool AL>
__device__ __forceinline__ void b3_st8(float *a, const float (&v)[8]) {
    if constexpr (AL) {
        *reinterpret_cast<float4 *>(a) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(a + 4) = make_float4(v[4], v[5], v[6], v[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = v[k];
    }
}

// low face: cells NOP .. 1 from cell NOP+1
template <bool EXACT, int NOP>
__device__ __forceinline__ void b3_zlow(float (&v)[8], const float (&m)[8], float c) {
#pragma unroll
    for (int k = NOP; k >= 1; k--) v[k] = b3_abc<EXACT>(m[k + 1], m[k], v[k + 1], c);
}

// high face: cells n1-1-NOP .. n1-2 from n1-2-NOP (v[7] is cell n1-1)
template <bool EXACT, int NOP>
__device__ __forceinline__ void b3_zhigh(float (&v)[8], const float (&m)[8], float c) {
#pragma unroll
    for (int k = NOP; k >= 1; k--) v[7 - k] = b3_abc<EXACT>(m[6 - k], m[7 - k], v[6 - k], c);
}

// sponge of the elements of an end that lie in the shell (mask bit per element; w = w1 at element 0)
template <bool EXACT, bool AL>
__device__ __forceinline__ void b3_damp8(float (&v)[8], const float *w, float wx, float wy, unsigned mask) {
    float wz[8];
    b3_ld8<AL>(wz, w);
#pragma unroll
    for (int k = 0; k < 8; k++)
        if ((mask >> k) & 1u) v[k] = b3_damp<EXACT>(v[k], wz[k], wx, wy);
}

// coefficients of cells z .. z+3 of a face line (cells past n1: 0)
template <bool AL>
__device__ __forceinline__ void b3_coef4(float (&b)[4], const float *row, int z, int n1) {
    if constexpr (AL) {
        const float4 x = __ldg(reinterpret_cast<const float4 *>(row + z));
        b[0] = x.x, b[1] = x.y, b[2] = x.z, b[3] = x.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) b[i] = z + i < n1 ? __ldg(row + z + i) : 0.f;
    }
}

// Cells z .. z+3 of a face's recurrence along axis AXIS (2 or 3): NOP cells
// outward (st) from the one at c0, all NOP + 2 shell cells sponged if damp.
// wv: the sponge factors along AXIS at c0, dw their step; wc: the other one.
template <bool EXACT, int NOP, int AXIS>
__device__ __forceinline__ void b3_chain4(const Bnd3Params &p, long long c0, long long st, const float (&b)[4], int z,
                                          bool damp, const float *wv, int dw, float wc) {
    auto ld = [](float (&v)[4], const float *a) {
        const float4 x = *reinterpret_cast<const float4 *>(a);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    };
    float v[4], f[4], m[NOP + 1][4], wz[4];
    ld(v, p.uo + c0);
    if (damp) {
        ld(f, p.uo + c0 + (NOP + 1) * st);
        ld(wz, p.w1 + z);
    }
#pragma unroll
    for (int k = 0; k <= NOP; k++) ld(m[k], p.um + c0 + k * st);
    auto put = [&](const float (&v)[4], int k) {
        float o[4];
        const float w = damp ? __ldg(wv + k * dw) : 1.f;
#pragma unroll
        for (int i = 0; i < 4; i++)
            o[i] = !damp ? v[i] : AXIS == 2 ? b3_damp<EXACT>(v[i], wz[i], w, wc) : b3_damp<EXACT>(v[i], wz[i], wc, w);
        *reinterpret_cast<float4 *>(p.uo + c0 + k * st) = make_float4(o[0], o[1], o[2], o[3]);
    };
    if (damp) {
        put(v, 0);
        put(f, NOP + 1);
    }
#pragma unroll
    for (int k = 1; k <= NOP; k++) {
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = b3_abc<EXACT>(m[k - 1][i], m[k][i], v[i], b[i]);
        put(v, k);
    }
}

// an axis-2 face of plane y, cells z .. z+3
template <bool EXACT, int NOP, bool AL>
__device__ __forceinline__ void b3_xchain(const Bnd3Params &p, int y, int z, bool low, bool damp) {
    const long long s2 = p.g.p1;
    const int xa = low ? NOP + 1 : p.g.n2 - NOP - 2, dx = low ? -1 : 1;
    float b[4];
    b3_coef4<AL>(b, (low ? p.xl : p.xh) + (long long)y * p.g.n1, z, p.g.n1);
    b3_chain4<EXACT, NOP, 2>(p, ((long long)y * p.g.n2 + xa) * s2 + z, dx * s2, b, z, damp, p.w2 + xa, dx,
                             damp ? __ldg(p.w3 + y) : 1.f);
}

// an end (0: cells 0..7, 1: cells n1-8..n1-1) of line `line` of the level the
// step read: from the compact copy of its line ends the previous step's
// launch wrote (em), else from the level itself
template <bool AL>
__device__ __forceinline__ void b3_mend(const Bnd3Params &p, float (&m)[8], long long line, int end) {
    if (p.em) return b3_ld8<true>(m, p.em + line * 16 + 8 * end);
    const float *r = p.um + line * p.g.p1;
    if (end == 0) b3_ld8<true>(m, r);
    else b3_ld8<AL>(m, r + p.g.n1 - 8);
}

// the compact copy of the new level's line ends (eo), read back from uo once
// the line's cells are final; part 0..3: 4 cells each
template <bool AL>
__device__ __forceinline__ void b3_eput_from_uo(const Bnd3Params &p, long long line, int part) {
    const float *o = p.uo + line * p.g.p1 + (part < 2 ? 4 * part : p.g.n1 - 16 + 4 * part);
    float4 v;
    if (AL || part < 2) v = *reinterpret_cast<const float4 *>(o);
    else v = make_float4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<float4 *>(p.eo)[line * 4 + part] = v;
}

// One end of line (y, x) (0: low, 1: high): the axis-1 recurrence and, with
// damp, the sponge of its shell cells; all eight cells are stored, so no source
// of this launch lies on them; the final values go to the compact copy
// if put (without a sponge and with a free surface the low end is not read,
// nor needed: the next step's low-end recurrence is off).
template <bool EXACT, int NOP, bool AL>
__device__ __forceinline__ void b3_end(const Bnd3Params &p, int y, int x, int end, bool damp, bool put) {
    constexpr unsigned LOW = (1u << (NOP + 2)) - 1u, HIGH = LOW << (6 - NOP);  // of 8, those in the shell
    const long long line = (long long)y * p.g.n2 + x;
    float v[8] = {}, m[8];
    const float wx = damp ? __ldg(p.w2 + x) : 1.f, wy = damp ? __ldg(p.w3 + y) : 1.f;
    if (end == 0) {
        if (p.top || damp) {
            float *o = p.uo + line * p.g.p1;
            b3_ld8<true>(v, o);
            if (p.top) {
                b3_mend<AL>(p, m, line, 0);
                b3_zlow<EXACT, NOP>(v, m, __ldg(p.zl + line));
            }
            if (damp) b3_damp8<EXACT, true>(v, p.w1, wx, wy, LOW);
            b3_st8<true>(o, v);
        }
    } else {
        float *o = p.uo + line * p.g.p1 + p.g.n1 - 8;
        b3_ld8<AL>(v, o);
        b3_mend<AL>(p, m, line, 1);
        b3_zhigh<EXACT, NOP>(v, m, __ldg(p.zh + line));
        if (damp) b3_damp8<EXACT, AL>(v, p.w1 + p.g.n1 - 8, wx, wy, HIGH);
        b3_st8<AL>(o, v);
    }
    if (put) b3_st8<true>(p.eo + line * 16 + 8 * end, v);
}

template <bool EXACT, int NOP, bool AL>
__global__ void __launch_bounds__(b3::NT, 3) k_bnd3(const Bnd3Params p) {
    using b3::NT;
    constexpr int SHELL = NOP + 2;
    const int tid = threadIdx.x;
    const int n1 = p.g.n1, n2 = p.g.n2, n3 = p.g.n3, nq = (n1 + 3) / 4;
    const long long s2 = p.g.p1, s3 = s2 * n2;
    const bool sponge = p.w1 != nullptr;
    int blk = blockIdx.x;

    if (blk < p.n_int) {  // ---- the axis-2 shell of a plane without axis-3 face cells
        const int y = SHELL + blk;
        if (tid < 4 * SHELL) {
            const int k = tid >> 1;
            b3_end<EXACT, NOP, AL>(p, y, k < SHELL ? k : n2 - 2 * SHELL + k, tid & 1, false, false);
        }
        __syncthreads();
        for (int l = tid; l < 2 * nq; l += NT) {
            const bool low = l < nq;
            b3_xchain<EXACT, NOP, AL>(p, y, 4 * (low ? l : l - nq), low, sponge);
        }
        if (p.eo) {
            __syncthreads();
            if (tid < 8 * SHELL) {
                const int k = tid >> 2, x = k < SHELL ? k : n2 - 2 * SHELL + k;
                b3_eput_from_uo<AL>(p, (long long)y * n2 + x, tid & 3);
            }
        }
        return;
    }
    blk -= p.n_int;
    if (blk < 2 * p.nxr * p.nzr) {  // ---- face block
        const int f = blk / (p.nxr * p.nzr), r = blk % (p.nxr * p.nzr), xr = r / p.nzr, zr = r % p.nzr;
        const int xa = (int)((long long)n2 * xr / p.nxr), xb = (int)((long long)n2 * (xr + 1) / p.nxr);
        const int qa = (int)((long long)nq * zr / p.nzr), qb = (int)((long long)nq * (zr + 1) / p.nzr);
        const int ya = f == 0 ? 0 : n3 - SHELL;  // planes [ya, ya + SHELL)
        const int ncol = xb - xa, nqz = qb - qa;
        // axis 1: the line ends inside this z-range
        const bool zlo = zr == 0, zhi = zr == p.nzr - 1;
        if ((zlo && p.top) || zhi) {
            for (int l = tid; l < 2 * SHELL * ncol; l += NT) {
                const int k = l >> 1;
                if (l & 1 ? zhi : zlo && p.top)
                    b3_end<EXACT, NOP, AL>(p, ya + k / ncol, xa + k % ncol, l & 1, false, false);
            }
            __syncthreads();
        }
        // axis 2: the x-ranges holding a face
        const bool xlo = xr == 0, xhi = xr == p.nxr - 1;
        if (xlo || xhi) {
            for (int l = tid; l < SHELL * nqz; l += NT) {
                const int y = ya + l / nqz, z = 4 * (qa + l % nqz);
                if (xlo) b3_xchain<EXACT, NOP, AL>(p, y, z, true, false);
                if (xhi) b3_xchain<EXACT, NOP, AL>(p, y, z, false, false);
            }
            __syncthreads();
        }
        // axis 3 and the sponge (all cells lie in the axis-3 shell; the pad cells of a line hold 0)
        const int y0 = f == 0 ? NOP + 1 : n3 - SHELL, dy = f == 0 ? -1 : 1;
        for (int l = tid; l < ncol * nqz; l += NT) {
            const int x = xa + l / nqz, z = 4 * (qa + l % nqz);
            float b[4];
            b3_coef4<AL>(b, (f == 0 ? p.yl : p.yh) + (long long)x * n1, z, n1);
            b3_chain4<EXACT, NOP, 3>(p, y0 * s3 + x * s2 + z, dy * s3, b, z, sponge, p.w3 + y0, dy,
                                     sponge ? __ldg(p.w2 + x) : 1.f);
        }
        if (p.eo && (zlo || zhi)) {  // the line ends this block holds, final now
            __syncthreads();
            for (int l = tid; l < SHELL * ncol * 4; l += NT) {
                const int k = l >> 2, part = l & 3;
                if (part < 2 ? zlo : zhi)
                    b3_eput_from_uo<AL>(p, (long long)(ya + k / ncol) * n2 + xa + k % ncol, part);
            }
        }
        return;
    }
    blk -= 2 * p.nxr * p.nzr;
    if (blk < p.end_blocks) {  // ---- axis-1 ends of the other lines
        const int ni = n2 - 2 * SHELL, t = blk * NT + tid, l = t >> 1;
        if (l < ni * p.n_int) b3_end<EXACT, NOP, AL>(p, SHELL + l / ni, SHELL + l % ni, t & 1, sponge, p.eo != nullptr);
        return;
    }
    blk -= p.end_blocks;
    if (blk < p.rec_blocks) {  // ---- receiver gather of um (its pending sponge applied)
        const int r = blk * NT + tid;
        if (r >= p.nr) return;
        const GeoPoint pt = p.rec[(long long)r * p.rec_stride];
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const long long n = pt.base + ((c & 1) ? 1 : 0) + ((c & 2) ? s2 : 0) + ((c & 4) ? s3 : 0);
            float v = __ldg(p.um + n);
            if (p.w1) {
                const int i3 = (int)(n / s3), rem = (int)(n % s3);
                v = fmul<EXACT>(v, __ldg(p.w1 + rem % (int)s2));
                v = fmul<EXACT>(v, __ldg(p.w2 + rem / (int)s2));
                v = fmul<EXACT>(v, __ldg(p.w3 + i3));
            }
            const float t = fmul<EXACT>(v, pt.w[c]);
            acc = (c == 0) ? t : fadd<EXACT>(acc, t);
        }
        p.rec_row[r] = acc;
        return;
    }
    blk -= p.rec_blocks;
    if (p.inj.n > 0) {  // ---- injection, one thread per cell
        const int k = blk * NT + tid;
        if (k >= p.inj.n) return;
        const long long n = p.inj.cell[k];
        float v = p.uo[n];
        const float vn = p.vel[n];
        for (int e = p.inj.start[k], e1 = p.inj.start[k + 1]; e < e1; e++) {
            const int2 en = p.inj.ent[e];
            const float dd =
                p.one_wavelet ? p.wav[(long long)p.it * p.ncs] : p.wav[(long long)p.it * p.ncs + (en.x >> 3)];
            v = fadd<EXACT>(v, fmul<EXACT>(fmul<EXACT>(dd, __int_as_float(en.y)), vn));
        }
        p.uo[n] = v;
        return;
    }
    if (blk == 0 && p.ns > 0 && tid == 0) {  // ---- injection, sources and corners in order
        for (int s = 0; s < p.ns; s++) {
            const float dd = p.one_wavelet ? p.wav[(long long)p.it * p.ncs] : p.wav[(long long)p.it * p.ncs + s];
            const GeoPoint pt = p.src[(long long)s * p.src_stride];
            for (int c = 0; c < 8; c++) {
                const long long n = pt.base + ((c & 1) ? 1 : 0) + ((c & 2) ? s2 : 0) + ((c & 4) ? s3 : 0);
                p.uo[n] = fadd<EXACT>(p.uo[n], fmul<EXACT>(fmul<EXACT>(dd, pt.w[c]), p.vel[n]));
            }
        }
    }
}

bool bnd3_eligible(int nop, const Grid &g) {
    // both ends of a line in their 8 cells, every face's shell apart from the opposite one
    return nop <= 4 && g.p1 % 4 == 0 && g.n1 >= 16 && g.n2 >= 2 * (nop + 2) && g.n3 >= 2 * (nop + 2);
}

template <bool EXACT, int NOP>
static void launch_bnd3_nop(const Bnd3Params &p, int grid, cudaStream_t s) {
    if (p.g.n1 % 4 == 0) k_bnd3<EXACT, NOP, true><<<grid, b3::NT, 0, s>>>(p);
    else k_bnd3<EXACT, NOP, false><<<grid, b3::NT, 0, s>>>(p);
}

void launch_bnd3(bool exact, Bnd3Params p, cudaStream_t s) {
    using namespace b3;
    p.n_int = p.g.n3 - 2 * (p.nop + 2);
    p.nxr = p.g.n2 / XR > 0 ? p.g.n2 / XR : 1;
    p.nzr = (p.g.n1 + 3) / 4 / ZQ > 0 ? (p.g.n1 + 3) / 4 / ZQ : 1;
    p.end_blocks = (int)((2LL * p.n_int * (p.g.n2 - 2 * (p.nop + 2)) + NT - 1) / NT);
    p.rec_blocks = p.rec_row ? (p.nr + NT - 1) / NT : 0;
    const int grid = p.n_int + 2 * p.nxr * p.nzr + p.end_blocks + p.rec_blocks + (p.inj.n > 0 ? (p.inj.n + NT - 1) / NT : p.ns > 0 ? 1 : 0);
    switch (p.nop) {
        case 1: return exact ? launch_bnd3_nop<true, 1>(p, grid, s) : launch_bnd3_nop<false, 1>(p, grid, s);
        case 2: return exact ? launch_bnd3_nop<true, 2>(p, grid, s) : launch_bnd3_nop<false, 2>(p, grid, s);
        case 3: return exact ? launch_bnd3_nop<true, 3>(p, grid, s) : launch_bnd3_nop<false, 3>(p, grid, s);
        default: return exact ? launch_bnd3_nop<true, 4>(p, grid, s) : launch_bnd3_nop<false, 4>(p, grid, s);
    }
}

// ---------------------------------------------------------------------------
// The boundary work before one adjoint step of the 3D gradient in one launch:
//  1. fold the previous adjoint step's kappa into mu on the shell (mu += W
//     kappa, kappa = 0; cells within nop + 2 of a face),
//  2. the transpose of the one-way ABC (abcone3d_apply, fdutil.c:2085-2177),
//     passes in reverse order (axis 3, axis 2, axis 1) and updates within a
//     line in reverse order: t = mu[i]; mu[i] = 0; mu[b] -= c t;
//     kappa[b] += t; kappa[i] += c t (b the inward neighbour of i),
//  3. g = I vel2 mu on every cell (I: at least nop from every face), the
//     field the adjoint step's stencil reads.
// Roles by block as in k_bnd3, so each cell's chain runs in one block: the
// axis-2 shell of a plane y in [6, n3-6) (fold, axis-2 transpose, then its
// lines' ends, then g); a face block (6 axis-3 face planes x about 16 columns
// x about 32 cells: fold and axis-3 transpose, axis 2, line ends, g); the ends of
// every other line with their g, one thread per end; and the g of all other
// cells, which nothing changes.  The result does not depend on block order.
// The g pass streams 12 bytes a cell and bounds it.  (A block per plane for all
// of its work: 51 us for 208 x 192 x 198 cells; so 24.6 us.)
namespace b3a {
__device__ __forceinline__ void tcell(float &mi, float &mb, float &kb, float &ki, float c) {
    const float v = mi;
    mi = 0.f;
    mb -= c * v;
    kb += v;
    ki += c * v;
}

__device__ __forceinline__ float wcell3(const Bnd3AdjParams &p, int z, int x, int y) {
    if (!p.w1) return 1.f;
    return __ldg(p.w1 + z) * __ldg(p.w2 + x) * __ldg(p.w3 + y);
}

// mu += W kappa, kappa = 0 (cells whose kappa is 0 keep their value)
__device__ __forceinline__ void fold(const Bnd3AdjParams &p, float &m, float &k, int z, int x, int y) {
    if (k != 0.f) {
        m += wcell3(p, z, x, y) * k;
        k = 0.f;
    }
}

__device__ __forceinline__ void ld4(float (&v)[4], const float *a) {
    const float4 t = *reinterpret_cast<const float4 *>(a);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
__device__ __forceinline__ void st4(float *a, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(a) = make_float4(v[0], v[1], v[2], v[3]);
}

// Cells z .. z+3 of a face along axis AXIS (2 or 3): the six shell cells from
// the face cell at c0 inward (st); optional fold, then the transposed updates
// of cells 4 .. 1 (high face: the one next to the face first) in registers.
// (x, y) is the face cell, d the step inward; row the face's coefficients.
template <int AXIS>
__device__ __forceinline__ void face4(const Bnd3AdjParams &p, long long c0, long long st, const float *row, int z, int x,
                                      int y, int d, bool dofold) {
    float m[6][4], k[6][4], c[4];
#pragma unroll
    for (int j = 0; j < 6; j++) {
        ld4(m[j], p.mu + c0 + j * st);
        ld4(k[j], p.kap + c0 + j * st);
    }
    {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(row + z));
        c[0] = t.x, c[1] = t.y, c[2] = t.z, c[3] = t.w;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (dofold)
#pragma unroll
            for (int j = 0; j < 6; j++)
                fold(p, m[j][i], k[j][i], z + i, AXIS == 2 ? x + j * d : x, AXIS == 3 ? y + j * d : y);
#pragma unroll
        for (int j = 1; j <= 4; j++) tcell(m[j][i], m[j + 1][i], k[j + 1][i], k[j][i], c[i]);
    }
#pragma unroll
    for (int j = 0; j < 6; j++) {
        st4(p.mu + c0 + j * st, m[j]);
        st4(p.kap + c0 + j * st, k[j]);
    }
}

// one end of line (y, x) (0: cells 0..7, 1: n1-8..n1-1; n1 % 4 == 0): optional
// fold of the shell cells, then the transposed updates, in registers (m: as left)
__device__ __forceinline__ void lend(const Bnd3AdjParams &p, int y, int x, int end, bool dofold, float (&m)[8]) {
    const long long line = (long long)y * p.g.n2 + x;
    const int z0 = end ? p.g.n1 - 8 : 0;
    float *M = p.mu + line * p.g.n1 + z0, *K = p.kap + line * p.g.n1 + z0;
    float k[8];
    b3_ld8<true>(m, M);
    b3_ld8<true>(k, K);
    if (dofold)
#pragma unroll
        for (int j = 0; j < 6; j++) {  // the shell: elements 0..5 or 2..7
            const int e = end ? j + 2 : j;
            if (end) fold(p, m[j + 2], k[j + 2], z0 + e, x, y);
            else fold(p, m[j], k[j], z0 + e, x, y);
        }
    if (end) {
        const float h = __ldg(p.zh + line);
#pragma unroll
        for (int j = 1; j <= 4; j++) tcell(m[7 - j], m[6 - j], k[6 - j], k[7 - j], h);
    } else if (p.top) {
        const float l = __ldg(p.zl + line);
#pragma unroll
        for (int j = 1; j <= 4; j++) tcell(m[j], m[j + 1], k[j + 1], k[j], l);
    }
    b3_st8<true>(M, m);
    b3_st8<true>(K, k);
}

// g = I vel2 mu on the 4 cells z .. z+3 of line (y, x) (z % 4 == 0), from
// loaded values
__device__ __forceinline__ void gstore(const Bnd3AdjParams &p, int y, int z, int x, float4 m, float4 v) {
    const int n1 = p.g.n1, n2 = p.g.n2, n3 = p.g.n3;
    const long long c = ((long long)y * n2 + x) * n1 + z;
    const bool rest = x >= 4 && x < n2 - 4 && y >= 4 && y < n3 - 4;
    float4 o;
    o.x = (rest && z >= 4 && z < n1 - 4) ? v.x * m.x : 0.f;
    o.y = (rest && z + 1 >= 4 && z + 1 < n1 - 4) ? v.y * m.y : 0.f;
    o.z = (rest && z + 2 >= 4 && z + 2 < n1 - 4) ? v.z * m.z : 0.f;
    o.w = (rest && z + 3 >= 4 && z + 3 < n1 - 4) ? v.w * m.w : 0.f;
    __stcs(reinterpret_cast<float4 *>(p.gout + c), o);
}

__device__ __forceinline__ void gcells(const Bnd3AdjParams &p, int y, int z, int x) {
    const long long c = ((long long)y * p.g.n2 + x) * p.g.n1 + z;
    gstore(p, y, z, x, *reinterpret_cast<const float4 *>(p.mu + c), __ldg(reinterpret_cast<const float4 *>(p.vel2 + c)));
}

}  // namespace b3a

__global__ void __launch_bounds__(b3::NT, 2) k_bnd3_adj(const Bnd3AdjParams p) {
    using namespace b3;
    using namespace b3a;
    const int tid = threadIdx.x;
    const int n1 = p.g.n1, n2 = p.g.n2, n3 = p.g.n3, nq = n1 / 4;
    const long long s2 = n1, s3 = (long long)n1 * n2;
    int blk = blockIdx.x;
    float m[8];

    if (blk < p.n_int) {  // ---- the axis-2 shell of a plane without axis-3 face cells
        const int y = SHELL + blk;
        for (int l = tid; l < 2 * nq; l += NT) {
            const bool low = l < nq;
            const int z = 4 * (low ? l : l - nq), x = low ? 0 : n2 - 1, d = low ? 1 : -1;
            face4<2>(p, (long long)y * s3 + x * s2 + z, d * s2, (low ? p.xl : p.xh) + (long long)y * n1, z, x, y, d, true);
        }
        __syncthreads();
        if (tid < 4 * SHELL) {
            const int k = tid >> 1;
            lend(p, y, k < SHELL ? k : n2 - 2 * SHELL + k, tid & 1, false, m);
        }
        __syncthreads();
        for (int l = tid; l < 2 * SHELL * nq; l += NT) {
            const int k = l / nq;
            gcells(p, y, 4 * (l % nq), k < SHELL ? k : n2 - 2 * SHELL + k);
        }
        return;
    }
    blk -= p.n_int;
    if (blk < 2 * p.nxr * p.nzr) {  // ---- face block
        const int f = blk / (p.nxr * p.nzr), r = blk % (p.nxr * p.nzr), xr = r / p.nzr, zr = r % p.nzr;
        const int xa = (int)((long long)n2 * xr / p.nxr), xb = (int)((long long)n2 * (xr + 1) / p.nxr);
        const int qa = (int)((long long)nq * zr / p.nzr), qb = (int)((long long)nq * (zr + 1) / p.nzr);
        const int ya = f == 0 ? 0 : n3 - SHELL;
        const int ncol = xb - xa, nqz = qb - qa;
        // fold (every cell lies in the axis-3 shell) and axis 3
        const int yf = f == 0 ? 0 : n3 - 1, dy = f == 0 ? 1 : -1;
        for (int l = tid; l < ncol * nqz; l += NT) {
            const int x = xa + l / nqz, z = 4 * (qa + l % nqz);
            face4<3>(p, yf * s3 + x * s2 + z, dy * s3, (f == 0 ? p.yl : p.yh) + (long long)x * n1, z, x, yf, dy, true);
        }
        __syncthreads();
        // axis 2: the x-ranges holding a face
        const bool xlo = xr == 0, xhi = xr == p.nxr - 1;
        if (xlo || xhi) {
            for (int l = tid; l < SHELL * nqz; l += NT) {
                const int y = ya + l / nqz, z = 4 * (qa + l % nqz);
                const long long c = (long long)y * s3 + z, row = (long long)y * n1;
                if (xhi) face4<2>(p, c + (n2 - 1) * s2, -s2, p.xh + row, z, n2 - 1, y, -1, false);
                if (xlo) face4<2>(p, c, s2, p.xl + row, z, 0, y, 1, false);
            }
            __syncthreads();
        }
        // axis 1: the line ends inside this z-range
        const bool zlo = zr == 0, zhi = zr == p.nzr - 1;
        if (zlo || zhi) {
            for (int l = tid; l < 2 * SHELL * ncol; l += NT) {
                const int k = l >> 1;
                if (l & 1 ? zhi : zlo && p.top) lend(p, ya + k / ncol, xa + k % ncol, l & 1, false, m);
            }
            __syncthreads();
        }
        for (int l = tid; l < SHELL * ncol * nqz; l += NT) {
            const int k = l / nqz;
            gcells(p, ya + k / ncol, 4 * (qa + l % nqz), xa + k % ncol);
        }
        return;
    }
    blk -= 2 * p.nxr * p.nzr;
    const int ni = n2 - 2 * SHELL;
    if (blk < p.end_blocks) {  // ---- axis-1 ends of the other lines, and their g
        const int t = blk * NT + tid, l = t >> 1, end = t & 1;
        if (l >= ni * p.n_int) return;
        const int y = SHELL + l / ni, x = SHELL + l % ni, z = end ? n1 - 8 : 0;
        float v[8];
        b3_ld8<true>(v, p.vel2 + ((long long)y * n2 + x) * n1 + z);
        lend(p, y, x, end, true, m);
        gstore(p, y, z, x, make_float4(m[0], m[1], m[2], m[3]), make_float4(v[0], v[1], v[2], v[3]));
        gstore(p, y, z + 4, x, make_float4(m[4], m[5], m[6], m[7]), make_float4(v[4], v[5], v[6], v[7]));
        return;
    }
    blk -= p.end_blocks;
    // ---- g of the cells no transposed update touches, four groups of 4 cells per thread in flight
    const int per = (ni * nq + 4 * NT - 1) / (4 * NT), y = SHELL + blk / per, l0 = blk % per * 4 * NT + tid;
    const long long base = ((long long)y * n2 + SHELL) * n1;
    float4 a[4], v[4];
    bool in[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int l = l0 + u * NT, q = l % nq;
        in[u] = l < ni * nq && q >= 2 && q < nq - 2;
        if (in[u]) {
            a[u] = *reinterpret_cast<const float4 *>(p.mu + base + 4LL * l);
            v[u] = __ldg(reinterpret_cast<const float4 *>(p.vel2 + base + 4LL * l));
        }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int l = l0 + u * NT;
        if (in[u]) gstore(p, y, 4 * (l % nq), SHELL + l / nq, a[u], v[u]);
    }
}

void launch_bnd3_adj(Bnd3AdjParams p, cudaStream_t s) {
    using namespace b3;
    const int nq = p.g.n1 / 4, ni = p.g.n2 - 2 * SHELL;
    p.n_int = p.g.n3 - 2 * SHELL;
    p.nxr = p.g.n2 / XR > 0 ? p.g.n2 / XR : 1;
    p.nzr = nq / ZQ > 0 ? nq / ZQ : 1;
    p.end_blocks = (int)((2LL * p.n_int * ni + NT - 1) / NT);
    const int inner = p.n_int * ((ni * nq + 4 * NT - 1) / (4 * NT));
    k_bnd3_adj<<<p.n_int + 2 * p.nxr * p.nzr + p.end_blocks + inner, NT, 0, s>>>(p);
}

}  // namespace awe
