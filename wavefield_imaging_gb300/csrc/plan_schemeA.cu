// Host side of the GPU-program scheme (MAWEFD{cart,spher}{2D,3D}gpu.cu):
// padding, sponge and metric tables, one-way coefficients, injection scales
// and the per-step launch sequence.  Host arithmetic follows the reference's
// float expressions (built with -ffp-contract=off); float arguments to the
// math functions use the float overloads, as the reference's CUDA C++ does.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "awe_internal.h"
#include "plan_impl.h"

namespace awe {

#define CUDA_TRY(expr)                                                                            \
    do {                                                                                          \
        cudaError_t e_ = (expr);                                                                  \
        if (e_ != cudaSuccess) {                                                                  \
            set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return AWE_ERR_CUDA;                                                                  \
        }                                                                                         \
    } while (0)
#define AWE_TRY(expr)                \
    do {                             \
        awe_status s_ = (expr);      \
        if (s_ != AWE_OK) return s_; \
    } while (0)

constexpr int kNopA = 4;  // cart_kernels.cu:401, spher_kernels.cu:402

template <class T>
static awe_status upload_t(awe_plan *p, T **dst, const T *src, size_t n) {
    if (!*dst) AWE_TRY(dev_alloc(p, (void **)dst, n * sizeof(T)));
    CUDA_TRY(cudaMemcpy(*dst, src, n * sizeof(T), cudaMemcpyHostToDevice));
    return AWE_OK;
}

static int floor_first(float o, float opad, float d, float eps) { return (int)(std::floor)((o - opad) / d + eps); }

// the two levels and the velocity
static awe_status alloc_levels(awe_plan *p) {
    for (float **q : {&p->u[0], &p->u[1], &p->vel})
        AWE_TRY(dev_alloc(p, (void **)q, (size_t)p->g.cells() * sizeof(float)));
    return AWE_OK;
}

awe_status planA_init(awe_plan *p) {
    awe_desc &d = p->d;
    p->ndim = d.ndim;
    p->nop = 1;
    const bool spher = d.coords == AWE_SPHER;
    const int geom = spher ? (d.ndim == 2 ? 2 : 3) : (d.ndim == 2 ? 0 : 1);
    const int nb = d.nb < kNopA ? kNopA : d.nb;  // MAWEFDcart2Dgpu.cu:144
    p->nbd = nb;
    p->g = Grid{d.n[0] + 2 * nb, d.n[1] + 2 * nb, d.ndim == 3 ? d.n[2] + 2 * nb : 1};
    const Grid &g = p->g;
    if (g.n1 < 12 || g.n2 < 12 || (d.ndim == 3 && g.n3 < 12)) {
        set_error("the GPU-program scheme needs at least 12 padded samples per axis");
        return AWE_ERR_UNSUPPORTED;
    }
    if (geom == 1 && d.n[0] != d.n[1]) {
        // sfAWEFDcart3Dgpu indexes the velocity and its one-way tables as if
        // nx == nz (cart_kernels.cu:456, MAWEFDcart3Dgpu.cu:271-294)
        set_error("the cartesian 3D GPU program is defined only for nx == nz (got nz=%d nx=%d)", d.n[0], d.n[1]);
        return AWE_ERR_UNSUPPORTED;
    }
    // TMA-staged spherical step for AWE_FAST; AWE_STEP_KERNEL=simple keeps the
    // register-march kernel (the tests compare both).  Lines of its levels
    // start on 16-byte boundaries: n1 % 4 != 0 takes padded ones from 2^17
    // cells on.  (A step of 185 x 122 x 122 ragged cells: 25 us against 33;
    // below, launches bound both, 19 us against 25, and the plan stays with
    // the kernels that step_kernel has always reported for such grids.)
    const char *kern = std::getenv("AWE_STEP_KERNEL");
    bool sph_tma = geom == 3 && d.precision == AWE_FAST && !(kern && std::strcmp(kern, "simple") == 0);
    if (sph_tma) {
        const Grid pitched(p->g.n1, p->g.n2, p->g.n3, (p->g.n1 + 3) / 4 * 4);
        sph_tma = sphA_tma_eligible(pitched, nb) && (p->g.n1 % 4 == 0 || pitched.cells() >= 1 << 17);
        // the register kernels take plain lines only: padded ones once their
        // levels are allocated and the tensor maps encoded
        if (sph_tma) {
            const Grid plain = p->g;
            p->g = pitched;
            sph_tma = alloc_levels(p) == AWE_OK && sphA_tma_maps(p->sph_maps, p->u, p->vel, p->g, 1);
            if (!sph_tma) {
                for (float **q : {&p->u[0], &p->u[1], &p->vel}) {
                    dev_free(p, *q);
                    *q = nullptr;
                }
                p->g = plain;
            }
        }
    }
    if (!sph_tma) AWE_TRY(alloc_levels(p));
    for (int a = 0; a < d.ndim; a++) p->opad[a] = d.o[a] - nb * d.d[a];

    StepAParams &pa = p->pa;
    pa = StepAParams{};
    pa.g = g;
    pa.geom = geom;
    pa.nd = d.ndim;
    pa.nb = nb;
    pa.dt2 = d.dt * d.dt;
    const int round1 = 8 * ((g.n1 + 7) / 8), round2 = 8 * ((g.n2 + 7) / 8);
    switch (geom) {
        case 0:  // cart 2D: kernel axes (x, z) = memory (2, 1)
            pa.pri[0] = 1, pa.pri[1] = 0;
            pa.mask = 1;  // freeSurf_2D unconditional (MAWEFDcart2Dgpu.cu:424)
            pa.spill = round2 - g.n2;
            pa.dd1 = d.d[0] * d.d[0];
            pa.dd2 = d.d[1] * d.d[1];
            break;
        case 1:  // cart 3D: kernel axes (x, y, z) = memory (2, 3, 1)
            pa.pri[0] = 1, pa.pri[1] = 2, pa.pri[2] = 0;
            pa.mask = 2;  // freeSurf_3D unconditional before the boundary (MAWEFDcart3Dgpu.cu:417)
            pa.dd1 = d.d[0] * d.d[0];
            pa.dd2 = d.d[1] * d.d[1];
            pa.dd3 = d.d[2] * d.d[2];
            break;
        case 2:  // polar: kernel axes (r, theta) = memory (1, 2)
            pa.pri[0] = 0, pa.pri[1] = 1;
            pa.mask = d.fsrf ? 3 : 0;
            pa.spill = round1 - g.n1;
            break;
        default:  // spherical: kernel axes (r, phi, theta) = memory (1, 3, 2)
            pa.pri[0] = 0, pa.pri[1] = 2, pa.pri[2] = 1;
            pa.mask = d.fsrf ? 3 : 0;
            pa.spill = round1 - g.n1;
            break;
    }
    (void)round1;

    // sponge factor by index, spongeKernel_2D/3D: exp(-|(i-1)^2 log(alpha)| / nb^2),
    // log of the float alpha in float (the C++ overload), the rest in double
    std::vector<double> dtab(nb + 1, 1.0);
    std::vector<float> ftab(nb + 1, 1.f);
    const float alpha = 0.90;
    for (int i = 1; i <= nb; i++) {
        dtab[i] = std::exp(-1.0 * std::fabs((std::pow((i - 1.0), 2) * (double)std::log(alpha)) / (std::pow(nb, 2))));
        ftab[i] = (float)dtab[i];
    }
    double *d_dtab = nullptr;
    float *d_ftab = nullptr;
    AWE_TRY(upload_t(p, &d_dtab, dtab.data(), dtab.size()));
    AWE_TRY(upload_t(p, &d_ftab, ftab.data(), ftab.size()));
    pa.dtab = d_dtab;
    pa.ftab = d_ftab;

    // metric tables, evaluated as the kernels do per cell (spher_kernels.cu:404-526)
    if (geom == 2) {
        const float dra = d.d[0], dth = d.d[1], ora = p->opad[0];
        std::vector<float> am(g.n1), ap(g.n1), b(g.n1), b0(g.n1);
        for (int ira = 0; ira < g.n1; ira++) {
            const float ra = dra * ira + ora;
            am[ira] = (1 / (dra * dra)) + (1 / (2 * ra * dra));
            ap[ira] = (1 / (dra * dra)) - (1 / (2 * ra * dra));
            b[ira] = (1 / (ra * ra * dth * dth));
            b0[ira] = (-2 / (ra * ra * dth * dth));
        }
        pa.a0 = (-2 / (dra * dra));
        float *t0 = nullptr, *t1 = nullptr, *t2 = nullptr, *t3 = nullptr;
        AWE_TRY(upload_t(p, &t0, am.data(), am.size()));
        AWE_TRY(upload_t(p, &t1, ap.data(), ap.size()));
        AWE_TRY(upload_t(p, &t2, b.data(), b.size()));
        AWE_TRY(upload_t(p, &t3, b0.data(), b0.size()));
        pa.tr0 = t0, pa.tr1 = t1, pa.tr2 = t2, pa.tr3 = t3;
    } else if (geom == 3) {
        const float dra = d.d[0], dth = d.d[1], dph = d.d[2], ora = p->opad[0], oth = p->opad[1];
        pa.dd1 = 2 * dra;
        pa.dd2 = dra * dra;
        pa.dd3 = 2 * dth;
        pa.dd4 = dth * dth;
        pa.dd5 = dph * dph;
        std::vector<float> a2(g.p1), cr(g.p1), B((size_t)g.p1 * g.n2), D((size_t)g.p1 * g.n2);
        for (int ira = 0; ira < g.n1; ira++) {
            const float ra = dra * ira + ora;
            a2[ira] = (2 / ra);
            cr[ira] = (1 / (ra * ra));
            for (int ith = 0; ith < g.n2; ith++) {
                const float th = dth * ith + oth;
                B[(size_t)ith * g.p1 + ira] = (std::cos(th) / (ra * ra * std::sin(th)));
                D[(size_t)ith * g.p1 + ira] = (1 / (ra * ra * std::sin(th) * std::sin(th)));
            }
        }
        float *t0 = nullptr, *t1 = nullptr, *u0 = nullptr, *u1 = nullptr;
        AWE_TRY(upload_t(p, &t0, a2.data(), a2.size()));
        AWE_TRY(upload_t(p, &t1, cr.data(), cr.size()));
        AWE_TRY(upload_t(p, &u0, B.data(), B.size()));
        AWE_TRY(upload_t(p, &u1, D.data(), D.size()));
        pa.tr0 = t0, pa.tr1 = t1, pa.tt0 = u0, pa.tt1 = u1;
    }

    const size_t cells = (size_t)g.cells();
    AWE_TRY(dev_alloc(p, (void **)&p->corner_off, 8 * sizeof(long long)));
    if (geom != 3) AWE_TRY(dev_alloc(p, (void **)&p->u3, cells * sizeof(float)));

    pa.nshot = 1;
    pa.shot_cells = g.cells();
    cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, p->device);
    if (p->num_sms < 1) p->num_sms = 1;
    pa.sms = p->num_sms;
    // (the TMA kernels' sponge index walks the axes in the spherical grid's
    // priority order (r, phi, theta) = memory axes (1, 3, 2), pa.pri above)
    if (sph_tma) {
        AWE_TRY(dev_alloc(p, (void **)&p->sched_counter, sizeof(unsigned long long)));
        AWE_TRY(dev_alloc(p, (void **)&p->d_err, sizeof(int)));
        CUDA_TRY(cudaMemset(p->sched_counter, 0, sizeof(unsigned long long)));
        CUDA_TRY(cudaMemset(p->d_err, 0, sizeof(int)));
        const char *spin = std::getenv("AWE_PIPELINE_SPIN_LIMIT");
        if (spin && *spin) p->spin_limit = std::atoll(spin);
        p->sph_tma = true;
    }
    // reciprocals of the Laplacian divisors (AWE_FAST multiplies; AWE_EXACT divides as the reference)
    const float dvs[5] = {pa.dd1, pa.dd2, pa.dd3, pa.dd4, pa.dd5};
    for (int j = 0; j < 5; j++) pa.rd[j] = dvs[j] != 0.f ? 1.f / dvs[j] : 0.f;

    // outputs: rows and snapshot windows as each program writes them
    const int jdata = d.jdata > 0 ? d.jdata : 1;
    p->nsmp = geom == 3 ? d.nt : d.nt / jdata;
    if (p->nsmp < 1) p->nsmp = 1;
    p->nsnap = d.jsnap > 0 ? (d.nt - 1) / d.jsnap + 1 : 0;
    const int npads[3] = {g.n1, g.n2, g.n3};
    for (int a = 0; a < 3; a++) {
        if (a >= d.ndim) {
            p->snap_f[a] = 0;
            p->snap_m[a] = 1;
        } else if (d.bnds) {
            p->snap_f[a] = 0;
            p->snap_m[a] = npads[a];
        } else {
            p->snap_m[a] = d.n[a];
            if (geom == 3) p->snap_f[a] = nb;                                                 // cut3d_sph
            else if (geom == 1) p->snap_f[a] = floor_first(d.o[a], p->opad[a], d.d[a], 0.0001f);  // cut3d
            else p->snap_f[a] = floor_first(d.o[a], p->opad[a], d.d[a], 0.f);                 // cut2d
        }
    }
    p->snap_transpose = geom == 2;
    p->snap_elems = (size_t)p->snap_m[0] * p->snap_m[1] * p->snap_m[2];
    return AWE_OK;
}

awe_status planA_model(awe_plan *p, const float *vel, const float *rfl) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    StepAParams &pa = p->pa;
    const size_t lines = (size_t)g.n2 * g.n3, cells = lines * g.n1;
    const int nb = p->nbd;
    p->inj_scale_ok = false;
    p->h_vel_raw.assign(cells, 0.f);
    expand_model(d.ndim, vel, p->h_vel_raw.data(), nb, d.n);
    CUDA_TRY(cudaDeviceSynchronize());  // earlier runs (on any stream) may still read the old model
    CUDA_TRY(cudaMemcpy2D(p->vel, g.p1 * sizeof(float), p->h_vel_raw.data(), g.n1 * sizeof(float),
                          g.n1 * sizeof(float), lines, cudaMemcpyHostToDevice));
    const std::vector<float> &v = p->h_vel_raw;
    const float dt = d.dt;
    auto coef = [](float q) { return (1 - q) / (1 + q); };
    if (pa.geom == 0) {
        // MAWEFDcart2Dgpu.cu:280-285: h_vel indexed x-fastest; only the last
        // x sample survives the boundary kernel's loop
        const int nxpad = g.n2, nzpad = g.n1;
        pa.b2lo = coef(v[(size_t)kNopA * nxpad + nxpad - 1] * (dt / d.d[0]));
        pa.b2hi = coef(v[(size_t)(nzpad - kNopA - 1) * nxpad + nxpad - 1] * (dt / d.d[0]));
        if (d.refl) {
            if (!rfl) {
                set_error("refl=y needs a reflectivity image");
                return AWE_ERR_INVALID;
            }
            p->h_rfl_pad.assign(cells, 0.f);
            expand_model(2, rfl, p->h_rfl_pad.data(), nb, d.n);
        }
    } else if (pa.geom == 2) {
        const int nrapad = g.n1, nthpad = g.n2;
        pa.b2lo = coef(v[(size_t)kNopA * nrapad + nrapad - 1] * (dt / d.d[1]));
        pa.b2hi = coef(v[(size_t)(nthpad - kNopA - 1) * nrapad + nrapad - 1] * (dt / d.d[1]));
    } else if (pa.geom == 1) {
        // MAWEFDcart3Dgpu.cu:271-294 with its flat indices (the y-high table
        // filled as the loop intends; the reference writes only its diagonal)
        const size_t nxpad = g.n2, nypad = g.n3, nzpad = g.n1, n2 = nxpad * nzpad;
        std::vector<float> bzl(nxpad * nypad), bzh(nxpad * nypad), bxl(nzpad * nypad), bxh(nzpad * nypad),
            byl(nxpad * nzpad), byh(nxpad * nzpad);
        for (size_t ix = 0; ix < nxpad; ix++)
            for (size_t iy = 0; iy < nypad; iy++) {
                bzl[iy * nxpad + ix] = coef(v[iy * n2 + kNopA * nxpad + ix] * (dt / d.d[0]));
                bzh[iy * nxpad + ix] = coef(v[iy * n2 + (nzpad - kNopA - 1) * nxpad + ix] * (dt / d.d[0]));
            }
        for (size_t iz = 0; iz < nzpad; iz++)
            for (size_t iy = 0; iy < nypad; iy++) {
                bxl[iy * nzpad + iz] = coef(v[iy * n2 + iz * nxpad + kNopA] * (dt / d.d[1]));
                bxh[iy * nzpad + iz] = coef(v[iy * n2 + iz * nxpad + nxpad - kNopA - 1] * (dt / d.d[1]));
            }
        for (size_t iz = 0; iz < nzpad; iz++)
            for (size_t ix = 0; ix < nxpad; ix++) {
                byl[iz * nxpad + ix] = coef(v[kNopA * n2 + iz * nxpad + ix] * (dt / d.d[2]));
                byh[iz * nxpad + ix] = coef(v[(nypad - kNopA - 1) * n2 + iz * nxpad + ix] * (dt / d.d[2]));
            }
        float *t[6];  // (kept from model to model)
        for (int k = 0; k < 6; k++) t[k] = const_cast<float *>(pa.tb[k]);
        AWE_TRY(upload_t(p, &t[0], bzl.data(), bzl.size()));
        AWE_TRY(upload_t(p, &t[1], bzh.data(), bzh.size()));
        AWE_TRY(upload_t(p, &t[2], bxl.data(), bxl.size()));
        AWE_TRY(upload_t(p, &t[3], bxh.data(), bxh.size()));
        AWE_TRY(upload_t(p, &t[4], byl.data(), byl.size()));
        AWE_TRY(upload_t(p, &t[5], byh.data(), byh.size()));
        for (int k = 0; k < 6; k++) pa.tb[k] = t[k];
    }
    return AWE_OK;
}

// reflectivity of inject_sources_{2D,3D}: first neighbour (kernel order, its
// own flat indexing) whose velocity differs; neighbours outside the array
// (where the reference reads out of bounds) count as equal
static float refl_scale(const std::vector<float> &v, long long s, long long rs, long long ps, int nd) {
    static const int o2[7][2] = {{1, 0}, {0, 1}, {1, 1}, {0, -1}, {-1, -1}, {1, -1}, {-1, 1}};
    static const int o3[26][3] = {{0, 1, 0},   {1, 0, 0},   {0, 0, 1},   {0, -1, 0},  {-1, 0, 0},  {0, 0, -1},
                                  {0, 1, 1},   {0, -1, -1}, {0, 1, -1},  {0, -1, 1},  {1, 1, 0},   {-1, -1, 0},
                                  {1, -1, 0},  {-1, 1, 0},  {1, 0, 1},   {-1, 0, -1}, {1, 0, -1},  {-1, 0, 1},
                                  {1, 0, -1},  {1, 1, 1},   {1, 1, -1},  {1, -1, 1},  {1, -1, -1}, {-1, 1, 1},
                                  {-1, 1, -1}, {-1, -1, 1}};
    const long long n = (long long)v.size();
    if (s < 0 || s >= n) return 0.f;
    const float v0 = v[s];
    const int cnt = nd == 2 ? 7 : 26;
    for (int k = 0; k < cnt; k++) {
        const long long t = nd == 2 ? s + o2[k][0] * rs + o2[k][1] : s + o3[k][0] * ps + o3[k][1] * rs + o3[k][2];
        if (t < 0 || t >= n) continue;
        if (v0 != v[t]) return std::fabs((v0 - v[t]) / (v0 + v[t]));
    }
    return 0.f;
}

awe_status planA_prepare(awe_plan *p) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const int geom = p->pa.geom, ns = p->ns;
    // few source corners are added by the step itself (2D: none on the line the
    // one-way boundary reads)
    static_assert(4 * kFusedSources <= kFusedCorners && 8 * kFusedSources <= kFusedCorners3, "fused corners");
    p->inj_fused = geom != 3 && p->move_mode < 0 && (int)p->h_src.size() <= kFusedSources;
    for (const GeoPoint &pt : p->h_src)
        for (int c = 0; d.ndim == 2 && p->inj_fused && c < 4; c++) {
            const long long n = pt.base + p->h_corner_off[c];
            if (geom == 0 ? n / g.n1 >= g.n2 - 1 : n % g.n1 >= g.n1 - 1) p->inj_fused = false;
        }
    if (d.expl == 0 || ns == 0 || p->inj_scale_ok) return AWE_OK;
    std::vector<float> sc((size_t)ns * 8, 1.f);
    for (int s = 0; s < ns; s++) {
        const Lint &l = p->h_src_lint[s];
        if (geom == 0 && d.refl) {  // inject_sources_2D_refl: rfl with the x-fastest flat index
            const long long nx = g.n2;
            const long long f[4] = {(long long)l.jz * nx + l.jx, (long long)(l.jz + 1) * nx + l.jx,
                                    (long long)l.jz * nx + l.jx + 1, (long long)(l.jz + 1) * nx + l.jx + 1};
            for (int c = 0; c < 4; c++) sc[s * 8 + c] = p->h_rfl_pad[f[c]];
            continue;
        }
        float r = 0.f;
        if (geom == 0) r = refl_scale(p->h_vel_raw, (long long)l.jz * g.n2 + l.jx, g.n2, 0, 2);
        else if (geom == 1)
            r = refl_scale(p->h_vel_raw, (long long)l.jy * g.n2 * g.n1 + (long long)l.jz * g.n2 + l.jx, g.n2,
                           (long long)g.n2 * g.n1, 3);
        else if (geom == 2) r = refl_scale(p->h_vel_raw, (long long)l.jz * g.n1 + l.jx, g.n1, 0, 2);
        else
            r = refl_scale(p->h_vel_raw, (long long)l.jy * g.n1 * g.n2 + (long long)l.jz * g.n1 + l.jx, g.n1,
                           (long long)g.n1 * g.n2, 3);
        for (int c = 0; c < 8; c++) sc[s * 8 + c] = r;
    }
    if (p->inj_scale) dev_free(p, p->inj_scale);
    p->inj_scale = nullptr;
    AWE_TRY(upload_t(p, &p->inj_scale, sc.data(), sc.size()));
    p->inj_scale_ok = true;
    return AWE_OK;
}

// Cartesian and polar: one launch a step (k_stepA2d.cu, k_stepA3d.cu).  Sources
// the step adds itself leave the levels without their injection, so the traces
// of step it - 1 come from the level step it reads; otherwise the injection and
// the gather keep their own launches around the step.
template <class Fused>
static awe_status run_fused(awe_plan *p, const float *d_wav, int ncs, float *d_dat, float *d_wfl, cudaStream_t s) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const StepAParams &pa = p->pa;
    const bool exact = d.precision == AWE_EXACT, scaled = d.expl != 0;
    const int nc = d.ndim == 3 ? 8 : 4;
    long long launches = 0;
    float *prv = p->u[0], *cur = p->u[1], *nxt = p->u3;
    Fused f{};
    if (p->inj_fused)
        for (size_t k = 0; k < p->h_src.size(); k++)
            for (int c = 0; c < nc; c++) {
                const long long n = p->h_src[k].base + p->h_corner_off[c];
                f.inj_i1[f.inj_n] = (int)(n % g.n1);
                f.inj_i2[f.inj_n] = (int)(n / g.n1 % g.n2);
                if constexpr (std::is_same<Fused, StepA3Fused>::value)
                    f.inj_i3[f.inj_n] = (int)(n / g.n1 / g.n2);
                f.inj_src[f.inj_n] = 8 * (int)k + c;
                f.inj_w[f.inj_n++] = p->h_src[k].w[c];
            }
    f.scale = p->inj_scale;
    f.scaled = scaled;
    f.wav = d_wav;
    f.ncs = ncs;
    // the trace row of step it, or -1 (cartesian 3D: MAWEFDcart3Dgpu.cu:432-442, pre-incremented)
    auto row_of = [&](int it) {
        const int r = d.ndim == 2 ? it : it % d.jdata == 0 ? it / d.jdata + 1 : -1;
        return p->nr > 0 && r < p->nsmp ? r : -1;
    };
    int isnap = 0;
    for (int it = 0; it < d.nt; it++) {
        f.it = it;
        f.nr = 0;
        const bool inj = !p->inj_fused && p->ns > 0;
        const bool own = inj || p->move_mode >= 0;  // the traces keep their own launch
        if (inj) {
            const PointsAt ps = points_at(p, p->src, p->ns, p->src_rows, it);
            if (p->inj.n > 0)
                launch_injectA_cells(exact, cur, p->inj_scale, p->inj, d_wav, it, scaled, s, ncs);
            else
                launch_injectA(exact, d.ndim, cur, ps.pts, p->inj_scale, p->ns, d_wav, it, scaled, p->corner_off, s,
                               ps.stride, ncs);
            launches++;
        }
        if (!own && it > 0 && row_of(it - 1) >= 0) {
            f.rec = p->rec;
            f.nr = p->nr;
            f.rec_row = d_dat + (size_t)row_of(it - 1) * p->nr;
        }
        prof_begin(p, s);
        if constexpr (std::is_same<Fused, StepA3Fused>::value)
            launch_stepA3(exact, cur, prv, nxt, p->vel, pa, f, s);
        else
            launch_stepA2(pa.geom, exact, cur, prv, nxt, p->vel, pa, f, s);
        prof_end(p, s);
        launches++;
        float *t = prv;
        prv = cur;
        cur = nxt;
        nxt = t;
        if (row_of(it) >= 0 && (own || it == d.nt - 1)) {
            const PointsAt pr = points_at(p, p->rec, p->nr, p->rec_rows, it);
            launch_extract_off(d.ndim, exact, cur, pr.pts, p->nr, d_dat + (size_t)row_of(it) * p->nr, nullptr, nullptr,
                               nullptr, g, p->corner_off, s, pr.stride);
            launches++;
        }
        if (p->nsnap > 0 && it % d.jsnap == 0) {
            float *frame = d_wfl ? d_wfl + (size_t)isnap * p->snap_elems : p->d_snap_tmp;
            if (frame) {
                if (p->snap_transpose)
                    launch_snapshot_transpose2(cur, frame, g, p->snap_f[0], p->snap_f[1], p->snap_m[0], p->snap_m[1],
                                               s);
                else
                    launch_snapshot(d.ndim, cur, frame, g, p->snap_f[0], p->snap_f[1], p->snap_f[2], p->snap_m[0],
                                    p->snap_m[1], p->snap_m[2], nullptr, nullptr, nullptr, s);
                launches++;
                AWE_TRY(deliver_snapshot(p, frame, isnap, it, s));
            }
            isnap++;
        }
    }
    p->launches = launches;
    return flush_snapshots(p);
}

// hook (may be null): called at the start of every iteration, before the
// injection, with prev = the previous level (sponge pending) and cur = the
// current level
awe_status planA_run(awe_plan *p, const float *d_wav, int ncs, float *d_dat, float *d_wfl, cudaStream_t s,
                     const StepHook *hook) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const StepAParams &pa = p->pa;
    const bool exact = d.precision == AWE_EXACT;
    const size_t bytes = (size_t)g.cells() * sizeof(float) * (pa.nshot > 0 ? pa.nshot : 1);
    const bool scaled = d.expl != 0;
    AWE_TRY(planA_prepare(p));
    CUDA_TRY(cudaMemsetAsync(p->u[0], 0, bytes, s));
    CUDA_TRY(cudaMemsetAsync(p->u[1], 0, bytes, s));
    CUDA_TRY(cudaMemsetAsync(d_dat, 0, (size_t)p->nsmp * p->nr * sizeof(float), s));
    if (p->nsnap > 0 && !d_wfl && p->snap_cb && !p->d_snap_tmp)
        AWE_TRY(dev_alloc(p, (void **)&p->d_snap_tmp, p->snap_elems * sizeof(float)));
    p->snap_pending = -1;  // a frame left queued by a failed run is not delivered
    if (d.ndim == 2) return run_fused<StepA2Fused>(p, d_wav, ncs, d_dat, d_wfl, s);
    if (pa.geom == 1) return run_fused<StepA3Fused>(p, d_wav, ncs, d_dat, d_wfl, s);

    if (p->sph_tma) {  // maps of this run's level fields; the work counter restarts with every run
        if (!sphA_tma_maps(p->sph_maps, p->u, p->vel, g, pa.nshot)) {
            set_error("tensor-map encoding of the spherical step failed");
            return AWE_ERR_CUDA;
        }
        const char *lenv = std::getenv("AWE_TMA_CHUNK");
        p->sph_shape = sphA_tma_shape(g, pa.nshot, p->num_sms, lenv ? std::atoi(lenv) : 0);
        CUDA_TRY(cudaMemsetAsync(p->sched_counter, 0, sizeof(unsigned long long), s));
        p->sched_base = 0;
    }
    long long launches = 0;
    float *cur = p->u[1], *nxt = p->u[0];
    int isnap = 0;
    for (int it = 0; it < d.nt; it++) {
        if (hook) AWE_TRY((*hook)(it, nxt, cur, s));
        if (p->ns > 0) {
            const PointsAt ps = points_at(p, p->src, p->ns, p->src_rows, it);
            if (p->move_mode < 0 && p->inj.n > 0)
                launch_injectA_cells(exact, cur, p->inj_scale, p->inj, d_wav, it, scaled, s, ncs);
            else
                launch_injectA(exact, d.ndim, cur, ps.pts, p->inj_scale, p->ns, d_wav, it, scaled, p->corner_off, s,
                               ps.stride, ncs);
            launches++;
        }
        prof_begin(p, s);
        if (p->sph_tma) {
            const int ic = cur == p->u[0] ? 0 : 1;  // nxt is the other level
            const cudaError_t e =
                launch_stepA_sph_tma(p->sph_maps[ic], p->sph_maps[2 + (1 - ic)], p->sph_maps[4], nxt, pa,
                                     p->sph_shape, p->sched_counter, p->sched_base, p->d_err, p->spin_limit, s);
            p->sched_base += (unsigned long long)p->sph_shape.items + p->sph_shape.grid;
            if (e != cudaSuccess) {
                set_error("spherical TMA step launch failed: %s", cudaGetErrorString(e));
                return AWE_ERR_CUDA;
            }
        } else {
            launch_stepA(exact, cur, nxt, p->vel, pa, s);
        }
        prof_end(p, s);
        launches++;
        std::swap(cur, nxt);  // cur: the new level (final); nxt: previous (sponge pending)
        if (p->nr > 0) {
            const PointsAt pr = points_at(p, p->rec, p->nr, p->rec_rows, it);
            launch_extract_off(d.ndim, exact, cur, pr.pts, p->nr, d_dat + (size_t)it * p->nr, nullptr, nullptr, nullptr,
                               g, p->corner_off, s, pr.stride);
            launches++;
        }
        if (p->nsnap > 0 && it % d.jsnap == 0) {
            float *frame = d_wfl ? d_wfl + (size_t)isnap * p->snap_elems : p->d_snap_tmp;
            if (frame) {
                launch_snapshot(d.ndim, cur, frame, g, p->snap_f[0], p->snap_f[1], p->snap_f[2], p->snap_m[0],
                                p->snap_m[1], p->snap_m[2], nullptr, nullptr, nullptr, s);
                launches++;
                AWE_TRY(deliver_snapshot(p, frame, isnap, it, s));
            }
            isnap++;
        }
    }
    p->launches = launches;
    return flush_snapshots(p);
}

}  // namespace awe
