// Host side of the CPU-program scheme (MAWEFDcart{2D,3D}cpu.c): padding,
// coefficient tables, model preparation and the per-step launch sequence.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
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
#define AWE_TRY(expr)                      \
    do {                                   \
        awe_status s_ = (expr);            \
        if (s_ != AWE_OK) return s_;       \
    } while (0)

// cut2d / cut3d_slice first index (fdutil.c:574-717): floor((o - opad)/d) in float
static int window_first(float o, float opad, float d) { return (int)(std::floor)((o - opad) / d); }

static awe_status upload(awe_plan *p, float **dst, const float *src, size_t n) {
    if (!*dst) AWE_TRY(dev_alloc(p, (void **)dst, n * sizeof(float)));
    CUDA_TRY(cudaMemcpy(*dst, src, n * sizeof(float), cudaMemcpyHostToDevice));
    return AWE_OK;
}

// Tile, steps per launch and columns per thread of k_tb2d.cu.  A launch costs
// about 1.5 us besides its steps, a step 0.35 us (barrier, load and arithmetic
// latency of a few warps) and 0.15 ns per cell of the region; a tile occupies
// an SM (512 threads of 4 x cx cells).  Fitted to 141 x 183 (4th order) to 1480
// x 1480 (8th order) cells, where the best of 17 shapes took 0.79 to 8.6 us a
// step and the one-step kernel 2.45 to 16.4.
static Tb2Shape tb2_shape(const Grid &g, int nop, int sms) {
    Tb2Shape best{};
    double cost = 1e30;
    for (int tz0 = 8; tz0 <= 104; tz0 += 4)
        for (int tx0 = 8; tx0 <= 104; tx0 += 4)
            for (int k = 1; k <= 12; k++) {
                Tb2Shape s{};
                s.k = k;
                s.ntz = (g.n1 + tz0 - 1) / tz0;
                s.ntx = (g.n2 + tx0 - 1) / tx0;
                s.tz = ((g.n1 + s.ntz - 1) / s.ntz + 3) / 4 * 4;  // even tiles
                s.tx = (g.n2 + s.ntx - 1) / s.ntx;
                s.hx = nop * k;
                s.hz = (s.hx + 3) / 4 * 4;
                s.rz = s.tz + 2 * s.hz;
                s.rx = (s.tx + 2 * s.hx + 3) / 4 * 4;
                for (s.cx = 1; s.cx <= 4 && (s.rz / 4) * (s.rx / s.cx) > kTb2Threads;) s.cx *= 2;
                if (s.cx > 4) break;
                const long long rounds = ((long long)s.ntz * s.ntx + sms - 1) / sms;
                const double c = rounds * (1.5 / k + 0.35 + 1.5e-4 * s.rz * s.rx);
                if (c < cost) {
                    cost = c;
                    best = s;
                }
            }
    best.ntz = (g.n1 + best.tz - 1) / best.tz;
    best.ntx = (g.n2 + best.tx - 1) / best.tx;
    return best;
}

// two level buffers with their padding columns, the longest lists of a tile, a word per thread
size_t tb2_smem(const Tb2Shape &sh, const int *most) {
    return (size_t)2 * (sh.rx + 8) * sh.rz * 4 + (size_t)most[0] * 40 + (size_t)most[1] * 16 + kTb2Threads * 4 +
           (size_t)most[2] * 4 * (1 + sh.k);
}

bool tb2_host_lists(const Tb2Shape &sh, const std::vector<Tb2Grid> &grids, int ntile, Tb2HostLists &out) {
    struct Cell {
        int tile, owner;  // owner: the thread that holds the cell
        int4 q;
    };
    std::vector<Cell> rc, cell;
    std::vector<const float *> rw;  // weights of the receivers in rc's first order
    std::vector<int2> ea;           // entries of the grids' cells, in (point, corner) order per cell
    size_t ns = 0;
    for (const Tb2Grid &g : grids) {
        // receivers by the tile of their base cell (all four corners are in its region)
        for (int r = 0; r < g.nrec; r++) {
            const int z = (int)(g.rec[r].base % g.n1), x = (int)(g.rec[r].base / g.n1);
            if (z >= g.n1 - 1 || x >= g.n2 - 1) return false;
            rc.push_back({g.tile0 + (x / sh.tx) * sh.ntz + z / sh.tz, (int)rw.size(), make_int4(z, x, r, 0)});
            rw.push_back(g.rec[r].w);
        }
        // cells that points inject into, each with its entries, in every tile whose region holds the cell
        ns += g.ninj;
        std::vector<std::pair<long long, int>> e;
        for (int s = 0; s < g.ninj; s++)
            for (int c = 0; c < 4; c++) {
                const long long n = g.inj[s].base + (c & 1) + (c >> 1) * (long long)g.n1;
                if (n >= (long long)g.n1 * g.n2) return false;
                e.push_back({n, 8 * s + c});
            }
        std::sort(e.begin(), e.end());
        const int ea0 = (int)ea.size();
        for (const auto &v : e) {
            int w;
            std::memcpy(&w, &g.inj[v.second >> 3].w[v.second & 7], sizeof w);
            ea.push_back(make_int2(v.second, w));
        }
        for (size_t k = 0, k1; k < e.size(); k = k1) {
            for (k1 = k; k1 < e.size() && e[k1].first == e[k].first;) k1++;
            const int z = (int)(e[k].first % g.n1), x = (int)(e[k].first / g.n1);
            for (int bx = std::max(0, (x - sh.hx) / sh.tx - 1); bx < g.ntx && bx * sh.tx - sh.hx <= x; bx++)
                for (int bz = std::max(0, (z - sh.hz) / sh.tz - 1); bz < sh.ntz && bz * sh.tz - sh.hz <= z; bz++) {
                    const int lx = x - bx * sh.tx + sh.hx, lz = z - bz * sh.tz + sh.hz;
                    if (lx < sh.rx && lz < sh.rz)
                        cell.push_back({g.tile0 + bx * sh.ntz + bz, lx / sh.cx * (sh.rz / 4) + lz / 4,
                                        make_int4(z, x, ea0 + (int)k, ea0 + (int)k1)});
                }
        }
    }
    auto order = [](const Cell &a, const Cell &b) { return a.tile != b.tile ? a.tile < b.tile : a.owner < b.owner; };
    std::stable_sort(rc.begin(), rc.end(), order);
    std::stable_sort(cell.begin(), cell.end(), order);
    std::vector<int> start[3];  // cells, entries, receivers
    for (auto &v : start) v.assign(ntile + 1, 0);
    std::vector<int2> ent;
    for (Cell &c : cell) {
        const int k0 = c.q.z, k1 = c.q.w;
        c.q.z = (int)ent.size();
        ent.insert(ent.end(), ea.begin() + k0, ea.begin() + k1);
        c.q.w = (int)ent.size();
        start[0][c.tile + 1]++;
        start[1][c.tile + 1] += k1 - k0;
    }
    for (const Cell &c : rc) start[2][c.tile + 1]++;
    int most[3] = {0, 0, 0};
    for (int k = 0; k < 3; k++)
        for (int q = 0; q < ntile; q++) {
            most[k] = std::max(most[k], start[k][q + 1]);
            start[k][q + 1] += start[k][q];
        }
    out.most[0] = most[2];
    out.most[1] = most[0];
    out.most[2] = most[1];
    if (most[0] >= 32768 || tb2_smem(sh, out.most) > kTb2SmemMax) return false;  // one tile's points do not fit
    // one buffer; sized for injected corners in four tiles each, so that points
    // that only move keep it (a captured time loop reads it)
    const size_t nst = (size_t)(ntile + 4) / 4 * 4 + 4, nr = rc.size();
    const size_t ncell = std::max(cell.size(), 16 * ns), nent = std::max(ent.size() + 1, 16 * ns + 1) / 2 * 2;
    size_t *off = out.off;
    off[0] = 0;
    off[1] = off[0] + nst;
    off[2] = off[1] + nst;
    off[3] = off[2] + nst;          // inj_cell
    off[4] = off[3] + 4 * ncell;    // rec_pt
    off[5] = off[4] + 4 * nr;       // inj_ent
    off[6] = off[5] + 2 * nent;     // rec_wt
    std::vector<int> &buf = out.buf;
    buf.assign(off[6] + 4 * nr, 0);
    for (int k = 0; k < 3; k++) std::copy(start[k].begin(), start[k].end(), buf.begin() + off[k]);
    for (size_t k = 0; k < cell.size(); k++) std::memcpy(&buf[off[3] + 4 * k], &cell[k].q, sizeof(int4));
    if (!ent.empty()) std::memcpy(&buf[off[5]], ent.data(), ent.size() * sizeof(int2));
    for (size_t k = 0; k < rc.size(); k++) {
        std::memcpy(&buf[off[4] + 4 * k], &rc[k].q, sizeof(int4));
        std::memcpy(&buf[off[6] + 4 * k], rw[rc[k].owner], 4 * sizeof(float));
    }
    return true;
}

awe_status set_tb2_lists(awe_plan *p, Tb2Lists &t, const std::vector<GeoPoint> &inj, const std::vector<GeoPoint> *rec) {
    t.ok = false;
    if (!p->tb2 || p->move_mode >= 0 || p->sponge_deferred) return AWE_OK;
    const Tb2Shape &sh = p->tb2_shape;
    const Tb2Grid grid{p->g.n1, p->g.n2, sh.ntx, 0, inj.data(), (int)inj.size(), rec ? rec->data() : nullptr,
                       rec ? (int)rec->size() : 0};
    Tb2HostLists h;
    if (!tb2_host_lists(sh, {grid}, sh.ntz * sh.ntx, h)) return AWE_OK;
    const size_t total = h.buf.size();
    std::copy(h.off, h.off + 7, t.off);
    std::copy(h.most, h.most + 3, t.most);
    if (t.cap < total) {
        dev_free(p, t.buf);
        t.buf = nullptr;
        t.cap = 0;
        if (dev_alloc_extra(p, (void **)&t.buf, total * sizeof(int)) != AWE_OK) return AWE_OK;
        t.cap = total;
    }
    CUDA_TRY(cudaMemcpy(t.buf, h.buf.data(), total * sizeof(int), cudaMemcpyHostToDevice));
    t.ok = true;
    return AWE_OK;
}

void tb2_set_lists(Tb2Params &q, const int *buf, const size_t *off, const int *most, bool inj, bool rec) {
    if (most[1] > 0 && inj) q.inj_start = buf + off[0];
    q.ent_start = buf + off[1];
    if (most[0] > 0 && rec) q.rec_start = buf + off[2];
    q.inj_cell = (const int4 *)(buf + off[3]);
    q.rec_pt = (const int4 *)(buf + off[4]);
    q.inj_ent = (const int2 *)(buf + off[5]);
    q.rec_wt = (const float *)(buf + off[6]);
    q.max_rec = most[0], q.max_cell = most[1], q.max_ent = most[2];
}

void tb2_launch(awe_plan *p, bool adj, const float *prv, const float *cur, float *oprv, float *ocur, float *slots,
                bool slot_level, int it, int k, const float *d_wav, int ncs, float *d_dat, cudaStream_t s) {
    const awe_desc &d = p->d;
    const Tb2Shape &sh = p->tb2_shape;
    const Tb2Lists &t = adj ? p->tb2_adj : p->tb2_fwd;
    Tb2Params q{};
    q.n1 = p->g.n1;
    q.n2 = p->g.n2;
    q.k = k;
    q.it = it;
    q.tz = sh.tz, q.tx = sh.tx, q.hz = sh.hz, q.hx = sh.hx, q.rz = sh.rz, q.rx = sh.rx;
    q.c0 = p->k.c0;
    for (int i = 0; i <= p->nop; i++) q.cz[i] = p->k.c[0][i], q.cx[i] = p->k.c[1][i];
    q.cur = cur, q.prv = prv, q.vel = p->vel, q.ocur = ocur, q.oprv = oprv;
    q.slots = slots;
    q.slot_stride = p->g.cells();
    q.slot_level = slot_level;
    if (d.dabc && !d.hybrid) q.w1 = p->w[0], q.w2 = p->w[1];
    q.ilo1 = p->wlo[0], q.ihi1 = p->whi[0], q.ilo2 = p->wlo[1], q.ihi2 = p->whi[1];
    tb2_set_lists(q, t.buf, t.off, t.most, d_wav != nullptr, d_dat != nullptr);
    q.wav = d_wav;
    q.ncs = ncs;
    q.jdata = d.jdata;
    q.nr = p->nr;
    q.dat = d_dat;
    prof_begin(p, s, adj ? AWE_PROF_ADJOINT : AWE_PROF_STEP);
    launch_tb2(p->nop, adj ? 2 : slots ? 3 : d.precision == AWE_EXACT ? 1 : 0, q, sh, tb2_smem(sh, t.most), s);
    prof_end(p, s);
}

// the one-way ABC's coefficient tables: cells of table k
static size_t abc_cells(const Grid &g, int k) {
    return k < 2 ? (size_t)g.n2 * g.n3 : k < 4 ? (size_t)g.n1 * g.n3 : (size_t)g.n1 * g.n2;
}

// the two levels, the model and its tables: all of them or none
static awe_status alloc_levels(awe_plan *p) {
    const awe_desc &d = p->d;
    std::vector<std::pair<float **, size_t>> want;
    for (float **q : {&p->u[0], &p->u[1], &p->vel}) want.push_back({q, (size_t)p->g.cells()});
    for (int k = 0; d.dabc && k < (d.ndim == 3 ? 6 : 4); k++) want.push_back({&p->abc[k], abc_cells(p->g, k)});
    awe_status st = AWE_OK;
    for (auto &w : want)
        if (st == AWE_OK) st = dev_alloc(p, (void **)w.first, w.second * sizeof(float));
    for (auto &w : want)
        if (st != AWE_OK) {
            dev_free(p, *w.first);
            *w.first = nullptr;
        }
    return st;
}

awe_status planB_init(awe_plan *p) {
    awe_desc &d = p->d;
    if (d.fdorder == 0) d.fdorder = 4;  // MAWEFDcart2Dcpu.c:126
    p->ndim = d.ndim;
    p->nop = d.fdorder / 2;
    int nb = d.nb;
    if (nb < p->nop) nb = p->nop;                              // :211
    if (d.dabc && d.hybrid && nb <= p->nop) nb = 2 * p->nop;  // :212
    p->nbd = nb;
    const int n3 = d.ndim == 3 ? d.n[2] : 1;
    p->g = Grid{d.n[0] + 2 * nb, d.n[1] + 2 * nb, d.ndim == 3 ? n3 + 2 * nb : 1};
    // AWE_STEP_KERNEL=simple forces the one-thread-per-cell kernels (the tests
    // compare both)
    const char *kern = std::getenv("AWE_STEP_KERNEL");
    const bool force_simple = kern && std::strcmp(kern, "simple") == 0;
    // lines of a 3D level on 16-byte boundaries, so that the TMA step takes any
    // n1; plain ones where memory does not hold them
    const Grid plain = p->g;
    {
        const Grid pitched(plain.n1, plain.n2, plain.n3, (plain.n1 + 3) / 4 * 4);
        // (k_stepB steps across padded lines with 32-bit offsets)
        const bool small = pitched.p1 == plain.p1 || pitched.s3() < 1LL << 29;
        if (!force_simple && small && stepB3_tma_eligible(d.ndim, p->nop, false, pitched)) p->g = pitched;
    }
    for (int a = 0; a < d.ndim; a++) p->opad[a] = d.o[a] - nb * d.d[a];  // fdutil_init
    float dd[3] = {d.d[0], d.d[1], d.ndim == 3 ? d.d[2] : 1.f};
    fd_coefficients(p->nop, d.ndim, dd, d.optfd, p->k);

    awe_status st = alloc_levels(p);
    if (st != AWE_OK && p->g.p1 != plain.p1) {
        p->g = plain;
        st = alloc_levels(p);
    }
    if (st != AWE_OK) return st;
    const size_t cells = (size_t)p->g.cells();
    AWE_TRY(dev_alloc(p, (void **)&p->corner_off, 8 * sizeof(long long)));

    if (d.dabc && !d.hybrid) {
        std::vector<float> w;
        sponge_weights(nb, w);
        const int len[3] = {p->g.n1, p->g.n2, p->g.n3};
        for (int a = 0; a < 3; a++) {
            std::vector<float> t(len[a], 1.f);
            if (a < d.ndim)
                for (int i = 0; i < nb && i < len[a]; i++) {
                    t[i] = w[nb - i - 1];
                    t[len[a] - 1 - i] = w[nb - i - 1];
                }
            undamped_range(t, p->wlo[a], p->whi[a]);
            t.resize((t.size() + 3) / 4 * 4, 1.f);  // read 4 at a time
            AWE_TRY(upload(p, &p->w[a], t.data(), t.size()));
        }
    }
    if (d.dabc && d.hybrid && nb - p->nop > 0) {
        std::vector<float> dm;
        hybrid_damp(nb - p->nop, dm);
        AWE_TRY(upload(p, &p->damp, dm.data(), dm.size()));
    }

    // TMA-staged step kernel for 3D up to 8th order
    if (!force_simple && stepB3_tma_eligible(d.ndim, p->nop, false, p->g)) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device);
        const char *lenv = std::getenv("AWE_TMA_CHUNK");
        p->tma_shape = stepB3_tma_shape(p->g, sms > 0 ? sms : 1, lenv ? std::atoi(lenv) : 0, p->nop);
        AWE_TRY(dev_alloc(p, (void **)&p->sched_counter, sizeof(unsigned long long)));
        AWE_TRY(dev_alloc(p, (void **)&p->d_err, sizeof(int)));
        CUDA_TRY(cudaMemset(p->sched_counter, 0, sizeof(unsigned long long)));
        CUDA_TRY(cudaMemset(p->d_err, 0, sizeof(int)));
        p->sched_base = 0;
        p->use_tma = stepB3_tma_maps(p->tmaps, p->u, p->vel, p->g, p->nop);
        // the gradient's TMA steps (L(u) stored, adjoint) are of 8th order, and
        // its FP64 result keeps the arithmetic of the kernels each grid has had
        p->tma_grad = p->use_tma && p->nop == 4 && p->g.n1 % 4 == 0;
        const char *spin = std::getenv("AWE_PIPELINE_SPIN_LIMIT");
        if (spin && *spin) p->spin_limit = std::atoll(spin);
    }
    if (d.ndim == 2 && !force_simple && p->nop <= 4 && !d.hybrid) {
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device);
        p->tb2_shape = tb2_shape(p->g, p->nop, sms > 0 ? sms : 1);
        // (without room for two more levels: one step a launch)
        p->tb2 = dev_alloc_extra(p, (void **)&p->tb2_u, 2 * cells * sizeof(float)) == AWE_OK;
    }
    // line-end copies of the 3D boundary launch (made before any capture of
    // the time loop; AWE_BND_ENDS=0, or no memory: the launch reads the level itself)
    const char *eenv = std::getenv("AWE_BND_ENDS");
    if (d.ndim == 3 && d.dabc && !d.hybrid && bnd3_eligible(p->nop, p->g) && !(eenv && std::strcmp(eenv, "0") == 0))
        for (int k = 0; k < 2; k++)
            if (dev_alloc_extra(p, (void **)&p->ends[k], (size_t)p->g.n2 * p->g.n3 * 16 * sizeof(float)) != AWE_OK) {
                dev_free(p, p->ends[0]);
                p->ends[0] = nullptr;
                break;
            }

    p->nsmp = (d.nt - 1) / d.jdata + 1;
    p->nsnap = d.jsnap > 0 ? (d.nt - 1) / d.jsnap + 1 : 0;
    for (int a = 0; a < 3; a++) {
        const int npad = a == 0 ? p->g.n1 : a == 1 ? p->g.n2 : p->g.n3;
        if (a >= d.ndim) {
            p->snap_f[a] = 0;
            p->snap_m[a] = 1;
        } else if (d.bnds) {
            p->snap_f[a] = 0;
            p->snap_m[a] = npad;
        } else {
            p->snap_f[a] = window_first(d.o[a], p->opad[a], d.d[a]);
            p->snap_m[a] = d.n[a];
        }
    }
    p->snap_elems = (size_t)p->snap_m[0] * p->snap_m[1] * p->snap_m[2];
    return AWE_OK;
}

awe_status planB_model(awe_plan *p, const float *vel, const float *den) {
    // The model goes to the device as passed, into a level buffer (the levels
    // are cleared at the start of every run), and the padded tables are made
    // there (k_model.cu): the same float operations as the host restatement
    // of fdutil.c's expand / abcone*_make, without a host pass over the
    // padded grid.
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const size_t cells = (size_t)g.cells();
    const size_t raw = (size_t)d.n[0] * d.n[1] * (d.ndim == 3 ? d.n[2] : 1);
    cudaStream_t s = p->stream;
    ModelPrep m{};
    m.g = g;
    m.n1 = d.n[0];
    m.n2 = d.n[1];
    m.n3 = d.ndim == 3 ? d.n[2] : 1;
    m.nb = p->nbd;
    m.nd = d.ndim;
    m.dt = d.dt;
    m.dt2 = d.dt * d.dt;
    m.d1 = d.d[0];
    m.d2 = d.d[1];
    m.d3 = d.ndim == 3 ? d.d[2] : 1.f;
    m.zero1 = (d.fsrf && !d.hybrid) ? std::min(p->nbd + 1, g.n1) : 0;
    float *stage = p->u[1];
    // no earlier work of this plan (on any stream) may still read the level
    // buffers or the model tables
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemcpyAsync(stage, vel, raw * sizeof(float), cudaMemcpyHostToDevice, s));
    if (d.dabc) {
        float *const tabs[6] = {p->abc[0], p->abc[1], p->abc[2], p->abc[3], p->abc[4], p->abc[5]};
        launch_model_abc(stage, m, tabs, s);
    }
    launch_model_pad(stage, p->vel, m, true, s);
    if (den) {
        CUDA_TRY(cudaMemcpyAsync(stage, den, raw * sizeof(float), cudaMemcpyHostToDevice, s));
        if (!p->den) AWE_TRY(dev_alloc(p, (void **)&p->den, cells * sizeof(float)));
        launch_model_pad(stage, p->den, m, false, s);
    } else if (p->den) {  // back to constant density
        dev_free(p, p->den);
        p->den = nullptr;
    }
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(s));
    return AWE_OK;
}

awe_status set_inj_cells(awe_plan *p) {
    const int nc = p->d.ndim == 3 ? 8 : 4, ns = (int)p->h_src.size();
    p->inj = InjCells{};
    // 2D steps add a few sources themselves; the gradient's fused adjoint step
    // (up to 2^24 cells) has lists of its own
    if (p->d.ndim == 2 && ns <= kFusedSources && p->g.cells() <= kFusedCells) return AWE_OK;
    std::vector<std::pair<long long, int>> e;  // (cell, source * 8 + corner)
    e.reserve((size_t)ns * nc);
    for (int s = 0; s < ns; s++)
        for (int c = 0; c < nc; c++) e.push_back({p->h_src[s].base + p->h_corner_off[c], 8 * s + c});
    std::sort(e.begin(), e.end());
    std::vector<long long> cell;
    std::vector<int> start;
    std::vector<int2> ent(e.size());
    for (size_t k = 0; k < e.size(); k++) {
        if (k == 0 || e[k].first != e[k - 1].first) {
            cell.push_back(e[k].first);
            start.push_back((int)k);
        }
        int w;
        std::memcpy(&w, &p->h_src[e[k].second >> 3].w[e[k].second & 7], sizeof w);
        ent[k] = make_int2(e[k].second, w);
    }
    start.push_back((int)e.size());
    if (cell.empty()) return AWE_OK;
    // sizes for every source at cells of its own, so that points that only
    // move keep the buffer (a captured time loop reads it)
    const size_t nmax = (size_t)ns * nc;
    const size_t o_ent = nmax * sizeof(long long), o_start = o_ent + nmax * sizeof(int2);
    const size_t bytes = o_start + (nmax + 1) * sizeof(int);
    if (p->inj_cap < bytes) {
        dev_free(p, p->inj_buf);
        p->inj_buf = nullptr;
        p->inj_cap = 0;
        // (without memory for them: one thread walks the sources)
        if (dev_alloc(p, &p->inj_buf, bytes) != AWE_OK) return AWE_OK;
        p->inj_cap = bytes;
    }
    char *b = (char *)p->inj_buf;
    CUDA_TRY(cudaMemcpy(b, cell.data(), cell.size() * sizeof(long long), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(b + o_ent, ent.data(), ent.size() * sizeof(int2), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(b + o_start, start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice));
    p->inj = InjCells{(int)cell.size(), (const long long *)b, (const int *)(b + o_start), (const int2 *)(b + o_ent)};
    return AWE_OK;
}

awe_status set_geometry_common(awe_plan *p, int ns, const float *sou, int nr, const float *rec) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const int nd = d.ndim;
    const long long s2 = g.s2(), s3 = g.s3();
    const bool spher = d.coords == AWE_SPHER;
    // reference fdm axes: cartesian z=axis1, x=axis2, y=axis3; spherical
    // programs map z=theta (axis 2), x=r (axis 1), y=phi (axis 3)
    // (MAWEFDspher3Dgpu.cu:167-173, MAWEFDspher2Dgpu.cu:151)
    FdmAxes f{};
    long long sz, sx, sy;
    if (!spher) {
        f = FdmAxes{p->opad[0], p->opad[1], p->opad[2], d.d[0], d.d[1], nd == 3 ? d.d[2] : 1.f, g.n1, g.n2, g.n3};
        sz = 1;
        sx = s2;
        sy = s3;
    } else {
        f = FdmAxes{p->opad[1], p->opad[0], p->opad[2], d.d[1], d.d[0], nd == 3 ? d.d[2] : 1.f, g.n2, g.n1, g.n3};
        sz = s2;
        sx = 1;
        sy = s3;
    }
    // corner order of lint*_make weights: (z, x[, y]) bits 001=z, 010=x, 100=y
    long long off[8];
    for (int c = 0; c < 8; c++) off[c] = ((c & 1) ? sz : 0) + ((c & 2) ? sx : 0) + ((c & 4) ? sy : 0);
    std::memcpy(p->h_corner_off, off, sizeof off);
    CUDA_TRY(cudaMemcpy(p->corner_off, off, sizeof off, cudaMemcpyHostToDevice));

    auto make = [&](const float *xyz, int n, std::vector<GeoPoint> &out, std::vector<Lint> *keep) {
        out.resize(n);
        if (keep) keep->resize(n);
        for (int i = 0; i < n; i++) {
            float x, y = 0.f, z;
            if (nd == 2) {
                x = xyz[2 * i];
                z = xyz[2 * i + 1];
            } else {
                x = xyz[3 * i];
                y = xyz[3 * i + 1];
                z = xyz[3 * i + 2];
            }
            Lint l = lint_make(nd, x, y, z, f);
            GeoPoint gp;
            gp.base = l.jz * sz + l.jx * sx + (nd == 3 ? l.jy * sy : 0);
            std::memcpy(gp.w, l.w, sizeof gp.w);
            out[i] = gp;
            if (keep) (*keep)[i] = l;
        }
    };
    make(sou, ns, p->h_src, &p->h_src_lint);
    make(rec, nr, p->h_rec, nullptr);
    // the point buffers are kept while large enough (a captured time loop
    // that read them stays valid)
    const int need_s = ns > 0 ? ns : 1, need_r = nr > 0 ? nr : 1;
    if (!p->src || p->src_cap < need_s) {
        if (p->src) dev_free(p, p->src);
        p->src = nullptr;
        p->src_cap = 0;
        AWE_TRY(dev_alloc(p, (void **)&p->src, need_s * sizeof(GeoPoint)));
        p->src_cap = need_s;
    }
    if (!p->rec || p->rec_cap < need_r) {
        if (p->rec) dev_free(p, p->rec);
        p->rec = nullptr;
        p->rec_cap = 0;
        AWE_TRY(dev_alloc(p, (void **)&p->rec, need_r * sizeof(GeoPoint)));
        p->rec_cap = need_r;
    }
    CUDA_TRY(cudaDeviceSynchronize());  // earlier runs may still read the old points
    if (ns) CUDA_TRY(cudaMemcpy(p->src, p->h_src.data(), ns * sizeof(GeoPoint), cudaMemcpyHostToDevice));
    if (nr) CUDA_TRY(cudaMemcpy(p->rec, p->h_rec.data(), nr * sizeof(GeoPoint), cudaMemcpyHostToDevice));
    p->ns = ns;
    p->nr = nr;

    // scheme CPU: a source node inside the sponge band but outside the
    // boundary shell would be sponged before its injection by the fused
    // step; such runs defer the whole sponge to after the injection.
    // src_in_shell: a corner lies on a cell that the 3D boundary launch stores
    // (the shell, and the eight cells it rewrites at each end of a line).  A
    // corner of weight 0 counts: its cell is read and stored all the same.
    p->sponge_deferred = false;
    p->src_in_shell = false;
    if (d.scheme == AWE_SCHEME_CPU && d.dabc && !d.hybrid) {
        const int shell = (nd == 3) ? p->nop + 2 : 0, ends = (nd == 3) ? std::max(shell, kBndEnd) : 0;
        const int nc = nd == 3 ? 8 : 4;
        for (const GeoPoint &gp : p->h_src)
            for (int c = 0; c < nc; c++) {
                const long long n = gp.base + off[c];
                const int i3 = (int)(n / s3), i2 = (int)((n % s3) / s2), i1 = (int)(n % s2);
                const int ii[3] = {i1, i2, i3}, nn[3] = {g.n1, g.n2, g.n3};
                bool band = false, inshell = false, stored = false;
                for (int a = 0; a < nd; a++) {
                    const int dist = std::min(ii[a], nn[a] - 1 - ii[a]);
                    band = band || dist < p->nbd;
                    inshell = inshell || dist < shell;
                    stored = stored || dist < (a == 0 ? ends : shell);
                }
                if (gp.w[c] != 0.f && band && !inshell) p->sponge_deferred = true;
                if (stored) p->src_in_shell = true;
            }
    }
    return AWE_OK;
}

bool stepB3_bnd(const awe_plan *p) {
    const awe_desc &d = p->d;
    const char *env = std::getenv("AWE_BND3");
    return d.scheme == AWE_SCHEME_CPU && d.ndim == 3 && d.dabc && !d.hybrid && !p->sponge_deferred &&
           bnd3_eligible(p->nop, p->g) && !(env && std::strcmp(env, "0") == 0);
}

StepBParams stepB_params(const awe_plan *p) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const bool sponge = d.dabc && !d.hybrid;
    StepBParams sp{};
    sp.g = g;
    sp.k = p->k;
    sp.nop = p->nop;
    sp.w1 = p->w[0];
    sp.w2 = p->w[1];
    sp.w3 = p->w[2];
    sp.damp_prev = sponge;
    sp.sponge_new = sponge && !p->sponge_deferred;
    sp.shell = (d.ndim == 3 && sponge) ? p->nop + 2 : 0;
    for (int a = 0; a < 3; a++) {
        sp.ilo[a] = sponge ? p->wlo[a] : 0;
        sp.ihi[a] = sponge ? p->whi[a] : (a == 0 ? g.n1 : a == 1 ? g.n2 : g.n3);
    }
    sp.prv = nullptr;
    sp.spin = p->spin_limit;
    return sp;
}

// One full time step it: the new level is written to `nxt`, which is the
// buffer holding the previous level (in place, prv_map == null or the TMA
// maps of that buffer) or a third buffer (out of place: `prv` names the
// previous level, and for the TMA kernel `cur_map`/`prv_map` are given).
awe_status stepB_full(awe_plan *p, const StepBParams &sp0, const float *prv, const float *cur, float *nxt, int it,
                      const float *d_wav, int ncs, const CUtensorMap *cur_map, const CUtensorMap *prv_map,
                      cudaStream_t s, long long &launches, float *lap_out, const GeoPoint *ext_pts, int ext_n,
                      int ext_stride, float *ext_row) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const bool exact = d.precision == AWE_EXACT;
    const bool sponge = d.dabc && !d.hybrid;
    const int shell = sp0.shell;
    StepBParams sp = sp0;
    sp.prv = (prv != nxt) ? prv : nullptr;
    // 2D: sources (few) and receivers ride in the step kernel's launch
    const bool fuse_src = d.ndim == 2 && p->ns > 0 && p->ns <= kFusedSources;
    if (fuse_src) {
        const PointsAt ps = points_at(p, p->src, p->ns, p->src_rows, it);
        sp.inj = ps.pts;
        sp.inj_n = p->ns;
        sp.inj_stride = ps.stride;
        sp.inj_wav = d_wav;
        sp.inj_it = it;
        sp.inj_ncs = ncs;
        sp.inj_one = ncs == 1;
    }
    if (d.ndim == 2 && ext_n > 0) {
        sp.ext = ext_pts;
        sp.ext_n = ext_n;
        sp.ext_stride = ext_stride;
        sp.ext_row = ext_row;
    }
    prof_begin(p, s);
    if (p->use_tma && !p->den && cur_map && prv_map) {  // (no density term there)
        cudaError_t e = launch_stepB3_tma_with(exact, *cur_map, *prv_map, p->tmaps[4], nxt, sp, p->tma_shape,
                                               p->sched_counter, p->sched_base, p->d_err, s, lap_out);
        p->sched_base += (unsigned long long)p->tma_shape.items + p->tma_shape.grid;
        if (e != cudaSuccess) {
            set_error("TMA step launch failed: %s", cudaGetErrorString(e));
            return AWE_ERR_CUDA;
        }
    } else {
        launch_stepB(d.ndim, p->nop, exact, p->den != nullptr, cur, nxt, p->vel, p->den, sp, s);
    }
    prof_end(p, s);
    launches++;
    const bool bnd = stepB3_bnd(p);
    // the boundary launch injects too, unless a source touches the cells the ABC reads
    const bool inj_in_bnd = bnd && !p->src_in_shell;
    if (p->ns > 0 && !fuse_src && !inj_in_bnd) {
        const PointsAt ps = points_at(p, p->src, p->ns, p->src_rows, it);
        if (p->move_mode < 0 && p->inj.n > 0)
            launch_injectB_cells(exact, nxt, p->vel, p->inj, d_wav, it, ncs, ncs == 1, s);
        else
            launch_injectB_off(d.ndim, exact, nxt, p->vel, ps.pts, p->ns, d_wav, it, ncs, ncs == 1, p->corner_off, s,
                               ps.stride);
        launches++;
    }
    if (bnd) {
        Bnd3Params bp{};
        bp.g = g;
        bp.nop = p->nop;
        bp.uo = nxt;
        bp.um = cur;
        bp.vel = p->vel;
        bp.zl = p->abc[0];
        bp.zh = p->abc[1];
        bp.xl = p->abc[2];
        bp.xh = p->abc[3];
        bp.yl = p->abc[4];
        bp.yh = p->abc[5];
        bp.w1 = p->w[0];
        bp.w2 = p->w[1];
        bp.w3 = p->w[2];
        bp.top = !d.fsrf;
        if (p->ends_run) {
            bp.em = p->ends[p->ends_idx];
            bp.eo = p->ends[1 - p->ends_idx];
            p->ends_idx ^= 1;
        }
        bp.rec = ext_pts;
        bp.nr = ext_n;
        bp.rec_stride = ext_stride;
        bp.rec_row = ext_n > 0 ? ext_row : nullptr;
        if (inj_in_bnd && p->ns > 0) {
            const PointsAt ps = points_at(p, p->src, p->ns, p->src_rows, it);
            bp.src = ps.pts;
            bp.ns = p->ns;
            bp.src_stride = ps.stride;
            if (p->move_mode < 0) bp.inj = p->inj;
            bp.wav = d_wav;
            bp.it = it;
            bp.ncs = ncs;
            bp.one_wavelet = ncs == 1;
        }
        launch_bnd3(exact, bp, s);
        launches++;
        return AWE_OK;
    }
    if (d.dabc) {
        AbcB abc{p->abc[0], p->abc[1], p->abc[2], p->abc[3], p->abc[4], p->abc[5]};
        if (d.hybrid) {
            launch_hybridB(d.ndim, p->nop, p->nbd, exact, d.fsrf, nxt, cur, abc, p->damp, g, s);
            launches += d.ndim;
        } else {
            // the axis-1 ABC pass also applies the shell sponge to the axis-1 ends of
            // lines the later passes leave alone (not when the sponge is deferred)
            const bool zf = sponge && !p->sponge_deferred && shell > 0 && d.ndim == 3 && abc_zfused(p->nop, g, shell);
            if (d.ndim == 3) {
                if (zf) launch_abconeB(3, p->nop, exact, d.fsrf, nxt, cur, abc, g, s, p->w[0], p->w[1], p->w[2], shell);
                else launch_abconeB(3, p->nop, exact, d.fsrf, nxt, cur, abc, g, s);
                launches += 3;
            }
            if (sponge && p->sponge_deferred) {
                launch_band_sponge(d.ndim, std::max(p->nbd, shell), exact, nxt, p->w[0], p->w[1], p->w[2], g, s);
                launches += d.ndim;  // one kernel per slab orientation
            } else if (shell > 0) {
                launch_band_sponge(d.ndim, shell, exact, nxt, p->w[0], p->w[1], p->w[2], g, s, zf ? 1 : 0);
                launches += d.ndim;
            }
        }
    }
    return AWE_OK;
}

awe_status planB_run(awe_plan *p, const float *d_wav, int ncs, float *d_dat, float *d_wfl, cudaStream_t s) {
    return planB_run_hooked(p, d_wav, ncs, d_dat, d_wfl, s, nullptr);
}

awe_status planB_run_hooked(awe_plan *p, const float *d_wav, int ncs, float *d_dat, float *d_wfl, cudaStream_t s,
                            const StepHook *hook, int hook_every) {
    const awe_desc &d = p->d;
    const Grid &g = p->g;
    const bool exact = d.precision == AWE_EXACT;
    const bool sponge = d.dabc && !d.hybrid;
    const size_t bytes = (size_t)g.cells() * sizeof(float);
    long long launches = 0;

    CUDA_TRY(cudaMemsetAsync(p->u[0], 0, bytes, s));
    CUDA_TRY(cudaMemsetAsync(p->u[1], 0, bytes, s));
    if (p->use_tma) {  // the TMA kernel's work counter restarts with every run (graph replays included)
        CUDA_TRY(cudaMemsetAsync(p->sched_counter, 0, sizeof(unsigned long long), s));
        p->sched_base = 0;
    }
    if (p->nsnap > 0 && !d_wfl && p->snap_cb && !p->d_snap_tmp)
        AWE_TRY(dev_alloc(p, (void **)&p->d_snap_tmp, p->snap_elems * sizeof(float)));
    // the boundary launches pass the line ends from step to step; the first
    // step reads those of the zero level
    struct EndsOff {
        awe_plan *p;
        ~EndsOff() { p->ends_run = false; }
    } ends_off{p};
    p->ends_run = false;
    if (p->ends[0] && stepB3_bnd(p)) {
        CUDA_TRY(cudaMemsetAsync(p->ends[0], 0, (size_t)g.n2 * g.n3 * 16 * sizeof(float), s));
        p->ends_idx = 0;
        p->ends_run = true;
    }
    p->snap_pending = -1;  // a frame left queued by a failed run is not delivered

    const StepBParams sp = stepB_params(p);
    const float *pw1 = sponge ? p->w[0] : nullptr;

    float *cur = p->u[1], *nxt = p->u[0];
    int icur = 1;
    int row = 0, isnap = 0;
    // 2D: the traces of step it (the level the step reads, pending sponge
    // applied, as the reference extracts after its swap) are gathered by the
    // step's own launch; 3D: by the step's boundary launch
    if (p->tb2_fwd.ok && !p->den) {
        // several steps a launch, stopping at steps whose levels the hook or a frame reads
        float *alt_prv = p->tb2_u, *alt_cur = p->tb2_u + g.cells();
        float *prv = nxt;
        const bool frames = p->nsnap > 0 && (d_wfl || p->d_snap_tmp);
        for (int it = 0; it < d.nt;) {
            if (hook && it % hook_every == 0) AWE_TRY((*hook)(it, prv, cur, s));
            if (frames && it % d.jsnap == 0) {
                float *frame = d_wfl ? d_wfl + (size_t)isnap * p->snap_elems : p->d_snap_tmp;
                launch_snapshot(2, cur, frame, g, p->snap_f[0], p->snap_f[1], p->snap_f[2], p->snap_m[0], p->snap_m[1],
                                p->snap_m[2], pw1, p->w[1], p->w[2], s);
                launches++;
                AWE_TRY(deliver_snapshot(p, frame, isnap, it, s));
                isnap++;
            }
            int k = std::min(p->tb2_shape.k, d.nt - it);
            if (hook) k = std::min(k, hook_every - it % hook_every);
            if (frames) k = std::min(k, d.jsnap - it % d.jsnap);
            tb2_launch(p, false, prv, cur, alt_prv, alt_cur, nullptr, false, it, k, d_wav, ncs, d_dat, s);
            launches++;
            std::swap(prv, alt_prv);
            std::swap(cur, alt_cur);
            it += k;
        }
        p->launches = launches;
        return flush_snapshots(p);
    }
    const bool fuse_rec = (d.ndim == 2 || stepB3_bnd(p)) && p->nr > 0;
    const bool tma = p->use_tma && (!hook || p->tma_grad);
    for (int it = 0; it < d.nt; it++) {
        if (hook) AWE_TRY((*hook)(it, nxt, cur, s));
        const bool ext = fuse_rec && it % d.jdata == 0;
        const PointsAt pe = points_at(p, p->rec, p->nr, p->rec_rows, it);
        AWE_TRY(stepB_full(p, sp, nxt, cur, nxt, it, d_wav, ncs, tma ? &p->tmaps[icur] : nullptr,
                           tma ? &p->tmaps[2 + (1 - icur)] : nullptr, s, launches, nullptr, pe.pts, ext ? p->nr : 0, pe.stride,
                           ext ? d_dat + (size_t)row * p->nr : nullptr));
        std::swap(cur, nxt);  // nxt now holds the time level `it` (sponge pending)
        icur ^= 1;
        if (p->nsnap > 0 && it % d.jsnap == 0) {
            float *frame = d_wfl ? d_wfl + (size_t)isnap * p->snap_elems : p->d_snap_tmp;
            if (frame) {
                launch_snapshot(d.ndim, nxt, frame, g, p->snap_f[0], p->snap_f[1], p->snap_f[2], p->snap_m[0],
                                p->snap_m[1], p->snap_m[2], pw1, p->w[1], p->w[2], s);
                launches++;
                AWE_TRY(deliver_snapshot(p, frame, isnap, it, s));
            }
            isnap++;
        }
        if (it % d.jdata == 0) {
            if (!fuse_rec) {
                const PointsAt pr = points_at(p, p->rec, p->nr, p->rec_rows, it);
                launch_extract_off(d.ndim, exact, nxt, pr.pts, p->nr, d_dat + (size_t)row * p->nr, pw1, p->w[1],
                                   p->w[2], g, p->corner_off, s, pr.stride);
                launches += p->nr > 0;
            }
            row++;
        }
    }
    p->launches = launches;
    return flush_snapshots(p);
}

}  // namespace awe
