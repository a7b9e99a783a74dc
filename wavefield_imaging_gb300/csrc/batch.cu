// Host side of the batched 2D forward (awe_batch_*): many shots along a
// track, each on its own window of one model (the c1-style survey of
// byrne_awe.py, one sfAWEFDcart2Dcpu run per window), advanced together.
//
// All shots' padded fields live in three concatenated arrays; every time step
// is one launch of k_batch2d over the flat (shot, tile) + (shot, receiver
// block) item list; the nt launches are captured once into a CUDA graph and
// replayed.  The autotuner times each tile shape and grid size on a few steps
// and keeps the fastest.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "awe_internal.h"

using namespace awe;

struct awe_batch {
    awe_desc d{};
    int device = 0;
    cudaStream_t stream = nullptr;
    int nop = 4, nb = 0, n1 = 0;  // padded rows
    Coef k{};
    std::vector<awe_shot> shots_in;
    std::vector<BatchShot> shots;
    std::vector<float> h_wz, h_wx;
    std::vector<int4> items;
    int ntile_items = 0;
    long long cells = 0, ndat = 0;
    int nsmp = 0;
    std::vector<std::pair<void *, size_t>> allocs;
    size_t held = 0;  // their bytes
    float *u[2] = {nullptr, nullptr}, *vel = nullptr, *wz = nullptr, *wx = nullptr, *wav = nullptr, *dat = nullptr;
    BatchShot *d_shots = nullptr;
    int4 *d_items = nullptr;
    size_t items_cap = 0;
    GeoPoint *src = nullptr, *rec = nullptr;
    bool model_set = false;
    int tile = 0, grid = 0, sms = 1;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    long long launches = 0;
    std::vector<GeoPoint> h_rec;
    // misfit gradient state
    int gT = 0, gseg = 0, gfmt = -1;
    long long gscale_per = 0;  // checkpoint scales per level: one per shot, or per 64-cell block (BFP16)
    float *slots = nullptr, *gX = nullptr, *gY = nullptr, *res = nullptr, *scales = nullptr, *dobs = nullptr;
    void *ckpt = nullptr;
    float2 *G = nullptr;  // gradient accumulators (compensated pairs)
    double *part = nullptr, *grad = nullptr;
    // receiver cells of the adjoint's residual term (-1: not built yet)
    BatchRecCell *rec_cells = nullptr;
    BatchRecW *rec_ws = nullptr;
    int nrec_cells = -1;
    int2 *win = nullptr;
    // column-march forward (k_batch2d_col): chunk length (0 = the tile kernels), its items and grid
    int colL = 0, col_grid = 0, ncol_items = 0;
    std::vector<int4> col_items;
    int4 *d_col_items = nullptr;
    size_t col_cap = 0;
    int *d_err = nullptr;  // set by a bulk-copy wait that timed out
    int col_adj_grid = 0;  // column-march adjoint's grid (0: the tile adjoint)
    // several steps a launch (k_tb2d.cu): possible for these points, the forward's; two more
    // levels, the tiles, the point lists of the forward and of the adjoint
    bool tb2_ok = false, tb2 = false, selected = false;  // selected: a kernel by awe_batch_select
    Tb2Shape tb2_shape{};
    std::vector<Tb2Grid> tb2_grids;
    int tb2_tiles = 0, tb2_ncols = 0;
    float *tb2_u = nullptr, *tb2_xy = nullptr;
    int2 *d_tb2_cols = nullptr;
    struct Lists {
        int *buf = nullptr;
        Tb2Tile *tiles = nullptr;
        size_t off[7] = {};
        int most[3] = {};
    } tb2_fwd, tb2_adj;
    bool tb2_grad = false, tb2_tried = false;  // the gradient's slots hold both sweeps of a segment; asked for
    bool grad_busy = false;                    // a call uses the gradient's buffers
    std::vector<GeoPoint> h_src;
};

#define CUDA_TRY(expr)                                                                            \
    do {                                                                                          \
        cudaError_t e_ = (expr);                                                                  \
        if (e_ != cudaSuccess) {                                                                  \
            set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
            return AWE_ERR_CUDA;                                                                  \
        }                                                                                         \
    } while (0)

static void drop_graph(awe_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
}

// Optional cap on the device memory one batch may hold (AWE_BATCH_BYTES_LIMIT,
// bytes, read at every allocation), as AWE_DEVICE_BYTES_LIMIT is for a plan.
static size_t batch_bytes_limit() {
    const char *e = std::getenv("AWE_BATCH_BYTES_LIMIT");
    return e && *e ? (size_t)std::strtoull(e, nullptr, 10) : (size_t)0;
}

// memory the batch can do without; null and AWE_ERR_NOMEM where there is none left
static awe_status balloc_extra(awe_batch *b, void **p, size_t bytes) {
    *p = nullptr;
    if (bytes == 0) bytes = 16;
    const size_t lim = batch_bytes_limit();
    if (lim && b->held + bytes > lim) {
        set_error("device memory limit: %zu bytes held + %zu requested > AWE_BATCH_BYTES_LIMIT %zu", b->held, bytes,
                  lim);
        return AWE_ERR_NOMEM;
    }
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        set_error("cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
        return AWE_ERR_NOMEM;
    }
    b->allocs.push_back({*p, bytes});
    b->held += bytes;
    return AWE_OK;
}

template <class T>
static void bfree(awe_batch *b, T *&p) {
    for (auto it = b->allocs.begin(); it != b->allocs.end(); ++it)
        if (it->first == (void *)p) {
            b->held -= it->second;
            b->allocs.erase(it);
            cudaFree(p);
            break;
        }
    p = nullptr;
}

// Gives back what the batch can do without: the gradient's slots for several
// steps a launch while no call uses them (the next one allocates what then
// fits), then the levels, lists and tiles of k_tb2d.cu.
static bool release_extra(awe_batch *b) {
    if (b->tb2_grad && !b->grad_busy) {
        bfree(b, b->slots);
        bfree(b, b->tb2_xy);
        b->gT = 0;
        b->tb2_grad = b->tb2_tried = false;
        return true;
    }
    if (!b->tb2_ok) return false;
    drop_graph(b);  // reads them
    bfree(b, b->tb2_u);
    bfree(b, b->tb2_xy);
    bfree(b, b->d_tb2_cols);
    for (awe_batch::Lists *l : {&b->tb2_fwd, &b->tb2_adj}) {
        bfree(b, l->buf);
        bfree(b, l->tiles);
    }
    b->tb2_ok = b->tb2 = b->tb2_grad = false;
    return true;
}

static awe_status balloc(awe_batch *b, void **p, size_t bytes) {
    awe_status st = balloc_extra(b, p, bytes);
    while (st != AWE_OK && release_extra(b)) st = balloc_extra(b, p, bytes);
    return st;
}

// items to a device buffer that is kept while large enough (the tuner tries
// several lists) and stays as it is if a larger one cannot be had; no launch
// that reads it may be in flight
static awe_status upload(awe_batch *b, const std::vector<int4> &v, int4 *&d, size_t &cap) {
    if (cap < v.size()) {
        int4 *larger = nullptr;
        const awe_status st = balloc(b, (void **)&larger, v.size() * sizeof(int4));
        if (st != AWE_OK) return st;
        bfree(b, d);
        d = larger;
        cap = v.size();
    }
    CUDA_TRY(cudaMemcpy(d, v.data(), v.size() * sizeof(int4), cudaMemcpyHostToDevice));
    return AWE_OK;
}

// the receiver blocks of every shot, after its tiles or column chunks
static void add_rec_items(const awe_batch *b, std::vector<int4> &v) {
    for (int s = 0; s < (int)b->shots.size(); s++)
        for (int r = 0; r < b->shots[s].nr; r += kBatchRecBlock) v.push_back(make_int4(s, r, 0, 1));
}

// the tile kernels' items (shot, tile) for a tile shape
static awe_status set_tile(awe_batch *b, int tile) {
    const int TZ = kBatchTiles[tile][0], TX = kBatchTiles[tile][1];
    std::vector<int4> v;
    for (int s = 0; s < (int)b->shots.size(); s++)
        for (int x0 = 0; x0 < b->shots[s].n2; x0 += TX)
            for (int z0 = 0; z0 < b->n1; z0 += TZ) v.push_back(make_int4(s, z0, x0, 0));
    const int n = (int)v.size();
    add_rec_items(b, v);
    const awe_status st = upload(b, v, b->d_items, b->items_cap);
    if (st != AWE_OK) return st;
    b->items.swap(v);
    b->ntile_items = n;
    b->tile = tile;
    return AWE_OK;
}

// the column march's items (shot, x0) for chunks of L columns
static awe_status set_columns(awe_batch *b, int L) {
    std::vector<int4> v;
    for (int s = 0; s < (int)b->shots.size(); s++)
        for (int x0 = 0; x0 < b->shots[s].n2; x0 += L) v.push_back(make_int4(s, 0, x0, 0));
    const int n = (int)v.size();
    add_rec_items(b, v);
    const awe_status st = upload(b, v, b->d_col_items, b->col_cap);
    if (st != AWE_OK) return st;
    b->col_items.swap(v);
    b->ncol_items = n;
    b->colL = L;
    return AWE_OK;
}

// Tile of k_tb2d.cu for all windows: 4 columns a thread, up to 256 threads, two
// blocks per SM (one loads while the other steps).  A tile of r cells with its
// halos takes about 2 us a launch and 0.25 us + 0.15 ns r a step alone on an SM,
// 1.2 times as long beside another; lines of a multiple of 8 strips read shared
// memory without bank conflicts (5 %).  Fitted to 12 windows of 592 x 580 cells at
// 8th order, where 48 x 48 cells took 14.3 us a step with 2 steps a launch, 18.1
// with one (56 x 56), 15.5 with three (40 x 40), and the one-step kernels 17.8.
static bool tb2_batch_shape(const std::vector<BatchShot> &shots, int n1, int nop, int sms, Tb2Shape &best) {
    long long ntx[31] = {};  // tile columns of all windows by tx / 4 (one pass: there may be thousands of windows)
    for (const BatchShot &sh : shots)
        for (int q = 2; q <= 30; q++) ntx[q] += (sh.n2 + 4 * q - 1) / (4 * q);
    double cost = 1e30;
    for (int tz0 = 8; tz0 <= 120; tz0 += 4)
        for (int tx = 8; tx <= 120; tx += 4)
            for (int k = 1; k <= 12; k++) {
                Tb2Shape s{};
                s.k = k;
                s.cx = 4;
                s.ntz = (n1 + tz0 - 1) / tz0;
                s.tz = ((n1 + s.ntz - 1) / s.ntz + 3) / 4 * 4;
                s.ntz = (n1 + s.tz - 1) / s.tz;
                s.tx = tx;
                s.hx = nop * k;
                s.hz = (s.hx + 3) / 4 * 4;
                s.rz = s.tz + 2 * s.hz;
                s.rx = (s.tx + 2 * s.hx + 3) / 4 * 4;
                if ((s.rz / 4) * (s.rx / 4) > kTb2BatchThreads) break;
                const long long tiles = s.ntz * ntx[tx / 4];
                const double r = (double)s.rz * s.rx;
                const double rounds = tiles <= sms ? 1.0 : std::max(1.0, 0.6 * tiles / sms);
                const double c = rounds * (2.0 / k + 0.25 + 1.5e-4 * r) * (s.rz % 32 ? 1.05 : 1.0);
                if (c < cost) {
                    cost = c;
                    best = s;
                }
            }
    return cost < 1e30;
}

static awe_status upload_lists(awe_batch *b, awe_batch::Lists &l, const Tb2HostLists &h) {
    const Tb2Shape &sh = b->tb2_shape;
    std::vector<Tb2Tile> tiles;
    for (size_t s = 0; s < b->shots.size(); s++)
        for (int k = 0; k < b->tb2_grids[s].ntx * sh.ntz; k++) {
            const BatchShot &q = b->shots[s];
            const int n = (int)tiles.size();
            const int *c = &h.buf[h.off[0] + n], *e = &h.buf[h.off[1] + n], *r = &h.buf[h.off[2] + n];
            tiles.push_back({q.off, q.dat_off, q.n2, q.wx_off, q.nr, k % sh.ntz * sh.tz, k / sh.ntz * sh.tx, r[0],
                             r[1] - r[0], c[0], c[1] - c[0], e[0], e[1] - e[0], 0});
        }
    awe_status st = balloc_extra(b, (void **)&l.buf, h.buf.size() * sizeof(int));
    if (st == AWE_OK) st = balloc_extra(b, (void **)&l.tiles, tiles.size() * sizeof(Tb2Tile));
    if (st != AWE_OK) {
        bfree(b, l.buf);
        return st;
    }
    CUDA_TRY(cudaMemcpy(l.tiles, tiles.data(), tiles.size() * sizeof(Tb2Tile), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(l.buf, h.buf.data(), h.buf.size() * sizeof(int), cudaMemcpyHostToDevice));
    std::copy(h.off, h.off + 7, l.off);
    std::copy(h.most, h.most + 3, l.most);
    return AWE_OK;
}

// tiles and point lists of k_tb2d.cu; b->tb2_ok stays false where it does not
// apply (order above 8, a source in the sponge, points on a window's last
// line, too many in a tile, no memory for two more levels)
static awe_status set_tb2(awe_batch *b) {
    const char *kern = std::getenv("AWE_STEP_KERNEL");
    if (b->nop > 4 || (kern && std::strcmp(kern, "simple") == 0)) return AWE_OK;
    for (const BatchShot &sh : b->shots)
        for (int k = 0; k < sh.ns; k++) {
            const GeoPoint &g = b->h_src[sh.src0 + k];
            for (int c = 0; c < 4; c++) {
                const long long n = g.base + (c & 1) + (c >> 1) * (long long)b->n1;
                if (g.w[c] == 0.f || n >= (long long)sh.n2 * b->n1) continue;
                if (b->h_wz[n % b->n1] != 1.f || b->h_wx[sh.wx_off + n / b->n1] != 1.f) return AWE_OK;
            }
        }
    if (!tb2_batch_shape(b->shots, b->n1, b->nop, std::max(b->sms, 1), b->tb2_shape)) return AWE_OK;
    const Tb2Shape &sh = b->tb2_shape;
    std::vector<int2> cols;
    for (int s = 0; s < (int)b->shots.size(); s++) {
        const BatchShot &q = b->shots[s];
        const int ntx = (q.n2 + sh.tx - 1) / sh.tx;
        b->tb2_grids.push_back({b->n1, q.n2, ntx, b->tb2_tiles, b->h_src.data() + q.src0, q.ns,
                                b->h_rec.data() + q.rec0, q.nr});
        b->tb2_tiles += ntx * sh.ntz;
        for (int x = 0; x < q.n2; x += 4) cols.push_back(make_int2(s, x));
    }
    b->tb2_ncols = (int)cols.size();
    Tb2HostLists h;
    if (!tb2_host_lists(sh, b->tb2_grids, b->tb2_tiles, h)) return AWE_OK;
    awe_status st = upload_lists(b, b->tb2_fwd, h);
    if (st == AWE_OK) st = balloc_extra(b, (void **)&b->d_tb2_cols, cols.size() * sizeof(int2));
    if (st == AWE_OK) st = balloc_extra(b, (void **)&b->tb2_u, (size_t)2 * b->cells * sizeof(float));
    if (st == AWE_ERR_NOMEM) {
        bfree(b, b->tb2_fwd.buf);
        bfree(b, b->tb2_fwd.tiles);
        bfree(b, b->d_tb2_cols);
        return AWE_OK;
    }
    if (st != AWE_OK) return st;
    CUDA_TRY(cudaMemcpy(b->d_tb2_cols, cols.data(), cols.size() * sizeof(int2), cudaMemcpyHostToDevice));
    b->tb2_ok = true;
    b->tb2 = b->tb2_ok;
    return AWE_OK;
}

// k steps of every window from levels prv, cur: it .. it + k - 1 forward, it ..
// it - k + 1 of the adjoint; slots: L of the levels read (adjoint: nu)
static void tb2_steps(awe_batch *b, bool adj, const float *prv, const float *cur, float *oprv, float *ocur,
                      float *slots, int it, int k, bool receivers, cudaStream_t s) {
    const Tb2Shape &sh = b->tb2_shape;
    const awe_batch::Lists &l = adj ? b->tb2_adj : b->tb2_fwd;
    Tb2Params q{};
    q.n1 = b->n1;
    q.k = k;
    q.it = it;
    q.tz = sh.tz, q.tx = sh.tx, q.hz = sh.hz, q.hx = sh.hx, q.rz = sh.rz, q.rx = sh.rx;
    q.c0 = b->k.c0;
    for (int i = 0; i <= b->nop; i++) q.cz[i] = b->k.c[0][i], q.cx[i] = b->k.c[1][i];
    q.cur = cur, q.prv = prv, q.vel = b->vel, q.ocur = ocur, q.oprv = oprv;
    q.slots = slots;
    q.slot_stride = b->cells;
    q.w1 = b->wz, q.w2 = b->wx;  // (all 1 without a sponge)
    undamped_range(b->h_wz, q.ilo1, q.ihi1);
    q.ilo2 = q.ilo1;  // (a window's axis-2 factors mirror the same profile: its high end is n2 - ilo2)
    tb2_set_lists(q, l.buf, l.off, l.most, true, receivers);
    q.wav = adj ? b->res : b->wav;
    q.ncs = 1;
    q.jdata = b->d.jdata;
    q.dat = b->dat;  // (read with q.rec_start only)
    q.tiles = l.tiles;
    launch_tb2_batch(b->nop, adj ? 2 : slots ? 3 : 0, q, sh, b->tb2_tiles, tb2_smem(sh, l.most), s);
}

static BatchStep step_params(const awe_batch *b, int it) {
    BatchStep p{};
    // level it lives in u[it & 1] (cur); the new level overwrites u[(it + 1) & 1]
    p.cur = b->u[it & 1];
    p.nxt = b->u[(it + 1) & 1];
    p.vel = b->vel;
    p.wz = b->wz;
    p.wx = b->wx;
    p.sponge = b->d.dabc ? 1 : 0;
    p.n1 = b->n1;
    p.c0 = b->k.c0;
    for (int i = 0; i <= kMaxNop; i++) {
        p.cz[i] = b->k.c[0][i];
        p.cx[i] = b->k.c[1][i];
    }
    p.src = b->src;
    p.rec = b->rec;
    p.wav = b->wav;
    p.it = it;
    p.dat = b->dat;
    p.row = (it % b->d.jdata == 0) ? it / b->d.jdata : -1;
    return p;
}

// one forward step with the chosen kernel; without receivers: the column or
// tile items alone (the gradient's recompute)
static void launch_fwd(awe_batch *b, const BatchStep &p, cudaStream_t s, bool receivers) {
    if (b->colL > 0)
        launch_batch2d_col(b->d_shots, b->d_col_items, receivers ? (int)b->col_items.size() : b->ncol_items,
                           b->col_grid, b->colL, p, b->d_err, s);
    else
        launch_batch2d(b->nop, b->tile, b->d_shots, b->d_items, receivers ? (int)b->items.size() : b->ntile_items,
                       b->grid, p, s);
}

// steps it0 .. it1 - 1; hook(it, prv, cur) sees the levels before every step it % every == 0
template <class Hook>
static void tb2_range(awe_batch *b, int it0, int it1, cudaStream_t s, int every, const Hook &hook) {
    float *prv = b->u[(it0 + 1) & 1], *cur = b->u[it0 & 1];
    float *prv2 = b->tb2_u, *cur2 = b->tb2_u + b->cells;
    for (int it = it0; it < it1;) {
        int k = std::min(b->tb2_shape.k, it1 - it);
        if (every > 0) {
            if (it % every == 0) hook(it, prv, cur);
            k = std::min(k, every - it % every);
        }
        tb2_steps(b, false, prv, cur, prv2, cur2, nullptr, it, k, b->ndat > 0, s);
        std::swap(prv, prv2);
        std::swap(cur, cur2);
        it += k;
    }
}

static void launch_range(awe_batch *b, int it0, int it1, cudaStream_t s) {
    if (b->tb2) return tb2_range(b, it0, it1, s, 0, [](int, float *, float *) {});
    for (int it = it0; it < it1; it++) {
        const BatchStep p = step_params(b, it);
        if (b->colL > 0)
            launch_batch2d_col(b->d_shots, b->d_col_items, (int)b->col_items.size(), b->col_grid, b->colL, p,
                               b->d_err, s);
        else
            launch_batch2d(b->nop, b->tile, b->d_shots, b->d_items, (int)b->items.size(), b->grid, p, s);
    }
}

static awe_status run_all(awe_batch *b, cudaStream_t s) {
    const size_t bytes = (size_t)b->cells * sizeof(float);
    CUDA_TRY(cudaMemsetAsync(b->u[0], 0, bytes, s));
    CUDA_TRY(cudaMemsetAsync(b->u[1], 0, bytes, s));
    CUDA_TRY(cudaMemsetAsync(b->d_err, 0, sizeof(int), s));
    if (!b->exec) {
        // capture the nt step launches once; replays reuse the same buffers
        cudaStream_t cs;
        CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            launch_range(b, 0, b->d.nt, cs);
            e = cudaStreamEndCapture(cs, &b->graph);
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&b->exec, b->graph, 0);
        cudaStreamDestroy(cs);
        if (e != cudaSuccess) {
            drop_graph(b);
            set_error("CUDA graph capture of the batched time loop failed: %s", cudaGetErrorString(e));
            return AWE_ERR_CUDA;
        }
    }
    CUDA_TRY(cudaGraphLaunch(b->exec, s));
    b->launches = b->tb2 ? (b->d.nt + b->tb2_shape.k - 1) / b->tb2_shape.k : b->d.nt;
    return AWE_OK;
}

extern "C" {

awe_status awe_batch_create(const awe_desc *desc, int nshots, const awe_shot *shots, int device, awe_batch **out) {
    if (!desc || !shots || !out || nshots <= 0) {
        set_error("null descriptor, shots or output, or no shots");
        return AWE_ERR_INVALID;
    }
    *out = nullptr;
    const awe_desc &d = *desc;
    if (d.scheme != AWE_SCHEME_CPU || d.coords != AWE_CART || d.ndim != 2) {
        set_error("awe_batch: 2D cartesian, scheme AWE_SCHEME_CPU only");
        return AWE_ERR_UNSUPPORTED;
    }
    if (d.hybrid || d.precision != AWE_FAST || d.jsnap > 0) {
        set_error("awe_batch: no hybrid ABC, no snapshots, AWE_FAST only");
        return AWE_ERR_UNSUPPORTED;
    }
    const int fdorder = d.fdorder ? d.fdorder : 4;
    if (fdorder < 2 || fdorder > 16 || fdorder % 2 || d.nt < 1 || d.dt <= 0 || d.n[0] < 1 || d.n[1] < 1 ||
        d.jdata < 1) {
        set_error("awe_batch: bad descriptor (fdorder 2..16 even, nt >= 1, dt > 0, jdata >= 1)");
        return AWE_ERR_INVALID;
    }
    for (int s = 0; s < nshots; s++) {
        const awe_shot &sh = shots[s];
        if (sh.x0 < 0 || sh.nx < 1 || sh.x0 + sh.nx > d.n[1] || sh.ns < 0 || sh.nr < 0 ||
            (sh.ns > 0 && !sh.sou) || (sh.nr > 0 && !sh.rec)) {
            set_error("awe_batch: shot %d: window [%d, %d) outside the model's %d columns or bad points", s, sh.x0,
                      sh.x0 + sh.nx, d.n[1]);
            return AWE_ERR_INVALID;
        }
    }
    if (cudaSetDevice(device) != cudaSuccess) {
        set_error("no CUDA device %d", device);
        return AWE_ERR_NODEVICE;
    }
    awe_batch *b = new awe_batch();
    b->d = d;
    b->d.fdorder = fdorder;
    b->device = device;
    b->nop = fdorder / 2;
    int nb = d.nb;
    if (nb < b->nop) nb = b->nop;  // MAWEFDcart2Dcpu.c:211
    b->nb = nb;
    b->n1 = d.n[0] + 2 * nb;
    if (b->n1 % 4) {
        delete b;
        set_error("awe_batch: nz + 2 nb must be a multiple of 4 (16-byte rows)");
        return AWE_ERR_UNSUPPORTED;
    }
    float dd[3] = {d.d[0], d.d[1], 1.f};
    fd_coefficients(b->nop, 2, dd, d.optfd, b->k);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, device);
    b->grid = 4 * std::max(b->sms, 1);
    b->shots_in.assign(shots, shots + nshots);
    cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);

    // layout: shot s occupies (nx_s + 2 nb) columns of n1 floats
    std::vector<float> w;
    if (d.dabc) sponge_weights(nb, w);
    auto table = [&](int n) {
        std::vector<float> t(n, 1.f);
        if (d.dabc)
            for (int i = 0; i < nb && i < n; i++) t[i] = t[n - 1 - i] = w[nb - i - 1];
        return t;
    };
    b->h_wz = table(b->n1);
    long long off = 0, doff = 0;
    b->nsmp = (d.nt - 1) / d.jdata + 1;
    std::vector<GeoPoint> hs, hr;
    for (int s = 0; s < nshots; s++) {
        const awe_shot &in = shots[s];
        BatchShot sh{};
        sh.off = off;
        sh.n2 = in.nx + 2 * nb;
        sh.wx_off = (int)b->h_wx.size();
        std::vector<float> tx = table(sh.n2);
        b->h_wx.insert(b->h_wx.end(), tx.begin(), tx.end());
        // the window's padded origin (fdutil_init on the cropped axes)
        const float oz = d.o[0] - nb * d.d[0], ox = d.o[1] + in.x0 * d.d[1] - nb * d.d[1];
        FdmAxes f{oz, ox, 0.f, d.d[0], d.d[1], 1.f, b->n1, sh.n2, 1};
        auto point = [&](const float *xz) {
            Lint l = lint_make(2, xz[0], 0.f, xz[1], f);
            GeoPoint g{};
            g.base = (long long)l.jx * b->n1 + l.jz;
            for (int c = 0; c < 4; c++) g.w[c] = l.w[c];
            return g;
        };
        sh.ns = in.ns;
        sh.src0 = (int)hs.size();
        for (int i = 0; i < in.ns; i++) hs.push_back(point(in.sou + 2 * i));
        sh.nr = in.nr;
        sh.rec0 = (int)hr.size();
        for (int i = 0; i < in.nr; i++) hr.push_back(point(in.rec + 2 * i));
        sh.dat_off = doff;
        doff += (long long)b->nsmp * in.nr;
        off += (long long)sh.n2 * b->n1;
        b->shots.push_back(sh);
    }
    b->cells = off;
    b->ndat = doff;
    b->h_rec = hr;
    b->h_src = hs;
    awe_status st = AWE_OK;
    const size_t cb = (size_t)off * sizeof(float);
    for (void **p : {(void **)&b->u[0], (void **)&b->u[1], (void **)&b->vel})
        if (st == AWE_OK) st = balloc(b, p, cb);
    if (st == AWE_OK) st = balloc(b, (void **)&b->wz, b->h_wz.size() * sizeof(float));
    if (st == AWE_OK) st = balloc(b, (void **)&b->wx, b->h_wx.size() * sizeof(float));
    if (st == AWE_OK) st = balloc(b, (void **)&b->wav, (size_t)d.nt * sizeof(float));
    if (st == AWE_OK) st = balloc(b, (void **)&b->dat, (size_t)std::max(doff, 1LL) * sizeof(float));
    if (st == AWE_OK) st = balloc(b, (void **)&b->d_shots, b->shots.size() * sizeof(BatchShot));
    if (st == AWE_OK) st = balloc(b, (void **)&b->src, std::max<size_t>(hs.size(), 1) * sizeof(GeoPoint));
    if (st == AWE_OK) st = balloc(b, (void **)&b->rec, std::max<size_t>(hr.size(), 1) * sizeof(GeoPoint));
    if (st == AWE_OK) st = balloc(b, (void **)&b->d_err, sizeof(int));
    if (st == AWE_OK && cudaMemset(b->d_err, 0, sizeof(int)) != cudaSuccess) st = AWE_ERR_CUDA;
    if (st == AWE_OK) {
        cudaMemcpy(b->wz, b->h_wz.data(), b->h_wz.size() * sizeof(float), cudaMemcpyHostToDevice);
        cudaMemcpy(b->wx, b->h_wx.data(), b->h_wx.size() * sizeof(float), cudaMemcpyHostToDevice);
        cudaMemcpy(b->d_shots, b->shots.data(), b->shots.size() * sizeof(BatchShot), cudaMemcpyHostToDevice);
        if (!hs.empty()) cudaMemcpy(b->src, hs.data(), hs.size() * sizeof(GeoPoint), cudaMemcpyHostToDevice);
        if (!hr.empty()) cudaMemcpy(b->rec, hr.data(), hr.size() * sizeof(GeoPoint), cudaMemcpyHostToDevice);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_error("batch upload failed: %s", cudaGetErrorString(e));
            st = AWE_ERR_CUDA;
        }
    }
    if (st == AWE_OK) st = set_tile(b, 0);
    if (st == AWE_OK) st = set_tb2(b);
    if (st != AWE_OK) {
        awe_batch_destroy(b);
        return st;
    }
    *out = b;
    return AWE_OK;
}

awe_status awe_batch_destroy(awe_batch *b) {
    if (!b) return AWE_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    drop_graph(b);
    for (auto &a : b->allocs) cudaFree(a.first);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return AWE_OK;
}

awe_status awe_batch_set_model(awe_batch *b, const float *vel) {
    if (!b || !vel) {
        set_error("null batch or model");
        return AWE_ERR_INVALID;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    const awe_desc &d = b->d;
    const int nz = d.n[0];
    std::vector<float> all((size_t)b->cells);
    const float dt2 = d.dt * d.dt;
    for (size_t s = 0; s < b->shots.size(); s++) {
        const awe_shot &in = b->shots_in[s];
        const BatchShot &sh = b->shots[s];
        // window, padded by edge replication (expand2d, fdutil.c:435-458), then v^2 dt^2
        const int n[2] = {nz, in.nx};
        expand_model(2, vel + (size_t)in.x0 * nz, all.data() + sh.off, b->nb, n);
        float *v = all.data() + sh.off;
        for (long long i = 0; i < (long long)sh.n2 * b->n1; i++) v[i] *= v[i] * dt2;  // MAWEFDcart2Dcpu.c:290
        if (d.fsrf)
            for (int x = 0; x < sh.n2; x++)
                for (int z = 0; z < b->nb + 1 && z < b->n1; z++) v[(size_t)x * b->n1 + z] = 0.f;  // :292-295
    }
    CUDA_TRY(cudaDeviceSynchronize());  // earlier runs (on any stream) may still read the old model
    CUDA_TRY(cudaMemcpy(b->vel, all.data(), all.size() * sizeof(float), cudaMemcpyHostToDevice));
    b->model_set = true;
    return AWE_OK;
}

awe_status awe_batch_forward_device(awe_batch *b, const float *d_wav, float *d_dat, void *stream) {
    if (!b || !d_wav || !d_dat) {
        set_error("null batch, wavelet or data pointer");
        return AWE_ERR_INVALID;
    }
    if (!b->model_set) {
        set_error("awe_batch_set_model must precede awe_batch_forward");
        return AWE_ERR_STATE;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    cudaStream_t s = stream ? (cudaStream_t)stream : b->stream;
    CUDA_TRY(cudaMemcpyAsync(b->wav, d_wav, (size_t)b->d.nt * sizeof(float), cudaMemcpyDeviceToDevice, s));
    awe_status st = run_all(b, s);
    if (st != AWE_OK) return st;
    CUDA_TRY(cudaMemcpyAsync(d_dat, b->dat, (size_t)b->ndat * sizeof(float), cudaMemcpyDeviceToDevice, s));
    return AWE_OK;
}

awe_status awe_batch_forward(awe_batch *b, const float *wav, float *dat) {
    if (!b || !wav || !dat) {
        set_error("null batch, wavelet or data pointer");
        return AWE_ERR_INVALID;
    }
    if (!b->model_set) {
        set_error("awe_batch_set_model must precede awe_batch_forward");
        return AWE_ERR_STATE;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    CUDA_TRY(cudaMemcpyAsync(b->wav, wav, (size_t)b->d.nt * sizeof(float), cudaMemcpyHostToDevice, b->stream));
    awe_status st = run_all(b, b->stream);
    if (st != AWE_OK) return st;
    CUDA_TRY(cudaMemcpyAsync(dat, b->dat, (size_t)b->ndat * sizeof(float), cudaMemcpyDeviceToHost, b->stream));
    CUDA_TRY(cudaStreamSynchronize(b->stream));
    int bad = 0;
    CUDA_TRY(cudaMemcpy(&bad, b->d_err, sizeof bad, cudaMemcpyDeviceToHost));
    if (bad) {
        set_error("awe_batch_forward: a bulk-copy wait of the column kernel timed out; results are invalid");
        return AWE_ERR_CUDA;
    }
    return AWE_OK;
}

awe_status awe_batch_tune(awe_batch *b, int steps, int *tile_out, int *grid_out) {
    if (!b || steps < 1) {
        set_error("null batch or steps < 1");
        return AWE_ERR_INVALID;
    }
    if (!b->model_set) {
        set_error("awe_batch_set_model must precede awe_batch_tune");
        return AWE_ERR_STATE;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    CUDA_TRY(cudaDeviceSynchronize());  // no earlier run (on any stream) still reads the items
    drop_graph(b);  // recaptured with the chosen kernel on the next forward
    steps = std::min(steps, b->d.nt);
    cudaEvent_t e0, e1;
    CUDA_TRY(cudaEventCreate(&e0));
    CUDA_TRY(cudaEventCreate(&e1));
    float best = 1e30f, tb2_ms = 1e30f;
    int best_tile = b->tile, best_grid = b->grid;
    const size_t bytes = (size_t)b->cells * sizeof(float);
    // (once: the time of a step does not depend on what the levels hold)
    CUDA_TRY(cudaMemsetAsync(b->u[0], 0, bytes, b->stream));
    CUDA_TRY(cudaMemsetAsync(b->u[1], 0, bytes, b->stream));
    b->colL = 0;
    if (b->tb2_ok) {
        const int n = std::min((steps + b->tb2_shape.k - 1) / b->tb2_shape.k * b->tb2_shape.k, b->d.nt);
        b->tb2 = true;
        launch_range(b, 0, std::min(n, b->tb2_shape.k), b->stream);  // warm
        cudaEventRecord(e0, b->stream);
        launch_range(b, 0, n, b->stream);
        cudaEventRecord(e1, b->stream);
        CUDA_TRY(cudaEventSynchronize(e1));
        cudaEventElapsedTime(&tb2_ms, e0, e1);
        tb2_ms *= (float)steps / n;
        b->tb2 = false;
    }
    for (int t = 0; t < kBatchNumTiles; t++) {
        awe_status st = set_tile(b, t);
        if (st != AWE_OK) return st;
        for (int mult : {2, 4, 8, 16}) {
            b->grid = mult * b->sms;
            launch_range(b, 0, 1, b->stream);  // warm
            cudaEventRecord(e0, b->stream);
            launch_range(b, 0, steps, b->stream);
            cudaEventRecord(e1, b->stream);
            CUDA_TRY(cudaEventSynchronize(e1));
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                best_tile = t;
                best_grid = b->grid;
            }
        }
    }
    // the column-march kernel: chunk lengths x (1, 2) persistent waves
    b->grid = best_grid;
    int best_col = 0, best_col_grid = 0;
    const int cpsm = batch2d_col_shape(b->nop, b->n1, nullptr) ? batch2d_col_ctas_per_sm(b->n1) : 0;
    // and the chunk length whose items take the fewest column times in whole
    // waves (L + 8 a chunk): 48 windows of 592 x 580 had 484 items of 64 columns
    // on 608 slots
    int Lw = 64;
    long long cols_best = -1;
    for (int L = 12; cpsm > 0 && L <= 128; L++) {
        long long items = 0;
        for (const BatchShot &sh : b->shots) items += (sh.n2 + L - 1) / L;
        const long long t = (items + (long long)cpsm * b->sms - 1) / ((long long)cpsm * b->sms) * (L + 8);
        if (cols_best < 0 || t < cols_best) cols_best = t, Lw = L;
    }
    std::vector<int> chunks = {16, 32, 64};
    if (Lw != 16 && Lw != 32 && Lw != 64) chunks.push_back(Lw);
    for (int L : chunks) {
        if (cpsm <= 0) break;
        awe_status st = set_columns(b, L);
        if (st != AWE_OK) return st;
        for (int mult : {1, 2}) {
            b->col_grid = mult * cpsm * b->sms;
            launch_range(b, 0, 1, b->stream);  // warm
            cudaEventRecord(e0, b->stream);
            launch_range(b, 0, steps, b->stream);
            cudaEventRecord(e1, b->stream);
            CUDA_TRY(cudaEventSynchronize(e1));
            float ms = 0;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                best_col = L;
                best_col_grid = b->col_grid;
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    b->colL = 0;
    if (best_col > 0) {
        awe_status st = set_columns(b, best_col);
        if (st != AWE_OK) return st;
        b->col_grid = best_col_grid;
    }
    b->tb2 = b->tb2_ok && tb2_ms < best;
    b->selected = false;
    int bad = 0;
    CUDA_TRY(cudaMemcpy(&bad, b->d_err, sizeof bad, cudaMemcpyDeviceToHost));
    if (bad) {
        set_error("awe_batch_tune: a bulk-copy wait of the column kernel timed out");
        return AWE_ERR_CUDA;
    }
    awe_status st = set_tile(b, best_tile);
    if (st != AWE_OK) return st;
    CUDA_TRY(cudaGetLastError());
    if (tile_out) *tile_out = b->tb2 ? kBatchNumTiles + 1 : b->colL > 0 ? kBatchNumTiles : best_tile;
    if (grid_out) *grid_out = b->tb2 ? b->tb2_tiles : b->colL > 0 ? b->col_grid : best_grid;
    return AWE_OK;
}

// receiver cells of every shot (cells the adjoint injects residuals into),
// each with its corners in (receiver, corner) order
static awe_status build_rec_cells(awe_batch *b) {
    std::vector<BatchRecCell> cells;
    std::vector<BatchRecW> ws;
    for (size_t s = 0; s < b->shots.size(); s++) {
        const BatchShot &sh = b->shots[s];
        std::map<long long, std::vector<BatchRecW>> per;
        for (int r = 0; r < sh.nr; r++) {
            const GeoPoint &g = b->h_rec[sh.rec0 + r];
            for (int c = 0; c < 4; c++) {
                const long long node = g.base + (c & 1) + (c >> 1) * (long long)b->n1;
                if (node < 0 || node >= (long long)sh.n2 * b->n1) continue;
                per[node].push_back(BatchRecW{r, g.w[c]});
            }
        }
        for (const auto &kv : per) {
            const int e0 = (int)ws.size();
            ws.insert(ws.end(), kv.second.begin(), kv.second.end());
            cells.push_back(BatchRecCell{sh.off + kv.first, (int)s, (int)(kv.first / b->n1), (int)(kv.first % b->n1),
                                         e0, (int)ws.size(), 0});
        }
    }
    bfree(b, b->rec_cells);
    bfree(b, b->rec_ws);
    awe_status st = balloc(b, (void **)&b->rec_cells, std::max<size_t>(cells.size(), 1) * sizeof(BatchRecCell));
    if (st == AWE_OK) st = balloc(b, (void **)&b->rec_ws, std::max<size_t>(ws.size(), 1) * sizeof(BatchRecW));
    if (st != AWE_OK) return st;
    if (!cells.empty()) {
        CUDA_TRY(cudaMemcpy(b->rec_cells, cells.data(), cells.size() * sizeof(BatchRecCell), cudaMemcpyHostToDevice));
        CUDA_TRY(cudaMemcpy(b->rec_ws, ws.data(), ws.size() * sizeof(BatchRecW), cudaMemcpyHostToDevice));
    }
    b->nrec_cells = (int)cells.size();
    return AWE_OK;
}

static awe_status grad_alloc(awe_batch *b, int T, int fmt) {
    const bool want = b->tb2_ok && !b->selected;
    if (b->gT == T && b->gfmt == fmt && (b->tb2_grad || b->tb2_tried || !want)) return AWE_OK;
    b->gT = 0;
    b->tb2_grad = b->tb2_tried = false;
    bfree(b, b->slots);
    bfree(b, b->ckpt);
    bfree(b, b->scales);
    const int nseg = (b->d.nt + T - 1) / T;
    const size_t es = fmt == AWE_CKPT_FP32 ? 4 : 2, cb = (size_t)b->cells * sizeof(float);
    const size_t nd = (size_t)std::max(b->ndat, 1LL);
    b->gscale_per = fmt == AWE_CKPT_BFP16 ? (b->cells + kBfpBlock - 1) / kBfpBlock : (long long)b->shots.size();
    const bool first = !b->win;
    const std::pair<void **, size_t> need[] = {
        {&b->ckpt, (size_t)2 * nseg * b->cells * es},
        {(void **)&b->scales, (size_t)2 * nseg * b->gscale_per * sizeof(float)},
        {(void **)&b->gX, cb},
        {(void **)&b->gY, cb},
        {(void **)&b->G, (size_t)b->cells * sizeof(float2)},
        {(void **)&b->res, nd * sizeof(float)},
        {(void **)&b->dobs, nd * sizeof(float)},
        {(void **)&b->part, ((nd + 1023) / 1024) * sizeof(double)},
        {(void **)&b->grad, (size_t)b->d.n[0] * b->d.n[1] * sizeof(double)},
        {(void **)&b->win, b->shots.size() * sizeof(int2)}};
    awe_status st = AWE_OK;
    for (const auto &q : need)
        if (st == AWE_OK && !*q.first) st = balloc(b, q.first, q.second);
    if (st != AWE_OK) return st;
    if (first) {
        std::vector<int2> w(b->shots.size());
        for (size_t s = 0; s < w.size(); s++) w[s] = make_int2(b->shots_in[s].x0, b->shots_in[s].nx);
        CUDA_TRY(cudaMemcpy(b->win, w.data(), w.size() * sizeof(int2), cudaMemcpyHostToDevice));
    }
    if (b->nrec_cells < 0) {
        st = build_rec_cells(b);
        if (st != AWE_OK) return st;
    }
    // several steps a launch: slots for both sweeps of a segment and two more
    // levels, where memory is left for them when all else is allocated.  Per step,
    // against the fastest one-step kernels (592 x 580 windows, 60 steps, 8th order):
    // 12 windows 76 us and 107, 24: 144 and 204, 48: 257 and 262, 128 (which
    // stream from HBM): 650 and 664; at 4th order 12: 61 and 97, 128: 516 and 880;
    // two windows of 220 x 200: 13 and 23
    if (b->tb2_ok && want) {
        b->tb2_tried = true;
        if (!b->tb2_adj.buf) {
            std::vector<Tb2Grid> grids = b->tb2_grids;
            for (Tb2Grid &g : grids) g.inj = g.rec, g.ninj = g.nrec, g.rec = nullptr, g.nrec = 0;
            Tb2HostLists h;
            if (tb2_host_lists(b->tb2_shape, grids, b->tb2_tiles, h)) {
                st = upload_lists(b, b->tb2_adj, h);
                if (st != AWE_OK && st != AWE_ERR_NOMEM) return st;
            }
        }
        b->tb2_grad = b->tb2_adj.buf && balloc_extra(b, (void **)&b->tb2_xy, 2 * cb) == AWE_OK &&
                      balloc_extra(b, (void **)&b->slots, (size_t)std::max(2 * T, T + 1) * cb) == AWE_OK;
        if (!b->tb2_grad) bfree(b, b->tb2_xy);
    }
    if (!b->tb2_grad) st = balloc(b, (void **)&b->slots, (size_t)(T + 1) * cb);
    if (st != AWE_OK) return st;
    b->gT = T;
    b->gfmt = fmt;
    b->gseg = nseg;
    return AWE_OK;
}

static BatchAdj adj_params(const awe_batch *b, int it, const float *V) {
    BatchAdj p{};
    p.V = V;
    p.vel = b->vel;
    p.G = b->G;
    p.wz = b->wz;
    p.wx = b->wx;
    p.sponge = b->d.dabc ? 1 : 0;
    p.n1 = b->n1;
    p.c0 = b->k.c0;
    for (int i = 0; i <= kMaxNop; i++) {
        p.cz[i] = b->k.c[0][i];
        p.cx[i] = b->k.c[1][i];
    }
    p.src = b->src;
    p.wav = b->wav;
    p.it = it;
    p.res = b->res;
    p.row = (it % b->d.jdata == 0) ? it / b->d.jdata : -1;
    return p;
}

// the whole gradient as one launch sequence on stream s (capturable)
static awe_status grad_sequence(awe_batch *b, cudaStream_t s) {
    const long long cells = b->cells;
    const size_t cb = (size_t)cells * sizeof(float);
    const int T = b->gT, ns = (int)b->shots.size();
    const bool tb2 = b->tb2_grad && !b->selected;
    const size_t es = b->gfmt == AWE_CKPT_FP32 ? 4 : 2;
    auto ck = [&](int idx) { return (void *)((char *)b->ckpt + (size_t)idx * cells * es); };
    auto sc = [&](int idx) { return b->scales + (size_t)idx * b->gscale_per; };
    // forward with checkpoints of both levels at every segment start
    CUDA_TRY(cudaMemsetAsync(b->d_err, 0, sizeof(int), s));
    CUDA_TRY(cudaMemsetAsync(b->u[0], 0, cb, s));
    CUDA_TRY(cudaMemsetAsync(b->u[1], 0, cb, s));
    auto store = [&](int it, float *prv, float *cur) {
        const int seg = it / T;
        launch_batch_ckpt(true, b->gfmt, b->d_shots, ns, prv, ck(2 * seg), sc(2 * seg), b->n1, cells, s);
        launch_batch_ckpt(true, b->gfmt, b->d_shots, ns, cur, ck(2 * seg + 1), sc(2 * seg + 1), b->n1, cells, s);
    };
    if (b->tb2) tb2_range(b, 0, b->d.nt, s, T, store);
    else
        for (int it = 0; it < b->d.nt; it++) {
            BatchStep p = step_params(b, it);
            if (it % T == 0) store(it, p.nxt, (float *)p.cur);
            launch_fwd(b, p, s, true);
        }
    launch_residual_flat(b->dat, b->dobs, b->res, b->ndat, b->part, s);
    // adjoint sweep, last segment first
    CUDA_TRY(cudaMemsetAsync(b->gX, 0, cb, s));
    CUDA_TRY(cudaMemsetAsync(b->gY, 0, cb, s));
    CUDA_TRY(cudaMemsetAsync(b->G, 0, (size_t)cells * sizeof(float2), s));
    float *X = b->gX, *Y = b->gY;
    float *X2 = b->tb2_xy, *Y2 = X2 + cells;  // (tb2)
    for (int seg = b->gseg - 1; seg >= 0; seg--) {
        const int k0 = seg * T, k1 = std::min(k0 + T, b->d.nt);
        if (tb2) {
            // both sweeps of the segment, several steps a launch, then its imaging condition at once
            const int K = b->tb2_shape.k;
            float *nu0 = b->slots + (size_t)T * cells;
            float *A = b->u[0], *B = b->u[1], *A2 = b->tb2_u, *B2 = b->tb2_u + cells;
            launch_batch_ckpt(false, b->gfmt, b->d_shots, ns, A, ck(2 * seg), sc(2 * seg), b->n1, cells, s);
            launch_batch_ckpt(false, b->gfmt, b->d_shots, ns, B, ck(2 * seg + 1), sc(2 * seg + 1), b->n1, cells, s);
            for (int k = k0; k < k1; k += K) {
                tb2_steps(b, false, A, B, A2, B2, b->slots + (size_t)(k - k0) * cells, k, std::min(K, k1 - k), false, s);
                std::swap(A, A2);
                std::swap(B, B2);
            }
            for (int k = k1 - 1; k >= k0;) {
                const int n = std::min(K, k - k0 + 1);
                tb2_steps(b, true, Y, X, Y2, X2, nu0 + (size_t)(k1 - 1 - k) * cells, k, n, false, s);
                std::swap(X, X2);
                std::swap(Y, Y2);
                k -= n;
            }
            launch_batch_image(b->G, b->slots, nu0, cells, b->d_shots, b->d_tb2_cols, b->tb2_ncols, b->n1, b->nop,
                               b->src, b->wav, k0, k1, s);
            continue;
        }
        launch_batch_ckpt(false, b->gfmt, b->d_shots, ns, b->slots, ck(2 * seg), sc(2 * seg), b->n1, cells, s);
        launch_batch_ckpt(false, b->gfmt, b->d_shots, ns, b->slots + cells, ck(2 * seg + 1), sc(2 * seg + 1), b->n1,
                          cells, s);
        for (int k = k0; k <= k1 - 2; k++) {
            const int j = k - k0;
            BatchStep p = step_params(b, k);
            p.prv = b->slots + (size_t)j * cells;
            p.cur = b->slots + (size_t)(j + 1) * cells;
            p.nxt = b->slots + (size_t)(j + 2) * cells;
            p.row = -1;
            launch_fwd(b, p, s, false);
        }
        for (int k = k1 - 1; k >= k0; k--) {
            BatchAdj p = adj_params(b, k, b->slots + (size_t)(k - k0 + 1) * cells);
            p.X = X;
            p.Y = Y;
            if (b->colL > 0 && b->col_adj_grid > 0)
                launch_batch2d_col_adj(b->d_shots, b->d_col_items, b->ncol_items, b->col_adj_grid, b->colL, p,
                                       b->d_err, s);
            else
                launch_batch2d_adj(b->nop, b->tile, b->d_shots, b->d_items, b->ntile_items, b->grid, p, s);
            launch_batch_rec_adj(b->rec_cells, b->nrec_cells, b->rec_ws, b->d_shots, p, s);
            std::swap(X, Y);
        }
    }
    launch_batch_grad_fold(b->d_shots, b->win, ns, b->G, b->vel, b->d.dt, b->n1, b->nb, b->d.n[0], b->d.n[1],
                           b->grad, s);
    return AWE_OK;
}

awe_status awe_batch_gradient(awe_batch *b, const float *wav, const float *dobs, const awe_grad_opts *opts,
                              double *grad, double *misfit) {
    if (!b || !wav || !dobs || !grad || !misfit) {
        set_error("null batch, wavelet, data, gradient or misfit pointer");
        return AWE_ERR_INVALID;
    }
    if (!b->model_set) {
        set_error("awe_batch_set_model must precede awe_batch_gradient");
        return AWE_ERR_STATE;
    }
    awe_grad_opts o{0, AWE_CKPT_BFP16};
    if (opts) o = *opts;
    if (o.ckpt_format != AWE_CKPT_BF16 && o.ckpt_format != AWE_CKPT_FP32 && o.ckpt_format != AWE_CKPT_FP16 &&
        o.ckpt_format != AWE_CKPT_BFP16) {
        set_error("awe_batch_gradient: unknown checkpoint format %d", o.ckpt_format);
        return AWE_ERR_INVALID;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    int T = o.ckpt_every > 0 ? o.ckpt_every : (int)std::ceil(std::sqrt((double)b->d.nt));
    T = std::max(1, std::min(T, b->d.nt));
    struct Use {
        awe_batch *b;
        explicit Use(awe_batch *q) : b(q) { b->grad_busy = true; }
        ~Use() { b->grad_busy = false; }
    } use(b);
    awe_status st = grad_alloc(b, T, o.ckpt_format);
    if (st == AWE_OK) {
        const int cpsm = b->colL > 0 ? batch2d_col_adj_ctas_per_sm(b->n1) : 0;
        b->col_adj_grid = cpsm > 0 ? cpsm * b->sms : 0;
    }
    if (st != AWE_OK) return st;
    cudaStream_t s = b->stream;
    CUDA_TRY(cudaMemcpyAsync(b->wav, wav, (size_t)b->d.nt * sizeof(float), cudaMemcpyHostToDevice, s));
    CUDA_TRY(cudaMemcpyAsync(b->dobs, dobs, (size_t)b->ndat * sizeof(float), cudaMemcpyHostToDevice, s));
    st = grad_sequence(b, s);
    if (st != AWE_OK) return st;
    const size_t nparts = (size_t)((b->ndat + 1023) / 1024);
    std::vector<double> parts(nparts);
    if (nparts) CUDA_TRY(cudaMemcpyAsync(parts.data(), b->part, nparts * sizeof(double), cudaMemcpyDeviceToHost, s));
    CUDA_TRY(cudaMemcpyAsync(grad, b->grad, (size_t)b->d.n[0] * b->d.n[1] * sizeof(double), cudaMemcpyDeviceToHost,
                             s));
    CUDA_TRY(cudaStreamSynchronize(s));
    CUDA_TRY(cudaGetLastError());
    int bad = 0;
    CUDA_TRY(cudaMemcpy(&bad, b->d_err, sizeof bad, cudaMemcpyDeviceToHost));
    if (bad) {
        set_error("awe_batch_gradient: a bulk-copy wait of the column kernel timed out; results are invalid");
        return AWE_ERR_CUDA;
    }
    double J = 0;
    for (double v : parts) J += 0.5 * v;
    *misfit = J;
    return AWE_OK;
}

awe_status awe_batch_select(awe_batch *b, int kernel, int chunk, int grid) {
    if (!b || kernel < 0 || kernel > kBatchNumTiles + 1) {
        set_error("awe_batch_select: kernel must be 0-%d", kBatchNumTiles + 1);
        return AWE_ERR_INVALID;
    }
    CUDA_TRY(cudaSetDevice(b->device));
    CUDA_TRY(cudaDeviceSynchronize());  // no earlier run (on any stream) still reads the items
    if (kernel == kBatchNumTiles + 1) {
        if (!b->tb2_ok) {
            set_error("awe_batch_select: several steps a launch need order 8 or less, no source in the sponge, no "
                      "point on a window's last line, few enough in a tile, and memory for two more levels");
            return AWE_ERR_UNSUPPORTED;
        }
        drop_graph(b);
        b->tb2 = true;
        b->selected = false;
        return AWE_OK;
    }
    drop_graph(b);
    if (kernel < kBatchNumTiles) {
        const awe_status st = set_tile(b, kernel);
        if (st != AWE_OK) return st;
        b->grid = grid > 0 ? grid : 4 * std::max(b->sms, 1);
        b->colL = 0;
        b->tb2 = false;
        b->selected = true;
        return AWE_OK;
    }
    if (chunk < 1 || !batch2d_col_shape(b->nop, b->n1, nullptr)) {
        set_error("awe_batch_select: the column march needs 8th order, nz + 2 nb <= 2048 and chunk >= 1");
        return AWE_ERR_UNSUPPORTED;
    }
    const int cpsm = batch2d_col_ctas_per_sm(b->n1);
    if (cpsm < 1) {
        set_error("awe_batch_select: the column march does not fit on this device");
        return AWE_ERR_UNSUPPORTED;
    }
    const awe_status st = set_columns(b, chunk);
    if (st != AWE_OK) return st;
    b->col_grid = grid > 0 ? grid : cpsm * b->sms;
    b->tb2 = false;
    b->selected = true;
    return AWE_OK;
}

awe_status awe_batch_info(const awe_batch *b, awe_batch_info_t *info) {
    if (!b || !info) {
        set_error("null argument");
        return AWE_ERR_INVALID;
    }
    info->nshots = (int)b->shots.size();
    info->nsmp = b->nsmp;
    info->total_samples = b->ndat;
    info->cells = b->cells;
    if (b->tb2) {
        info->tile_z = b->tb2_shape.tz;
        info->tile_x = b->tb2_shape.tx;
        info->grid = b->tb2_tiles;
        info->work_items = b->tb2_tiles;
    } else if (b->colL > 0) {  // column march: whole columns, chunks of colL
        info->tile_z = b->n1;
        info->tile_x = b->colL;
        info->grid = b->col_grid;
        info->work_items = (int)b->col_items.size();
    } else {
        info->tile_z = kBatchTiles[b->tile][0];
        info->tile_x = kBatchTiles[b->tile][1];
        info->grid = b->grid;
        info->work_items = (int)b->items.size();
    }
    info->launches_per_forward = b->tb2 ? (b->d.nt + b->tb2_shape.k - 1) / b->tb2_shape.k : b->d.nt;
    return AWE_OK;
}

}  // extern "C"
