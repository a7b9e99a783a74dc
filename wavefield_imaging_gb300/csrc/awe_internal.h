// Internal declarations shared by the engine's translation units.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "awe.h"

namespace awe {

constexpr int kMaxNop = 10;  // fdorder <= 20, as the reference's optfd tables

// Stencil coefficients, passed by value (kernel parameter space = constant bank).
struct Coef {
    float c0;                   // centre weight  (-2 * sum of all c)
    float c[3][kMaxNop + 1];    // second-derivative weights / d^2 per axis (1..nop)
    float b[3][kMaxNop + 1];    // first-derivative weights / d per axis (variable density)
};

// One interpolation point (source or receiver): flat index of the lowest
// corner and the 4 (2D) or 8 (3D) weights in the reference's corner order.
struct GeoPoint {
    long long base;
    float w[8];
};

// The cells a set of fixed sources injects into: entries [start[k], start[k+1])
// of `ent` are (source * 8 + corner, weight bits) of cell[k], in the reference's
// (source, corner) order, so one thread per cell adds what one thread walking
// every source would, in the same order.
struct InjCells {
    int n;  // cells; 0: none
    const long long *cell;
    const int *start;
    const int2 *ent;
};

// Padded grid, axis 1 fastest.  Lines are p1 >= n1 cells apart: a multiple of 4
// where a kernel's tensor maps or 16-byte accesses want it (the cells past n1
// hold nothing that is read), else n1.
struct Grid {
    int n1 = 0, n2 = 0, n3 = 0;  // n3 = 1 in 2D
    int p1 = 0;
    Grid() = default;
    Grid(int a, int b, int c, int p = 0) : n1(a), n2(b), n3(c), p1(p ? p : a) {}
    long long s2() const { return p1; }
    long long s3() const { return (long long)p1 * n2; }
    long long cells() const { return (long long)p1 * n2 * n3; }  // of storage
};

// ---- scheme of the reference CPU programs (MAWEFDcart{2D,3D}cpu.c) ----
struct StepBParams {
    Grid g;
    Coef k;
    int nop;
    const float *w1, *w2, *w3;  // per-axis sponge factor (1 where undamped); null = no sponge
    int damp_prev;              // prev level carries the sponge of the previous step
    int sponge_new;             // apply the sponge to the new level in the step kernel
    int shell;                  // cells within `shell` of a face are stored raw (boundary pass follows)
    int ilo[3], ihi[3];         // per axis, every sponge factor in [ilo, ihi) is exactly 1
    const float *prv;           // previous level when stepping out of place (null: read nxt in place)
    // 2D only, fused point work: sources added to the new level after its
    // update (k_injectB's arithmetic and order) ...
    const GeoPoint *inj;
    int inj_n, inj_stride, inj_ncs, inj_one, inj_it;
    const float *inj_wav;
    // ... and receivers gathered from `cur` (the level this launch reads,
    // pending sponge applied) by extra blocks after the cell blocks
    const GeoPoint *ext;
    int ext_n, ext_stride;
    float *ext_row;
    // polls allowed to a pipelined kernel's waits for its own copies before it
    // reports a timeout (< 0: the kernel's default); the drain after a timeout
    // always keeps the default
    long long spin;
};

// [lo, hi): the indices of a sponge factor table whose entries are exactly 1
// and that no entry != 1 lies between (the undamped interior of that axis)
void undamped_range(const std::vector<float> &w, int &lo, int &hi);

void launch_stepB(int ndim, int nop, bool exact, bool rho, const float *cur, float *nxt, const float *vel,
                  const float *den, const StepBParams &p, cudaStream_t s);

// ---- several 2D steps in one launch (k_tb2d.cu) ----
constexpr int kTb2Threads = 512, kTb2BatchThreads = 256;
constexpr size_t kTb2SmemMax = 200 * 1024;
// tile of tz x tx cells, k steps a launch, region of the tile and its halos
// (rz x rx; hz >= nop k a multiple of 4, hx = nop k), cx columns a thread
struct Tb2Shape {
    int k, tz, tx, hz, hx, rz, rx, ntz, ntx, cx;
};
// a tile of a batch: its window and its points in the lists (read at once, so
// that the loads of its cells are not behind a chain of small ones)
struct __align__(16) Tb2Tile {
    long long off, dat_off;  // first cell and first trace sample of the window
    int n2, wx_off, nr;      // its columns, first axis-2 sponge factor, receivers
    int z0, x0;              // first cell of the tile
    int rec0, nrec, cell0, ncell, ent0, nent, pad;
};
struct BatchShot;
struct Tb2Params {
    int n1, n2, k, it;
    int tz, tx, hz, hx, rz, rx;
    float c0, cz[5], cx[5];
    const float *cur, *prv, *vel;  // levels it, it - 1; v^2 dt^2
    float *ocur, *oprv;            // levels it + k, it + k - 1 (other buffers)
    // stored by step j at slots + j * slot_stride (null: nothing): L of the level
    // it reads, or (slot_level) that level; the adjoint step nu_k
    float *slots;
    long long slot_stride;
    int slot_level;
    const float *w1, *w2;            // sponge factors (null: no sponge; a batch: never null)
    int ilo1, ihi1, ilo2, ihi2;      // every factor in the range is 1
    // per tile: source cells of its region (z, x, first and last entry) with
    // their entries (source * 8 + corner, weight bits), and the receivers of its
    // cells (z, x, receiver) with their weights; the longest lists of a tile
    const int *inj_start, *ent_start, *rec_start;
    const int4 *inj_cell, *rec_pt;
    const int2 *inj_ent;
    const float *rec_wt;
    int max_rec, max_cell, max_ent;
    const float *wav;
    int ncs, jdata, nr;
    float *dat;
    const Tb2Tile *tiles;  // a batch: one block each (n2, nr, w2, wav of the adjoint and dat are per window)
};
// the lists of one grid's points (its tiles from tile0 on, ntx columns of them)
struct Tb2Grid {
    int n1, n2, ntx, tile0;
    const GeoPoint *inj;
    int ninj;
    const GeoPoint *rec;
    int nrec;
};
struct Tb2HostLists {
    std::vector<int> buf;
    size_t off[7];  // of Tb2Params' lists, in their order
    int most[3];    // max_rec, max_cell, max_ent
};
// false: points on a grid's last line, or more in a tile than fit
bool tb2_host_lists(const Tb2Shape &sh, const std::vector<Tb2Grid> &grids, int ntile, Tb2HostLists &out);
size_t tb2_smem(const Tb2Shape &sh, const int *most);
// points, lists and their sizes of a launch (buf: the lists on the device)
void tb2_set_lists(Tb2Params &q, const int *buf, const size_t *off, const int *most, bool inj, bool rec);
// the batch: ntile blocks; mode 0, 2 or 3, cx = 4
void launch_tb2_batch(int nop, int mode, const Tb2Params &p, const Tb2Shape &sh, int ntile, size_t smem,
                      cudaStream_t s);
// imaging condition of a segment of the batch (k_tb2_image); cols: (shot, first of 4 columns)
void launch_batch_image(float2 *G, const float *lap, const float *nu, long long stride, const BatchShot *shots,
                        const int2 *cols, int ncols, int n1, int nop, const GeoPoint *src, const float *wav, int k0,
                        int k1, cudaStream_t s);
// mode 0: AWE_FAST, 1: AWE_EXACT, 2: the adjoint step, 3: AWE_FAST with slots
void launch_tb2(int nop, int mode, const Tb2Params &p, const Tb2Shape &sh, size_t smem, cudaStream_t s);

struct AbcB {
    const float *zl, *zh;  // [n3][n2]
    const float *xl, *xh;  // [n3][n1]
    const float *yl, *yh;  // [n2][n1]
};
// w1 != null (3D): lines at least `band` from the axis-2/3 faces also get the
// sponge of their axis-1 ends in the axis-1 pass (when abc_zfused says the
// fused form applies); launch_band_sponge(..., zfused = 1) then skips them
void launch_abconeB(int ndim, int nop, bool exact, int fsrf, float *uo, const float *um, const AbcB &a,
                    const Grid &g, cudaStream_t s, const float *w1 = nullptr, const float *w2 = nullptr,
                    const float *w3 = nullptr, int band = 0);
bool abc_zfused(int nop, const Grid &g, int band);
void launch_hybridB(int ndim, int nop, int nbd, bool exact, int fsrf, float *uo, const float *um, const AbcB &a,
                    const float *damp, const Grid &g, cudaStream_t s);
void launch_band_sponge(int ndim, int width, bool exact, float *u, const float *w1, const float *w2,
                        const float *w3, const Grid &g, cudaStream_t s, int zfused = 0);

// Model preparation of the CPU-program scheme on the device (k_model.cu):
// padded v^2 dt^2 (free-surface rows zeroed) or a plain padded copy, and the
// one-way ABC coefficient tables, from the model as passed ([n3][n2][n1]).
struct ModelPrep {
    Grid g;                 // padded grid
    int n1, n2, n3, nb, nd;  // model size, padding, dimensions
    float dt, dt2, d1, d2, d3;
    int zero1;              // axis-1 samples set to 0 on every line (free surface), 0: none
};
void launch_model_pad(const float *raw, float *out, const ModelPrep &m, bool vel2, cudaStream_t s);
void launch_model_abc(const float *raw, const ModelPrep &m, float *const abc[6], cudaStream_t s);

// The boundary work of a 3D step in one launch (k_boundary3.cu): one-way ABC
// of the six faces, sponge of the shell the step kernel left unsponged
// (cells within nop + 2 of a face), the receiver gather of the level the step
// read, and the injection (ns > 0; only when no source corner lies on a cell
// that the launch's other blocks store: that shell, and the kBndEnd cells at
// each end of a line, which are loaded and stored together).
constexpr int kBndEnd = 8;
struct Bnd3Params {
    Grid g;
    float *uo;        // the new level
    const float *um;  // the level the step read
    const float *vel; // v^2 dt^2 (injection)
    const float *zl, *zh, *xl, *xh, *yl, *yh;  // one-way coefficients
    const float *w1, *w2, *w3;                 // sponge factors (null: no sponge)
    int top;                                   // axis-1 low face (0 with a free surface)
    const GeoPoint *rec;
    int nr, rec_stride;
    float *rec_row;  // null: no gather this step
    const GeoPoint *src;
    int ns, src_stride;
    InjCells inj;  // fixed sources by cell (n = 0: walk src)
    const float *wav;
    int it, ncs, one_wavelet;
    int n_int, nxr, nzr, end_blocks, rec_blocks;  // set by launch_bnd3
    int nop;                          // 1 .. 4
    // compact copies of the line ends ([n3][n2][16]: axis-1 cells 0..7, then
    // n1-8..n1-1) of um (em: written by the previous step's launch; null:
    // read um itself) and of the new level once final (eo; null: none)
    const float *em;
    float *eo;
};
bool bnd3_eligible(int nop, const Grid &g);
void launch_bnd3(bool exact, Bnd3Params p, cudaStream_t s);

// The boundary work before one adjoint step of the 3D gradient in one launch
// (k_boundary3.cu): mu += W kappa on the shell (kappa = 0), the transposed
// one-way ABC of the six faces (mu and kappa updated), and g = I vel2 mu on
// every cell.  nop = 4, bnd3_eligible.
struct Bnd3AdjParams {
    Grid g;
    float *mu, *kap, *gout;
    const float *vel2;
    const float *zl, *zh, *xl, *xh, *yl, *yh;
    const float *w1, *w2, *w3;  // sponge factors of the fold (null: weight 1)
    int top;                    // axis-1 low face (0 with a free surface)
    int n_int, nxr, nzr, end_blocks;  // set by launch_bnd3_adj
};
void launch_bnd3_adj(Bnd3AdjParams p, cudaStream_t s);

// injection into the new level scaled by vel (v^2 dt^2): u += (dd*w)*vel.
// off[c] = flat offset of corner c from the point's base index.
// stride: distance between consecutive points in pts (moving geometries)
void launch_injectB_off(int ndim, bool exact, float *u, const float *vel, const GeoPoint *pts, int ns,
                        const float *wav, int it, int ncs, bool one_wavelet, const long long *off, cudaStream_t s,
                        int stride = 1);

// the same from a cell list (fixed sources)
void launch_injectB_cells(bool exact, float *u, const float *vel, const InjCells &c, const float *wav, int it, int ncs,
                          bool one_wavelet, cudaStream_t s);

// receiver gather; when w1 != null the sponge factors are applied to each node
// value first (the field carries a pending sponge)
void launch_extract_off(int ndim, bool exact, const float *u, const GeoPoint *pts, int nr, float *dat_row,
                        const float *w1, const float *w2, const float *w3, const Grid &g, const long long *off,
                        cudaStream_t s, int stride = 1);

// copy a window (or the whole padded grid) of u into dst, applying pending sponge
void launch_snapshot(int ndim, const float *u, float *dst, const Grid &g, int f1, int f2, int f3, int m1, int m2,
                     int m3, const float *w1, const float *w2, const float *w3, cudaStream_t s);

// ---- scheme of the reference GPU programs (MAWEFD{cart,spher}{2D,3D}gpu.cu) ----
struct StepAParams {
    Grid g;
    int geom;        // 0 cart 2D, 1 cart 3D, 2 polar 2D, 3 spherical 3D
    int nd;          // 2 or 3
    int nb;          // sponge width
    int pri[3];      // sponge priority over memory axes (the kernel's x, y, z)
    int mask;        // 0 none, 1 cart 2D x band, 2 cart 3D z < nb, 3 r band (polar/spherical)
    int spill;       // samples of the next line zeroed by the free-surface grid rounding
    float dt2;
    float dd1, dd2, dd3, dd4, dd5;  // divisors of the Laplacian terms
    float rd[5];                    // their reciprocals (AWE_FAST)
    float a0;                       // polar centre weight -2/dra^2
    const float *tr0, *tr1, *tr2, *tr3;  // per-radius tables
    const float *tt0, *tt1;              // per-(theta, r) tables (spherical)
    const double *dtab;                  // sponge factor by index (FP64, as the reference)
    const float *ftab;                   // the same rounded to float (FAST mode)
    float b2lo, b2hi;                    // 2D one-way coefficients at the last sample
    const float *tb[6];                  // cart 3D one-way coefficient tables
    int nshot;                           // shots advanced together (spherical 3D, AWE_FAST), fields back to back
    long long shot_cells;                // cells of one shot's field
    int sms;                             // of the device
};
// out of place (the spherical AWE_FAST march kernels): prv the previous level, out the new one
void launch_stepA_oop(const float *cur, const float *prv, float *out, const float *vel,
                      const StepAParams &p, cudaStream_t s);
void launch_stepA(bool exact, const float *cur, float *nxt, const float *vel, const StepAParams &p, cudaStream_t s);
// 2D step in one launch (k_stepA2d.cu): out of place (cur, prv and nxt differ)
constexpr int kFusedCorners = 32;  // one bit per corner in the block's mask
struct StepA2Fused {
    // source corners whose injection is added when a level is read (inj_n = 0:
    // the levels hold it already), in (source, corner) order; none on the last
    // line that the one-way boundary reads
    int inj_n;
    int inj_i1[kFusedCorners], inj_i2[kFusedCorners];  // cell
    int inj_src[kFusedCorners];                        // source * 8 + corner
    float inj_w[kFusedCorners];
    const float *scale;
    int scaled;
    const float *wav;
    int it, ncs;
    // receivers gathered from cur (nr = 0: none)
    const GeoPoint *rec;
    int nr;
    float *rec_row;
};
void launch_stepA2(int geom, bool exact, const float *cur, const float *prv, float *nxt, const float *vel,
                   const StepAParams &p, const StepA2Fused &f, cudaStream_t s);
// cartesian 3D step in one launch (k_stepA3d.cu), the same for 3D
constexpr int kFusedCorners3 = 64;  // one bit per corner in the block's mask
struct StepA3Fused {
    int inj_n;
    int inj_i1[kFusedCorners3], inj_i2[kFusedCorners3], inj_i3[kFusedCorners3];
    int inj_src[kFusedCorners3];
    float inj_w[kFusedCorners3];
    const float *scale;
    int scaled;
    const float *wav;
    int it, ncs;
    const GeoPoint *rec;
    int nr;
    float *rec_row;
};
void launch_stepA3(bool exact, const float *cur, const float *prv, float *nxt, const float *vel, const StepAParams &p,
                   const StepA3Fused &f, cudaStream_t s);
// adjoint of the spherical step (AWE_FAST): Y <- W M (L^T(I c X) + 2 X - W Y),
// G += X L(A) on the interior (xcorr: G += X A; A null: none); receivers z += W M (w r)
void launch_adjA_sph(const float *X, float *Y, const float *A, const float *vel, float2 *G, const StepAParams &p,
                     cudaStream_t s, bool xcorr = false);
void launch_rec_adjA(float *z, const GeoPoint *pts, int nr, const float *r, const StepAParams &p, const long long *off,
                     cudaStream_t s);
// wav [nt][ncs]: ncs = 1 (one wavelet for every source) or ns
void launch_injectA(bool exact, int ndim, float *u, const GeoPoint *pts, const float *scale, int ns, const float *wav,
                    int it, bool scaled, const long long *off, cudaStream_t s, int stride = 1, int ncs = 1);
void launch_injectA_cells(bool exact, float *u, const float *scale, const InjCells &c, const float *wav, int it,
                          bool scaled, cudaStream_t s, int ncs);
void launch_snapshot_transpose2(const float *u, float *dst, const Grid &g, int f1, int f2, int m1, int m2,
                                cudaStream_t s);

// ---- adjoint of the CPU-program scheme (k_adjoint.cu) ----
struct AdjParams {
    Grid g;
    Coef k;
    int nd, nop;
    const float *w1, *w2, *w3;  // sponge axis factors; null = no sponge
    int xcorr;                  // imaging condition: G += I nu V (cross-correlation) instead of I nu L(V)
    // point terms fused into the step (null: none), per padded cell i the
    // entries [start[i], start[i + 1]) as (point index, weight bits):
    // receivers mu += W (W (w r[point])) with r = rrow; sources G += nu (wav w)
    const int *rc_start, *sc_start;
    const int2 *rc_ent, *sc_ent;
    const float *rrow;     // this step's residual row (null: no receiver term this step)
    const float *wav;      // wavelet (null: no source term)
    int it, ncs, one_wavelet;
};
void launch_adjB(const float *X, float *Y, const float *V, const float *vel, float2 *G, const AdjParams &p,
                 cudaStream_t s);
void launch_tb2_image(float2 *G, const float *lap, const float *nu, long long stride, const AdjParams &p, int k0,
                      int k1, cudaStream_t s);
void launch_abc_adjB(int nop, int fsrf, float *mu, float *kap, const AbcB &a, const Grid &g, cudaStream_t s);
void launch_kap_fold(float *mu, float *kap, const AdjParams &p, cudaStream_t s);
// receiver residuals into mu and the source term of the gradient (c.n = 0: none)
void launch_points_adj(float *mu, const GeoPoint *pts, int nr, const float *r, const AdjParams &p, const long long *off,
                       float2 *G, const float *nu, const InjCells &c, const float *wav, int it, int ncs,
                       bool one_wavelet, cudaStream_t s);
void launch_residual(const float *d, const float *dobs, float *r, int nrows, int nr, double *row_sum, cudaStream_t s);
// n1, p1: checkpoints hold the n cells of the levels' lines without their padding
void launch_ckpt_store16(bool fp16, const float *u, long long n, unsigned int *amax, void *q, float *scale, int grid,
                         cudaStream_t s, int n1 = 1, int p1 = 1);
void launch_ckpt_load16(bool fp16, const void *q, long long n, const float *scale, float *u, int grid,
                        cudaStream_t s, int n1 = 1, int p1 = 1);
// block floating point checkpoints: kBfpBlock consecutive cells share one FP32 scale
constexpr int kBfpBlock = 64;
constexpr float kBfpTiny = 1e-30f;  // blocks with max |v| <= this are stored as zero
void launch_ckpt_store_bfp(const float *u, long long n, short *q, float *scale, int grid, cudaStream_t s, int n1 = 1,
                           int p1 = 1);
void launch_ckpt_load_bfp(const short *q, const float *scale, long long n, float *u, int grid, cudaStream_t s,
                          int n1 = 1, int p1 = 1);
// image on the model grid: the padded grid's model window of G
void launch_add_f64(double *dst, const double *src, long long n, cudaStream_t s);
void launch_image_cut(const float2 *G, const Grid &g, int nb, const int *n, int nd, double *out, cudaStream_t s);
// vel2: v^2 dt^2 per padded cell, or the velocity itself (raw_v: c = dt^2 v^2);
// zero1: samples of every line that a free surface sets to 0
void launch_grad_fold(const float2 *G, const float *vel2, float dt, const Grid &g, int nb, const int *n, int nd,
                      double *out, cudaStream_t s, bool raw_v = false, int zero1 = 0);

// ---- batched 2D forward (k_batch2d.cu) ----
struct BatchShot {
    long long off;      // first cell of the shot's padded grid in the concatenated fields
    int n2;             // padded columns
    int wx_off;         // first entry of its axis-2 sponge table
    int ns, src0;       // sources: count, first index in the point table
    int nr, rec0;       // receivers
    long long dat_off;  // first sample of its traces [nsmp][nr]
};
struct BatchStep {
    const float *cur;
    float *nxt;
    const float *vel;
    const float *wz, *wx;  // sponge tables (axis 1 common, axis 2 per shot)
    int sponge;
    int n1;  // padded rows (axis 1), common
    float c0, cz[kMaxNop + 1], cx[kMaxNop + 1];
    const GeoPoint *src, *rec;
    const float *wav;  // one wavelet, [nt]
    int it;
    float *dat;
    int row;            // trace row written by this step, -1: none
    const float *prv;   // previous level when stepping out of place (null: in place in nxt)
};
// a padded cell that receivers inject adjoint residuals into, with its
// receiver corners [e0, e1) in (receiver, corner) order
struct BatchRecCell {
    long long gi;  // cell of the concatenated padded grids
    int shot, x, z, e0, e1, pad;
};
struct BatchRecW {
    int r;    // receiver index within the shot
    float w;  // interpolation weight
};
struct BatchAdj {
    const float *X;  // nu_k
    float *Y;        // nu_{k+1} in, mu_k out
    const float *V;  // forward level V_k
    const float *vel;
    float2 *G;  // dJ/dvel2 accumulators (compensated pairs), per shot, padded grids
    const float *wz, *wx;
    int sponge, n1;
    float c0, cz[kMaxNop + 1], cx[kMaxNop + 1];
    const GeoPoint *src;
    const float *wav;
    int it;
    const float *res;  // residuals, laid out as the traces
    int row;           // residual row of this step, -1: none
};
void launch_batch2d_adj(int nop, int tile, const BatchShot *shots, const int4 *items, int nitems, int grid,
                        const BatchAdj &p, cudaStream_t s);
void launch_batch_ckpt(bool store, int fmt, const BatchShot *shots, int nshots, float *u, void *q, float *scales,
                       int n1, long long cells, cudaStream_t s);
void launch_residual_flat(const float *d, const float *dobs, float *r, long long n, double *part, cudaStream_t s);
void launch_batch_grad_fold(const BatchShot *shots, const int2 *win, int nshots, const float2 *G, const float *vel2,
                            float dt, int n1, int nb, int nz, int nxm, double *out, cudaStream_t s);
// column-march forward (k_batch2d_col.cu): 8th order, n1 % 4 == 0, n1 <= 2048;
// returns the threads per CTA (0 if the shape is not covered) and the dynamic shared memory
int batch2d_col_shape(int nop, int n1, size_t *smem);
int batch2d_col_ctas_per_sm(int n1);
void launch_batch2d_col(const BatchShot *shots, const int4 *items, int nitems, int grid, int L, const BatchStep &p,
                        int *err, cudaStream_t s);
// adjoint step as a column march (same arithmetic as k_batch2d_adj)
int batch2d_col_adj_ctas_per_sm(int n1);
void launch_batch2d_col_adj(const BatchShot *shots, const int4 *items, int nitems, int grid, int L,
                            const BatchAdj &p, int *err, cudaStream_t s);
// the adjoint step's receiver term W R^T r on mu (p.Y), after either adjoint
// kernel: one thread per receiver cell, its corners in order
void launch_batch_rec_adj(const BatchRecCell *cells, int ncells, const BatchRecW *ws, const BatchShot *shots,
                          const BatchAdj &p, cudaStream_t s);
constexpr int kBatchNumTiles = 4;
constexpr int kBatchRecBlock = 128;  // receivers per receiver item (<= threads of every tile shape)
extern const int kBatchTiles[kBatchNumTiles][2];
void launch_batch2d(int nop, int tile, const BatchShot *shots, const int4 *items, int nitems, int grid,
                    const BatchStep &p, cudaStream_t s);

// ---- host-side math (bit-identical to the reference's float evaluation) ----
void fd_coefficients(int nop, int ndim, const float *dd, int optfd, Coef &k);
void sponge_weights(int nb, std::vector<float> &w);   // fdutil.c sponge_make
void hybrid_damp(int ntransit, std::vector<float> &w);  // MAWEFDcart*cpu.c damp_make
// fdutil.c lint2d_make / lint3d_make for one point, in the reference's fdm
// axes (z, x, y): origin of the padded grid, spacing, padded size.
struct FdmAxes {
    float oz, ox, oy, dz, dx, dy;
    int nz, nx, ny;
};
struct Lint {
    int jz, jx, jy;
    float w[8];
};
Lint lint_make(int ndim, float x, float y, float z, const FdmAxes &f);
void expand_model(int ndim, const float *a, float *b, int nb, const int *n);

void set_error(const char *fmt, ...);
// the descriptor checks of awe_plan_create (sizes, spacing, time axis,
// scheme, order, intervals, precision)
awe_status check_desc(const awe_desc *d);

// ---- TMA-staged 3D 8th-order step (k_stepB3_tma.cu) ----
struct Step3Launch {
    int grid, L, ntz, ntx, nchunks, items;
    size_t smem;
};
bool stepB3_tma_eligible(int ndim, int nop, bool rho, const Grid &g);
// (orders 2 to 8; g.p1 a multiple of 4)
bool stepB3_tma_maps(CUtensorMap *maps, float *const u[2], const float *vel, const Grid &g, int nop);
int march_planes(int n3, long long columns, int slots, int halo);
Step3Launch stepB3_tma_shape(const Grid &g, int num_sms, int L, int nop = 4);
// lap_out (AWE_FAST only, may be null): also store L(cur) of interior cells
cudaError_t launch_stepB3_tma_with(bool exact, const CUtensorMap &cur, const CUtensorMap &prv, const CUtensorMap &vel,
                                   float *nxt, const StepBParams &sp, const Step3Launch &sh,
                                   unsigned long long *counter, unsigned long long base, int *err, cudaStream_t s,
                                   float *lap_out);
cudaError_t launch_stepB3_adj(const CUtensorMap &g_halo, const CUtensorMap &y_tile, const CUtensorMap &x_tile,
                              float *Y, const float *lap_v, float2 *grad, const StepBParams &sp,
                              const Step3Launch &sh, unsigned long long *counter, unsigned long long base, int *err,
                              cudaStream_t s);
// g = I vel2 nu (cells at least nop from every face), elementwise
void launch_adj_g(const float *nu, const float *vel2, float *g, const Grid &gr, int nop, cudaStream_t s);
// p1: cells from line to line (0: n1)
bool make_tmap_3d(CUtensorMap *m, const float *base, int n1, int n2, int n3, int b1, int b2, int p1 = 0);
// tensor-map boxes of the TMA step: the current level's halo box and the tile box
void stepB3_tma_boxes(int *halo1, int *halo2, int *tile1, int *tile2);

// TMA-staged spherical step (GPU-program scheme, AWE_FAST); Step3Launch's
// ntz/ntx count the r and theta tiles, items include the shots
bool sphA_tma_eligible(const Grid &g, int nb);
// maps: [0] u[0] halo box, [1] u[1] halo box, [2] u[0] tile, [3] u[1] tile, [4] vel tile
bool sphA_tma_maps(CUtensorMap *maps, float *const u[2], const float *vel, const Grid &g, int nshot);
Step3Launch sphA_tma_shape(const Grid &g, int nshot, int num_sms, int L);
// cur_f0, prv_f0: plane offsets of the two levels in their maps (levels
// stacked along phi, as the gradient's recompute slots); nxt: the new level
cudaError_t launch_stepA_sph_tma(const CUtensorMap &cur, const CUtensorMap &prv, const CUtensorMap &vel, float *nxt,
                                 const StepAParams &pa, const Step3Launch &sh, unsigned long long *counter,
                                 unsigned long long base, int *err, long long spin, cudaStream_t s, int cur_f0 = 0,
                                 int prv_f0 = 0);
// adjoint step of the spherical scheme (the k_adjA_sph2 update, TMA-staged):
// x_halo / v_halo / a_halo = 72 x 18 box maps of z_{j+1}, the velocity and the
// forward levels (A_j at plane offset a_f0); y_tile / g_tile = tile maps of
// Y (z_{j+2} in, z_j out) and of G (the gradient or image accumulators,
// sphA_tma_pair_map)
// halo-box (72 x 18) and, when tile is not null, tile-box (64 x 16) maps of
// nlevels fields stacked along phi from base
bool sphA_tma_level_maps(CUtensorMap *halo, CUtensorMap *tile, const float *base, const Grid &g, int nlevels);
bool sphA_tma_pair_map(CUtensorMap *m, const float2 *base, const Grid &g);
cudaError_t launch_adjA_sph_tma(const CUtensorMap &x_halo, const CUtensorMap &v_halo, const CUtensorMap &a_halo,
                                int a_f0, const CUtensorMap &y_tile, const CUtensorMap &g_tile, float *Y, float2 *G,
                                const StepAParams &pa, const Step3Launch &sh, unsigned long long *counter,
                                unsigned long long base, int *err, long long spin, bool xcorr, cudaStream_t s);

}  // namespace awe
