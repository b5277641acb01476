// extern "C" boundary of the cs2d library: validation, launch geometry, errors.
// Mirrors the checks of the reference host binding
// (src/cusoflex/selective_scan_oflex.cpp:188-245 and :298-391) on raw pointers.
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <initializer_list>

#include "cs2d_blk.cuh"
#include "cs2d_pair.cuh"
#include "cs2d_common.cuh"

namespace cs2d {
cudaError_t launch_fwd(const Dev &P, int L, int grid, cudaStream_t st);
cudaError_t launch_bwd(const Dev &P, int L, int grid, cudaStream_t st);
cudaError_t launch_fwd_serial(const Dev &P, int L, int grid, cudaStream_t st);   // one CTA walks all groups of its tile
cudaError_t launch_bwd_serial(const Dev &P, int L, int grid, cudaStream_t st);
cudaError_t launch_stream_fwd(const Dev &P, int L, int grid, cudaStream_t st);
cudaError_t launch_stream_bwd(const Dev &P, int L, int grid, cudaStream_t st);
int stream_pairs_per_cta(int L);
cudaError_t launch_walk_fwd(const Dev &P, int grid, cudaStream_t st);
cudaError_t launch_blk_fwd(const Blk &P, int NG, cudaStream_t st);
cudaError_t launch_blk_bwd(const Blk &P, int NG, cudaStream_t st);
cudaError_t launch_pair_fwd(const Pw &P, bool keep, cudaStream_t st);
cudaError_t launch_pair_bwd(const Pw &P, cudaStream_t st);
void walk_geometry(int ncols, int *swd, int *lr);
int walk_channels_per_cta(int lr);
size_t walk_bc_bytes(int batch, int groups, int nrows, int ncols);
size_t fwd_smem_bytes(int L, int CG, int NPp, int W, int es, bool bulk, int CT, bool tiled, bool ws);
size_t bwd_smem_bytes(int L, int CG, int NPp, int CT, bool acc, int W, int es, int eso, bool bulk, bool tiled, bool ws);
static __device__ int g_cs2d_status = 0;  // see ERR_* in cs2d_status.h

// Device address of the status word on the current device (looked up once per device).
static int *status_ptr() {
    static int *ptr[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!ptr[dev] && cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr[dev]), g_cs2d_status) != cudaSuccess)
        ptr[dev] = nullptr;
    return ptr[dev];
}

static thread_local char g_err[512] = "";
static std::atomic<int64_t> g_launches{0};

__attribute__((format(printf, 2, 3))) static int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

struct Geometry { int L, NPp, CG, CP, CT, npass, ntiles, grid, nck, acc, bulk, ws; };

static const size_t kMaxSmem = 227 * 1024;   // largest dynamic shared memory of one CTA
static const size_t kSmSmem = 228 * 1024;    // shared memory of one SM; every resident CTA also reserves 1 KB
static const size_t kCtaReserve = 1024;
static const int kSMs = 148;

// Lanes per row, state-pair slots, channels per pass and per CTA, and the grid.
// serial: the CTAs walk all groups of their channel tile one after the other (direction merge), so the
// grid has no group dimension.
static int plan(const cs2d_problem *p, bool backward, bool bulk_ok, bool tiled, Geometry *g, bool serial = false) {
    const int W = p->ncols, es = p->io_dtype == CS2D_F32 ? 4 : 2, eso = p->out_dtype == CS2D_F32 ? 4 : 2;
    const int strips = (p->ncols + STRIP - 1) / STRIP;
    int L = 1;
    while (L < strips) L <<= 1;
    if (L > 32) return fail(CS2D_ERR_INVALID, "internal: a column tile of %d columns", p->ncols);
    const int NP = (p->dstate + 1) / 2;
    int NPp = 1;
    while (NPp < NP) NPp <<= 1;
    const int dpg = p->dim / p->n_groups;
    // Channel groups per pass: fill the CTA up to 8 warps, but keep the staged
    // per-channel tiles small enough that the shared memory fits.
    int CG = MAX_WARPS / NPp;
    while (CG > 1 && (backward ? bwd_smem_bytes(L, CG, NPp, CG * (32 / L), false, W, es, eso, false, tiled, false) > kMaxSmem
                               : 2 * (fwd_smem_bytes(L, CG, NPp, W, es, false, CG * (32 / L), tiled, false) + kCtaReserve) > kSmSmem))
        CG >>= 1;
    const int CP = CG * (32 / L);
    const int pmax = (dpg + CP - 1) / CP;  // passes that cover a whole group
    // Channels per CTA (1..8 passes): B/C staging and the dB/dC atomics are paid once per CTA,
    // but the grid has to fill whole waves (5.2 waves waste 14% of the machine in the last one).
    const int slots = kSMs * (backward ? 1 : 2);
    // Cost model: a CTA pays the B/C staging of a row block once (about one pass worth of
    // work when a warp holds a single channel, 1/CW of it otherwise) plus np passes, and the
    // launch takes waves(np) rounds of CTAs.
    int npass = 1;
    double best = 1e300;
    const double stage = 1.0 / (32 / L);
    for (int np = 1; np <= (pmax < 8 ? pmax : 8); ++np) {
        const int64_t chunks = (dpg + np * CP - 1) / (np * CP);
        const int64_t grid = (int64_t)p->batch * (serial ? 1 : p->n_groups) * chunks;
        const int64_t waves = (grid + slots - 1) / slots;
        const double cost = (double)waves * (stage + np);
        if (cost < best - 1e-9) { best = cost; npass = np; }
    }
    g->acc = 1;
    g->ws = 0;
    g->bulk = bulk_ok ? 1 : 0;
    if (backward) {
        // drop, in this order, the bulk staging buffers, then the dB/dC accumulators, then passes
        if (bwd_smem_bytes(L, CG, NPp, npass * CP, true, W, es, eso, g->bulk, tiled, false) > kMaxSmem) g->bulk = 0;
        if (bwd_smem_bytes(L, CG, NPp, npass * CP, true, W, es, eso, false, tiled, false) > kMaxSmem) g->acc = 0;
        while (npass > 1 && bwd_smem_bytes(L, CG, NPp, npass * CP, g->acc, W, es, eso, false, tiled, false) > kMaxSmem) --npass;
        if (bwd_smem_bytes(L, CG, NPp, npass * CP, g->acc, W, es, eso, false, tiled, false) > kMaxSmem)
            return fail(CS2D_ERR_UNSUPPORTED, "ncols=%d with dstate=%d needs more shared memory than one SM has",
                        p->ncols, p->dstate);
        // The common geometry (8 state-pair slots, one channel group, one column tile) runs
        // warp-specialised when the second tile set fits: staging warps replace the bulk copies.
        if (NPp == 8 && CG == 1 &&
            bwd_smem_bytes(L, CG, NPp, npass * CP, g->acc, W, es, eso, false, tiled, true) <= kMaxSmem) {
            g->ws = 1;
            g->bulk = 0;
        }
    } else {
        // keep two CTAs per SM
        if (2 * (fwd_smem_bytes(L, CG, NPp, W, es, g->bulk, npass * CP, tiled, false) + kCtaReserve) > kSmSmem) g->bulk = 0;
        if (fwd_smem_bytes(L, CG, NPp, W, es, false, npass * CP, tiled, false) > kMaxSmem)
            return fail(CS2D_ERR_UNSUPPORTED, "ncols=%d with dstate=%d needs more shared memory than one SM has",
                        p->ncols, p->dstate);
        // warp-specialised like the backward, as long as two CTAs still share an SM
        if (NPp == 8 && CG == 1 &&
            2 * (fwd_smem_bytes(L, CG, NPp, W, es, false, npass * CP, tiled, true) + kCtaReserve) <= kSmSmem) {
            g->ws = 1;
            g->bulk = 0;
        }
    }
    g->L = L; g->NPp = NPp; g->CG = CG; g->CP = CP; g->npass = npass; g->CT = npass * CP;
    g->ntiles = (dpg + g->CT - 1) / g->CT;
    g->grid = p->batch * (serial ? 1 : p->n_groups) * g->ntiles;
    g->nck = (p->nrows + RB - 1) / RB;
    return CS2D_OK;
}

static int validate(const cs2d_problem *p) {
    if (!p) return fail(CS2D_ERR_INVALID, "problem is NULL");
    if (p->batch <= 0 || p->dim <= 0 || p->nrows <= 0 || p->ncols <= 0 || p->dstate <= 0 || p->n_groups <= 0 ||
        p->delta_dim <= 0)
        return fail(CS2D_ERR_INVALID, "all sizes must be positive");
    if (p->io_dtype < CS2D_F32 || p->io_dtype > CS2D_BF16)
        return fail(CS2D_ERR_INVALID, "input type must be float32, float16 or bfloat16");
    if (p->out_dtype != p->io_dtype && p->out_dtype != CS2D_F32)
        return fail(CS2D_ERR_INVALID, "out/dout type must equal the input type or be float32");
    if (p->dim % p->n_groups) return fail(CS2D_ERR_INVALID, "dims should be dividable by n_groups");
    if (p->dim % p->delta_dim) return fail(CS2D_ERR_INVALID, "dims should be dividable by delta_dim");
    if (p->dstate > CS2D_MAX_DSTATE)
        return fail(CS2D_ERR_INVALID, "selective_scan only supports state dimension <= %d", CS2D_MAX_DSTATE);
    if (!p->u || !p->delta || !p->A || !p->B || !p->C) return fail(CS2D_ERR_INVALID, "u, delta, A, B, C must be given");
    return CS2D_OK;
}

// A tensor may be accessed four elements at a time when its base address is
// aligned to four elements and every stride that separates rows is a multiple
// of four (rows then start aligned whenever ncols is a multiple of four).
static bool vec_ok(const void *ptr, int esize, int ncols, std::initializer_list<int64_t> strides) {
    if (ncols % 4) return false;
    if (reinterpret_cast<uintptr_t>(ptr) % (4 * esize)) return false;
    for (int64_t s : strides)
        if (s % 4) return false;
    return true;
}
static int esize(int dt) { return dt == CS2D_F32 ? 4 : 2; }
// the same for aligned 4-byte words: every fp32 element, or pairs of 16-bit elements of even-width rows
static bool word_ok(const void *ptr, int esize, int ncols, std::initializer_list<int64_t> strides) {
    const int ew = 4 / esize;   // elements per word
    if (ncols % ew) return false;
    if (reinterpret_cast<uintptr_t>(ptr) % 4) return false;
    for (int64_t s : strides)
        if (s % ew) return false;
    return true;
}
// the same for 8 elements at a time (the streaming kernels' one-word strips of 16-bit types)
static bool vec8_ok(const void *ptr, int esize, int ncols, std::initializer_list<int64_t> strides) {
    if (ncols % 8) return false;
    if (reinterpret_cast<uintptr_t>(ptr) % (8 * esize)) return false;
    for (int64_t s : strides)
        if (s % 8) return false;
    return true;
}

// A (batch, channel, nrows, ncols) tensor can be fetched with bulk copies of whole
// row blocks when its rows are 16-byte multiples, rows of a plane are contiguous,
// and the base address and the plane/batch strides are 16-byte multiples.
static bool bulk_ok1(const void *ptr, int es, int ncols, int64_t bs, int64_t ds, int64_t hs) {
    return ptr && (ncols * es) % 16 == 0 && hs == ncols && reinterpret_cast<uintptr_t>(ptr) % 16 == 0 &&
           (bs * es) % 16 == 0 && (ds * es) % 16 == 0;
}

static void fill(Dev &d, const cs2d_problem *p, const Geometry &g) {
    d.batch = p->batch; d.dim = p->dim; d.H = p->nrows; d.W = p->ncols; d.N = p->dstate; d.G = p->n_groups;
    d.ddim = p->delta_dim; d.io_dt = p->io_dtype; d.out_dt = p->out_dtype; d.softplus = p->delta_softplus;
    d.dpg = p->dim / p->n_groups; d.drep = p->dim / p->delta_dim;
    d.acc_dbc = g.acc; d.bulk = g.bulk; d.ws = g.ws; d.NPp = g.NPp; d.CG = g.CG; d.CT = g.CT; d.npass = g.npass; d.ntiles = g.ntiles; d.nck = g.nck;
    d.u = p->u; d.delta = p->delta; d.B = p->B; d.C = p->C; d.A = p->A; d.D = p->D; d.bias = p->delta_bias;
    d.decay = p->A_decay;
    d.u_bs = p->u_bs; d.u_ds = p->u_ds; d.u_hs = p->u_hs;
    d.dl_bs = p->delta_bs; d.dl_ds = p->delta_ds; d.dl_hs = p->delta_hs;
    d.A_ds = p->A_ds; d.A_ns = p->A_ns;
    d.B_bs = p->B_bs; d.B_gs = p->B_gs; d.B_ns = p->B_ns; d.B_hs = p->B_hs;
    d.C_bs = p->C_bs; d.C_gs = p->C_gs; d.C_ns = p->C_ns; d.C_hs = p->C_hs;
    const int es = esize(p->io_dtype);
    d.vec = 0; d.vec8 = 0; d.vec2 = 0;
    if (vec_ok(p->u, es, p->ncols, {p->u_bs, p->u_ds, p->u_hs})) d.vec |= VEC_U;
    if (vec_ok(p->delta, es, p->ncols, {p->delta_bs, p->delta_ds, p->delta_hs})) d.vec |= VEC_DELTA;
    if (vec_ok(p->B, es, p->ncols, {p->B_bs, p->B_gs, p->B_ns, p->B_hs})) d.vec |= VEC_B;
    if (vec_ok(p->C, es, p->ncols, {p->C_bs, p->C_gs, p->C_ns, p->C_hs})) d.vec |= VEC_C;
    d.adj = nullptr;
    d.det = 0; d.det_ts = 0;
    d.mw = nullptr; d.dw = nullptr;
    d.cshift = 0;
    d.ck_roll = 0;
    d.ck_pairs = 0;
    d.ck_wp = g.L * STRIP;
    d.wbt = nullptr; d.wct = nullptr;
    d.dir_serial = 0; d.merge_store = 0;
    d.status = nullptr;
    d.tile_left = d.tile_right = 0; d.Wout = p->ncols;
    d.flip_h = d.flip_w = 0; d.u_shared = 0;
    d.edge_in = nullptr; d.edge_out = nullptr; d.adj_in = nullptr; d.adj_out = nullptr;
    d.du = d.ddelta = nullptr; d.dA = d.dB = d.dC = d.dD = d.dbias = d.ddecay = nullptr;
}
}  // namespace cs2d

using namespace cs2d;

extern "C" {

// ---- column tiles ------------------------------------------------------------------------
// A launch covers at most 256 columns (32 lanes x 8).  Wider rows are cut into tiles of 256
// columns that are processed by successive launches on the same stream: left to right in
// the forward (each tile leaves h and s of its last column for its right neighbour), right
// to left in the backward (each tile leaves dh and ds of its first column for its left
// neighbour).  Stream order is the only synchronisation between tiles.
static const int kTileCols = 32 * STRIP;
// Rows that need several tiles anyway are cut into 64-column tiles: those run the 8-lane kernels
// (four channels per warp, dB/dC tiles in shared memory, warp-specialised), which cost far less per
// element than the 32-lane ones a 256-column tile would use.
static const int kNarrowTileCols = 8 * STRIP;
static int tile_cols(int ncols) { return ncols > kTileCols ? kNarrowTileCols : kTileCols; }
static int n_tiles(int ncols) { return (ncols + tile_cols(ncols) - 1) / tile_cols(ncols); }

struct TileView {
    cs2d_problem q;   // the problem restricted to the tile (pointers moved, ncols = tile width)
    int c0;           // first column
    Geometry g;
    size_t saved_off, saved_bytes, adj_off, adj_bytes;   // byte offsets inside saved / scratch
};

static const char *at(const void *p, int64_t elems, int es) {
    return p ? reinterpret_cast<const char *>(p) + elems * es : nullptr;
}

// Fills `tv` for tile t and returns the bytes of the per-tile buffers; edge buffers follow them.
static int tile_view(const cs2d_problem *p, int t, bool backward, bool bulk_ok, TileView *tv, bool serial = false) {
    const int es = esize(p->io_dtype);
    const int tc = tile_cols(p->ncols);
    tv->c0 = t * tc;
    tv->q = *p;
    tv->q.ncols = p->ncols - tv->c0 < tc ? p->ncols - tv->c0 : tc;
    tv->q.u = at(p->u, tv->c0, es);
    tv->q.delta = at(p->delta, tv->c0, es);
    tv->q.B = at(p->B, tv->c0, es);
    tv->q.C = at(p->C, tv->c0, es);
    int rc = plan(&tv->q, backward, bulk_ok, n_tiles(p->ncols) > 1, &tv->g, serial);
    if (rc) return rc;
    const size_t per = (size_t)p->batch * p->dim * tv->g.NPp * (tv->g.L * STRIP) * sizeof(float2);
    tv->saved_bytes = per * tv->g.nck;
    tv->adj_bytes = per;
    return CS2D_OK;
}

static bool walk_shape(const cs2d_problem *p) { return p->dstate > 8 && p->ncols <= 8 * STRIP; }

// Which kernels run (the row-walk forward goes with the tile kernels: it writes the same checkpoints)
enum Family { PAIR, STREAM, BLK, TILE };
static Family family(const cs2d_problem *p, const cs2d_dirs *o);
static bool walk_fwd_ok(const cs2d_problem *p, const cs2d_dirs *o);
static bool pair_one(const cs2d_problem *p);
static bool pair_dirs(const cs2d_problem *p);
static bool tile_state(const cs2d_dirs *o) { return o && (o->flags & CS2D_DIRS_TILE_STATE); }   // the deterministic backward's checkpoints are wanted
static cs2d_dirs with_tile_state(const cs2d_dirs *o, bool on) {
    cs2d_dirs r = o ? *o : cs2d_dirs{};
    r.flags = on ? r.flags | CS2D_DIRS_TILE_STATE : r.flags & ~CS2D_DIRS_TILE_STATE;
    return r;
}
static int check_dirs(const cs2d_problem *p, const cs2d_dirs *o);
static size_t stream_state_bytes(const cs2d_problem *p);
static void blk_fill(Blk &k, int &NG, const cs2d_problem *p, const cs2d_dirs *o, bool backward);
static size_t blk_row_bytes(const Blk &k);
static size_t blk_team_bytes(const Blk &k, bool backward, int NG);
static size_t blk_col_bytes(const Blk &k);
static size_t blk_bc_bytes(const Blk &k, int NG);

// (two states fill a quarter of the lanes and are still 1.2 to 2.2 times as fast as on the tile kernels: 32x4x192x28x28 bf16
// training step 2171 -> 1194 us)
static bool blk_shape(const cs2d_problem *p) { return p->dstate > 1 && p->dim / p->n_groups >= 8; }

static void pair_fill(Pw &k, const cs2d_problem *p, const cs2d_dirs *o, bool backward, const void *img = nullptr, int64_t img_bs = 0,
                      int64_t img_ds = 0, int64_t img_hs = 0);
static size_t pair_row_bytes(const Pw &k);
static size_t pair_team_bytes(const Pw &k, bool backward);
static size_t pair_col_bytes(const Pw &k);

// (a warp of the pair-walk kernels works on 64 channels: too few of them and it is idle)
static bool pair_shape(const cs2d_problem *p) {
    return p->dstate == 1 && p->dim / p->n_groups >= 8 && p->delta_softplus && !p->A_decay && p->delta_dim == p->dim;
}

static size_t edge_bytes(const cs2d_problem *p, int NPp) {
    return (size_t)p->batch * p->dim * NPp * p->nrows * sizeof(float4);
}

// What a buffer holds: the forward's saved state, the rolling rows of a forward that no backward follows, the backward's scratch
enum Buffer { SAVED, ROLLING, SCRATCH };

// The tile kernels' layout: adjoint rows, or the forward's state rows - all checkpoints, or (rolling) one
// row per channel and state pair
static size_t layout_bytes(const cs2d_problem *p, Buffer what, bool walk) {
    const int nt = n_tiles(p->ncols);
    size_t total = 0;
    int NPp = 1;
    for (int t = 0; t < nt; ++t) {
        TileView tv;
        if (tile_view(p, t, what == SCRATCH, false, &tv) != CS2D_OK) return 0;
        total += what == SAVED ? tv.saved_bytes : tv.adj_bytes;
        NPp = tv.g.NPp;
    }
    total += (size_t)(nt - 1) * edge_bytes(p, NPp);
    // the row-walk forward keeps B and C, regrouped, behind the checkpoints
    if (what != SCRATCH && walk) total += walk_bc_bytes(p->batch, p->n_groups, p->nrows, p->ncols);
    return total;
}

static size_t blk_bytes(const cs2d_problem *p, Buffer what) {
    Blk k;
    int NG;
    blk_fill(k, NG, p, nullptr, what == SCRATCH);
    if (what == SCRATCH) return blk_team_bytes(k, true, NG);
    return blk_bc_bytes(k, NG) + (what == ROLLING ? blk_team_bytes(k, false, NG) : blk_row_bytes(k) + blk_col_bytes(k));
}
static size_t pair_bytes(const cs2d_problem *p, Buffer what) {
    Pw k;
    pair_fill(k, p, nullptr, what == SCRATCH);
    return what == SAVED ? pair_row_bytes(k) + pair_col_bytes(k) : pair_team_bytes(k, what == SCRATCH);
}

// Whatever the directions and flags
static size_t any_bytes(const cs2d_problem *p, Buffer what) {
    if (validate(p) != CS2D_OK) return 0;
    const size_t tile = layout_bytes(p, what, walk_shape(p));
    if (tile == 0) return 0;
    const size_t need = pair_shape(p) && (pair_one(p) || pair_dirs(p)) ? pair_bytes(p, what) : blk_shape(p) ? blk_bytes(p, what) : 0;
    return std::max(tile, need);
}

size_t cs2d_saved_bytes(const cs2d_problem *p) { return any_bytes(p, SAVED); }

size_t cs2d_bwd_scratch_bytes(const cs2d_problem *p) { return any_bytes(p, SCRATCH); }

size_t cs2d_fwd_only_scratch_bytes(const cs2d_problem *p) { return any_bytes(p, ROLLING); }

// The same for one set of directions and flags: what the kernels that will run use
static size_t exact_bytes(const cs2d_problem *p, const cs2d_dirs *o, Buffer what) {
    if (validate(p) != CS2D_OK || check_dirs(p, o) != CS2D_OK || layout_bytes(p, what, false) == 0) return 0;
    const Family f = family(p, o);
    size_t n = 16;   // (no buffer is empty)
    if (f == PAIR) n = pair_bytes(p, what);
    else if (f == STREAM && what == SAVED) n = stream_state_bytes(p);
    else if (f == BLK) n = blk_bytes(p, what);
    else if (f == TILE) n = layout_bytes(p, what, walk_fwd_ok(p, o));
    return std::max<size_t>(n, 16);
}
size_t cs2d_saved_bytes_dir(const cs2d_problem *p, const cs2d_dirs *o) {
    const size_t n = exact_bytes(p, o, SAVED);
    if (n == 0 || !tile_state(o)) return n;
    const cs2d_dirs other = with_tile_state(o, false);   // two states of one problem never have the same size
    return family(p, &other) != family(p, o) && exact_bytes(p, &other, SAVED) == n ? n + 16 : n;
}
size_t cs2d_bwd_scratch_bytes_dir(const cs2d_problem *p, const cs2d_dirs *o) { return exact_bytes(p, o, SCRATCH); }
size_t cs2d_fwd_only_scratch_bytes_dir(const cs2d_problem *p, const cs2d_dirs *o) { return exact_bytes(p, o, ROLLING); }

// A group that walks the columns right-to-left sees the tile's scan columns at mirrored image
// columns (Dev::cshift); 4-element accesses are only kept when that shift preserves 16-byte alignment.
static void tile_flip(Dev &d, int ncols, int c0, int tw, int nt) {
    if (nt <= 1 || !d.flip_w) return;
    d.cshift = (int64_t)ncols - 2 * (int64_t)c0 - tw;
    if (d.cshift % 8) d.vec = 0;
}

static int check_dirs(const cs2d_problem *p, const cs2d_dirs *o) {
    if (!o || (!o->flip_rows_mask && !o->flip_cols_mask && !o->shared_input && !o->merge_w)) return CS2D_OK;
    if (p->n_groups > 32) return fail(CS2D_ERR_INVALID, "direction masks cover at most 32 groups");
    return CS2D_OK;
}

// ---- streaming kernels (cs2d_stream.cu) -------------------------------------------------------
// A problem with a single state per channel, one scan orientation, no A_decay and rows of at most
// 128 columns (16 lanes of 8) runs on the streaming kernels: no shared-memory tiles, no backward scratch, and
// checkpoints that pack two channels per value (half the bytes of the tile kernels' layout).  The choice depends on
// nothing but these properties, so the forward and the backward of a problem always agree.
static bool has_dirs(const cs2d_dirs *o) {
    return o && (o->flip_rows_mask || o->flip_cols_mask || o->shared_input || o->merge_w);
}
static bool dirs_serial(const cs2d_dirs *o) { return o && o->merge_w && (o->flags & CS2D_DIRS_SERIAL); }   // one CTA walks all directions
static bool stream_ok(const cs2d_problem *p, const cs2d_dirs *o) {
    return p->dstate == 1 && !has_dirs(o) && !p->A_decay && p->ncols <= 16 * STRIP;
}
static int stream_lanes(const cs2d_problem *p) {
    const int strips = (p->ncols + STRIP - 1) / STRIP;
    int L = 1;
    while (L < strips) L <<= 1;
    return L;
}
static size_t stream_state_bytes(const cs2d_problem *p) {
    const size_t pairs = (size_t)p->batch * p->n_groups * ((p->dim / p->n_groups + 1) / 2);
    return pairs * ((p->nrows + STREAM_RB - 1) / STREAM_RB) * (stream_lanes(p) * STRIP) * sizeof(float2);
}
// Geometry shared by both streaming launches: lanes per row, CTAs per (batch, group), grid.
static void stream_fill(Dev &d, const cs2d_problem *p, int *L, int *grid) {
    Geometry g = {};
    g.L = stream_lanes(p);
    g.NPp = 1; g.CG = 1; g.CP = 1; g.CT = 1; g.npass = 1;
    const int npairs = (p->dim / p->n_groups + 1) / 2, pc = stream_pairs_per_cta(g.L);
    g.ntiles = (npairs + pc - 1) / pc;
    g.nck = (p->nrows + STREAM_RB - 1) / STREAM_RB;
    g.grid = p->batch * p->n_groups * g.ntiles;
    fill(d, p, g);
    const int es = esize(p->io_dtype);
    if (vec8_ok(p->u, es, p->ncols, {p->u_bs, p->u_ds, p->u_hs})) d.vec8 |= VEC_U;
    if (word_ok(p->u, es, p->ncols, {p->u_bs, p->u_ds, p->u_hs})) d.vec2 |= VEC_U;
    if (vec8_ok(p->delta, es, p->ncols, {p->delta_bs, p->delta_ds, p->delta_hs})) d.vec8 |= VEC_DELTA;
    if (word_ok(p->delta, es, p->ncols, {p->delta_bs, p->delta_ds, p->delta_hs})) d.vec2 |= VEC_DELTA;
    if (vec8_ok(p->B, es, p->ncols, {p->B_bs, p->B_gs, p->B_ns, p->B_hs})) d.vec8 |= VEC_B;
    if (word_ok(p->B, es, p->ncols, {p->B_bs, p->B_gs, p->B_ns, p->B_hs})) d.vec2 |= VEC_B;
    if (vec8_ok(p->C, es, p->ncols, {p->C_bs, p->C_gs, p->C_ns, p->C_hs})) d.vec8 |= VEC_C;
    if (word_ok(p->C, es, p->ncols, {p->C_bs, p->C_gs, p->C_ns, p->C_hs})) d.vec2 |= VEC_C;
    *L = g.L; *grid = g.grid;
}

// ---- row-walk forward (cs2d_walk_fwd.cu) ---------------------------------------------------------
// Rows of at most 64 columns with more than 8 states per channel and one scan orientation: the lanes
// of a row work one image row apart, so the recurrence needs no scan.  It writes y and the checkpoints
// exactly where the tile forward would, so the choice is invisible to the backward.
static bool walk_fwd_ok(const cs2d_problem *p, const cs2d_dirs *o) { return walk_shape(p) && !has_dirs(o); }

// ---- block-walk kernels (cs2d_blk_fwd.cu, cs2d_blk_bwd.cu) -------------------------------------------
static bool blk_ok(const cs2d_problem *p, const cs2d_dirs *o) { return blk_shape(p) && !dirs_serial(o) && !tile_state(o); }
// the parts of the saved state (or of the forward-only scratch)
static void blk_state(Blk &k, int NG, const void *saved, bool roll) {
    char *q = const_cast<char *>(static_cast<const char *>(saved));
    k.roll = roll;
    k.bc = reinterpret_cast<float2 *>(q);
    q += blk_bc_bytes(k, NG);
    k.row = reinterpret_cast<float4 *>(q);
    k.col = reinterpret_cast<float4 *>(q + blk_row_bytes(k));
}
static int blk_ctas(bool backward, int NG) { return !backward ? 4 : NG == 16 ? 3 : 2; }   // CTAs per SM
static void blk_fill(Blk &k, int &NG, const cs2d_problem *p, const cs2d_dirs *o, bool backward) {
    k = Blk{};
    k.H = p->nrows; k.W = p->ncols; k.N = p->dstate; k.G = p->n_groups; k.dpg = p->dim / p->n_groups;
    k.drep = p->dim / p->delta_dim;
    k.io_dt = p->io_dtype; k.out_dt = p->out_dtype; k.softplus = p->delta_softplus;
    k.u = p->u; k.delta = p->delta; k.B = p->B; k.C = p->C; k.A = p->A; k.D = p->D; k.bias = p->delta_bias; k.decay = p->A_decay;
    k.u_bs = p->u_bs; k.u_ds = p->u_ds; k.u_hs = p->u_hs;
    k.dl_bs = p->delta_bs; k.dl_ds = p->delta_ds; k.dl_hs = p->delta_hs;
    k.A_ds = p->A_ds; k.A_ns = p->A_ns;
    k.B_bs = p->B_bs; k.B_gs = p->B_gs; k.B_ns = p->B_ns; k.B_hs = p->B_hs;
    k.C_bs = p->C_bs; k.C_gs = p->C_gs; k.C_ns = p->C_ns; k.C_hs = p->C_hs;
    if (o) {
        k.flip_h = o->flip_rows_mask; k.flip_w = o->flip_cols_mask; k.shared = o->shared_input;
        k.mw = o->merge_w; k.dw = o->merge_dw;
    }
    k.nblk = (p->nrows + BK_R - 1) / BK_R; k.nstrip = (p->ncols + BK_S - 1) / BK_S;
    NG = 8;
    while (NG < p->dstate) NG <<= 1;
    k.nsl = (k.dpg + 1) / 2;
    k.NS = k.N <= 4 ? k.N + 1 : NG;
    k.NL = (int64_t)p->batch * k.G * k.nsl * k.NS;
    const int spw = 32 / NG, ctas = blk_ctas(backward, NG);   // slots per warp, CTAs per SM
    k.ntile = (k.nsl + spw - 1) / spw; k.items = p->batch * k.G * k.ntile;
    // Row workers: the number for which the longest chain of blocks that a worker walks takes the least time.  A block's time grows
    // with the warps that share a scheduler (measured on 56x56 maps, and used for all sizes; 1 / full: forward 2.6 / 4.8 us at 4, backward 6.4 / 11.2 us at 3), the
    // last round of CTAs is seldom full, a worker is 1.3 (forward) or 1 blocks behind the one before it, which makes it wait where rows
    // are short, and waiting for each other costs a little (us with 1, 2, 4, 8 workers; stage-1 backward, 3.46 rounds: 3880, 3854, 3870,
    // 4040; forward, 2.59: 1240, 1258, 1208, 1595; 16x4x192x16x28x28 forward, 7 rows, with 1, 2, 4: 200, 179, 220; 2x4x192x16x200x336 backward: 14100,
    // 8750, 6190, 6580; one 56x56 image: 632, 311, 236, 224; 3x4x51x7x45x61: 733, 371, 197, 156).  It is not always the fastest number: for
    // the image the rule takes four workers, 5 % behind eight.
    const double slope = backward ? 0.375 : 0.28, lag = backward ? 1 : 1.3;
    double best = 1e300;
    for (int rwl = 0; (1 << rwl) <= std::min(k.nblk, BK_MAXRW); ++rwl) {
        const int rw = 1 << rwl, warps = std::max(BK_WARPS, rw), cap = ctas * BK_WARPS / warps;   // CTAs per SM
        const int64_t teams = warps / rw, n = ((int64_t)k.items + teams - 1) / teams, full = n / (cap * kSMs), rest = n % (cap * kSMs);
        auto block = [&](int64_t per_sm) { return 1 + slope * (std::max<double>(1, per_sm * warps / 4.0) - 1); };
        const double last = rest ? block((rest + kSMs - 1) / kSMs) : 0;
        const double chain = (double)k.nblk / rw * (rw > 1 ? std::max<double>(k.nstrip, lag * rw) : k.nstrip) * (1 + (backward ? 0.03 : 0.015) * rwl);
        const double cost = chain * (full * block(cap) + last) + lag * (rw - 1) * (last > 0 ? last : block(cap));
        if (cost < best) { best = cost; k.rwl = rwl; k.warps = warps; k.grid = (int)std::min<int64_t>(n, cap * kSMs); }
    }
}
static size_t blk_row_bytes(const Blk &k) { return (size_t)(k.nblk - 1) * k.nstrip * 4 * k.NL * sizeof(float4); }
// One row (the forward's rolling h, the backward's adjoint) per warp, or team of row workers, that is on the GPU at a time: a
// team is done with it before its next item.  The bound does not depend on how the items are split, and so grows with the batch only.
static int64_t resident(int64_t items, int ctas, int warps) { return std::min(items, (int64_t)ctas * kSMs * warps); }
static size_t blk_team_row(const Blk &k) { return (size_t)k.nstrip * 4 * 32 * sizeof(float4); }
static size_t blk_team_bytes(const Blk &k, bool backward, int NG) {
    return (size_t)resident(k.items, blk_ctas(backward, NG), BK_WARPS) * blk_team_row(k);
}
static size_t blk_bc_bytes(const Blk &k, int NG) { return (size_t)(k.items / k.ntile) * k.nblk * k.nstrip * BK_PX * NG * sizeof(float2); }
static size_t blk_col_bytes(const Blk &k) { return (size_t)k.nblk * (k.nstrip - 1) * 4 * k.NL * sizeof(float4); }

// ---- pair-walk kernels (cs2d_pair_fwd.cu, cs2d_pair_bwd.cu) -------------------------------------------
// Directions, and rows of more than 128 columns: the alternative is the tile kernels, a CTA of which takes eight channels.  While
// those run in one round of CTAs they are the faster ones on long rows, until rows are cut into tiles (training step with flips
// and merge, bf16, tile / pair-walk us; 144 CTAs: 96 columns 1444 / 1126, 128: 2025 / 2189, 150: 3049 / 3171, 200: 3943 / 5186, 336: 39108 /
// 16668; 160 CTAs: 128: 3280 / 2164, 150: 5724 / 3516, 200: 7362 / 6131; fp32 144: 96: 1508 / 1412, 200: 3666 / 6659, 156: 7015 / 6673).
static bool pair_dirs(const cs2d_problem *p) {
    return p->ncols <= 96 || p->ncols > kTileCols || (int64_t)p->batch * p->n_groups * ((p->dim / p->n_groups + 7) / 8) > kSMs;
}
// One orientation: the alternative is the streaming kernels, which lose where they load a row element by element or word by word,
// once there are more warps' worth of channels (items) than SMs (training step, streaming / pair-walk us.  16-bit, 192 items:
// 9 columns 103 / 84, 10: 92 / 64, 12: 76 / 68, 14: 123 / 95, 21: 246 / 217, 37: 641 / 490, but at 128: 82 / 84, 60 / 64, 53 / 68, 79 / 95, 184 / 217,
// 379 / 361; 512 items of 18 columns 246 / 188, 22: 305 / 254, 256 of them 129 / 154, 158 / 188; 1152 items of 16: 155 / 157, 704 of 20: 258 / 314,
// 320 of 30: 321 / 382, 768 of 45: 2509 / 2567; a quarter of the channels per item, 37 columns: 635 / 723.  fp32, 768 items: 16 columns
// 236 / 229, 18: 610 / 510, 19: 617 / 574, 20: 380 / 572, 22: 794 / 742, 25: 848 / 1186; 64 items: 9: 82 / 78, 14: 125 / 88, 16: 90 / 91, 17: 115 / 170).
static bool pair_one(const cs2d_problem *p) {
    const int W = p->ncols, dpg = p->dim / p->n_groups;
    const int64_t items = (int64_t)p->batch * p->n_groups * ((dpg + PW_CH - 1) / PW_CH);
    if (p->io_dtype == CS2D_F32) return W <= 16 || (W % 4 && W < 24 && items > kSMs);
    if (W <= 8) return true;
    if (W % 2) return items > kSMs && (W <= 24 || (W < 45 && dpg >= PW_CH));
    return W < 16 ? items > kSMs : W % 4 && W <= 24 && items > 2 * kSMs;
}
static bool pair_ok(const cs2d_problem *p, const cs2d_dirs *o) {
    if (!pair_shape(p) || dirs_serial(o) || tile_state(o)) return false;
    return has_dirs(o) || p->ncols > 16 * STRIP ? pair_dirs(p) : pair_one(p);
}
static Family family(const cs2d_problem *p, const cs2d_dirs *o) {
    return pair_ok(p, o) ? PAIR : stream_ok(p, o) ? STREAM : blk_ok(p, o) ? BLK : TILE;
}
// Bytes that may be moved at once, `most` at most: a divisor of every size and stride (in bytes) and of the address
static int move_bytes(const void *ptr, std::initializer_list<int64_t> sizes, int most = 8) {
    uintptr_t x = reinterpret_cast<uintptr_t>(ptr) | (uintptr_t)most;
    for (int64_t s : sizes) x |= (uintptr_t)s;
    return (int)(x & (~x + 1));
}
static int pair_ctas(bool backward) { return backward ? 2 : 3; }   // CTAs per SM
static int lanes_for(int pieces) {
    int l = 8;
    while (l < pieces) l <<= 1;
    return l;
}
static void pair_state(Pw &k, const void *saved) {
    char *q = const_cast<char *>(static_cast<const char *>(saved));
    k.row = reinterpret_cast<float4 *>(q);
    q += pair_row_bytes(k);
    k.colq = reinterpret_cast<float4 *>(q);
    k.cola = reinterpret_cast<float2 *>(q + pair_col_bytes(k) / 3 * 2);
}
static void pair_fill(Pw &k, const cs2d_problem *p, const cs2d_dirs *o, bool backward, const void *img, int64_t img_bs, int64_t img_ds, int64_t img_hs) {   // img: out or dout
    k = Pw{};
    const int es = esize(p->io_dtype);
    k.H = p->nrows; k.W = p->ncols; k.G = p->n_groups; k.dpg = p->dim / p->n_groups; k.io_dt = p->io_dtype;
    k.u = p->u; k.delta = p->delta; k.B = p->B; k.C = p->C; k.A = p->A; k.D = p->D; k.bias = p->delta_bias;
    k.u_bs = p->u_bs; k.u_ds = p->u_ds; k.u_hs = p->u_hs;
    k.dl_bs = p->delta_bs; k.dl_ds = p->delta_ds; k.dl_hs = p->delta_hs; k.A_ds = p->A_ds;
    k.B_bs = p->B_bs; k.B_gs = p->B_gs; k.B_hs = p->B_hs;
    k.C_bs = p->C_bs; k.C_gs = p->C_gs; k.C_hs = p->C_hs;
    if (o) {
        k.flip_h = o->flip_rows_mask; k.flip_w = o->flip_cols_mask; k.shared = o->shared_input;
        k.mw = o->merge_w; k.dw = o->merge_dw;
    }
    k.f32 = p->io_dtype != CS2D_F32 && p->out_dtype == CS2D_F32;
    k.nblk = (k.H + PW_R - 1) / PW_R; k.nsub = (k.W + 7) / 8; k.wp = (k.W + 1) & ~1;
    k.nl = std::min(32, (k.dpg + 1) / 2 + 1);
    k.ntile = (k.dpg + PW_CH - 1) / PW_CH; k.items = p->batch * k.G * k.ntile;
    // How blocks are moved (see cs2d_pair.cuh): whole bands where every tensor's rows are contiguous and a band fits
    struct In { const void *p; int64_t bs, ds, hs; } in[3] = {{p->u, p->u_bs, p->u_ds, p->u_hs}, {p->delta, p->delta_bs, p->delta_ds, p->delta_hs}, {img, img_bs, img_ds, img_hs}};
    const int ni = backward && img && !k.f32 ? 3 : 2;
    k.lin = PW_R * k.W * es + (k.W & 1 ? 2 : 0) <= 128;
    for (int i = 0; i < ni; ++i) k.lin = k.lin && in[i].hs == k.W;
    if (!backward && img && !k.mw && !k.f32) k.lin = k.lin && img_hs == k.W;
    k.vin = 8;
    for (int i = 0; i < ni; ++i)
        k.vin = std::min(k.vin, k.lin ? move_bytes(in[i].p, {in[i].bs * es, in[i].ds * es, (int64_t)PW_R * k.W * es, (int64_t)k.H * k.W * es})
                                      : move_bytes(in[i].p, {in[i].bs * es, in[i].ds * es, in[i].hs * es, (int64_t)k.W * es}));
    k.al = 16;
    for (int i = 0; i < ni; ++i)
        k.al = std::min(k.al, k.lin ? move_bytes(in[i].p, {in[i].bs * es, in[i].ds * es, (int64_t)PW_R * k.W * es, (int64_t)k.H * k.W * es}, 16)
                                    : move_bytes(in[i].p, {in[i].bs * es, in[i].ds * es, in[i].hs * es, (int64_t)k.W * es}, 16));
    if (k.W & 1) k.vin = std::min(k.vin, es);
    k.el = k.vin < 2 * es;
    if (k.vin < 4) k.vin = 4;
    k.ck = !k.el && (k.al == 16 || (!backward && k.lin && 16 - k.al + PW_R * k.W * es <= 128));   // (how far that is worth it: see there)
    k.fs = k.el && es == 2 && !k.lin ? 8 : 32 / es;
    k.nstrip = k.lin ? 1 : (k.W + k.fs - 1) / k.fs;
    k.lpin = k.lin ? lanes_for((PW_R * k.W * es + (k.el && es == 2 ? 2 : 0) + k.vin - 1) / k.vin) : 4 * (k.el && es == 2 ? 8 : 32 / k.vin);
    // Row workers: as few as fill the GPU; with short rows a worker waits for the others at the end of a band
    const int ctas = pair_ctas(backward);
    const int64_t slots = (int64_t)kSMs * ctas * PW_WARPS;
    double best = 1e300;
    for (int rwl = 0; rwl < 3; ++rwl) {
        const int rw = 1 << rwl;
        if (rw > 1 && k.nblk < rw) break;
        const int period = k.nstrip < rw ? rw : k.nstrip;
        const int64_t npass = (k.nblk + rw - 1) / rw, rounds = ((int64_t)k.items * rw + slots - 1) / slots;
        const double cost = (double)rounds * (npass * period + rw - 1);
        if (cost < best * 0.9) { best = cost; k.rwl = rwl; k.npass = (int)npass; k.period = period; }
    }
    const int64_t need = ((int64_t)k.items + (PW_WARPS >> k.rwl) - 1) / (PW_WARPS >> k.rwl), cap = ctas * kSMs;
    k.grid = (int)(need < cap ? need : cap);
}
static size_t pair_row_bytes(const Pw &k) { return (size_t)k.items * (k.nblk - 1) * k.wp * k.nl * sizeof(float4); }
static size_t pair_team_bytes(const Pw &k, bool backward) { return (size_t)resident(k.items, pair_ctas(backward), PW_WARPS) * k.wp * 32 * sizeof(float4); }
static size_t pair_col_bytes(const Pw &k) { return (size_t)k.items * k.nblk * (k.nsub - 1) * PW_R * k.nl * 24; }
// pieces of results that take the place of inputs in shared memory
static int pair_vout(const Pw &k, const void *ptr, int es, int64_t bs, int64_t ds, int64_t hs) {
    if (k.el && es == 2) return 2;
    if (k.lin) return move_bytes(ptr, {bs * es, ds * es, (int64_t)PW_R * k.W * es, (int64_t)k.H * k.W * es}, k.ck ? 16 : 8);
    return move_bytes(ptr, {bs * es, ds * es, hs * es, (int64_t)k.W * es}, k.ck ? 16 : 8);
}
// `vout`: bytes of a piece that every result which leaves through shared memory allows (16: none of the call's does)
static void pair_out(Pw &k, int es, int vout) {
    // Chunks have no stores of single 16-bit elements, and their blocks are 32 pieces per channel at most: results that lie in the middle of
    // words (a view's, given by the caller) leave the form without chunks instead
    if (vout < 4) k.ck = 0;
    k.vout = std::min(vout, k.ck ? k.al : k.vin);
    k.lpout = k.lin ? lanes_for(PW_R * k.W * es / k.vout) : 4 * k.fs * es / k.vout;
}

static int fwd_impl(const cs2d_problem *p, const cs2d_dirs *o, void *out, int64_t out_bs, int64_t out_ds,
                    int64_t out_hs, void *saved, void *stream, bool rolling = false) {
    int rc = validate(p);
    if (rc) return rc;
    if ((rc = check_dirs(p, o))) return rc;
    const bool dirs = has_dirs(o);
    if (!out || !saved) return fail(CS2D_ERR_INVALID, "out and saved must be given");
    if (o && o->merge_w && p->out_dtype != CS2D_F32)
        return fail(CS2D_ERR_INVALID, "the direction merge adds onto an fp32 image: out_dtype must be CS2D_F32");
    if (reinterpret_cast<uintptr_t>(saved) & 15) return fail(CS2D_ERR_INVALID, "saved must be 16-byte aligned");
    int *status = status_ptr();
    if (!status) return fail(CS2D_ERR_CUDA, "cannot locate the device status word");
    const Family fam = family(p, o);
    if (fam == PAIR) {
        Pw k;
        pair_fill(k, p, o, false, out, out_bs, out_ds, out_hs);
        k.out = out; k.o_bs = out_bs; k.o_ds = out_ds; k.o_hs = out_hs;
        const int es = esize(p->io_dtype);
        pair_out(k, es, k.mw || k.f32 ? 16 : pair_vout(k, out, es, out_bs, out_ds, out_hs));
        k.v32 = move_bytes(out, {out_bs * 4, out_ds * 4, out_hs * 4, (int64_t)k.W * 4}) == 8;
        pair_state(k, saved);
        cudaError_t e = launch_pair_fwd(k, !rolling, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "forward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
        return CS2D_OK;
    }
    if (fam == STREAM) {
        Dev d;
        int L, grid;
        stream_fill(d, p, &L, &grid);
        d.out = out; d.o_bs = out_bs; d.o_ds = out_ds; d.o_hs = out_hs;
        if (vec_ok(out, esize(p->out_dtype), p->ncols, {out_bs, out_ds, out_hs})) d.vec |= VEC_OUT;
        if (vec8_ok(out, esize(p->out_dtype), p->ncols, {out_bs, out_ds, out_hs})) d.vec8 |= VEC_OUT;
        if (word_ok(out, esize(p->out_dtype), p->ncols, {out_bs, out_ds, out_hs})) d.vec2 |= VEC_OUT;
        d.saved = reinterpret_cast<float2 *>(saved);
        d.ck_roll = rolling;
        d.status = status;
        cudaError_t e = launch_stream_fwd(d, L, grid, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "forward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
        return CS2D_OK;
    }
    if (fam == BLK) {
        Blk k;
        int NG;
        blk_fill(k, NG, p, o, false);
        k.status = status;
        k.out = out; k.o_bs = out_bs; k.o_ds = out_ds; k.o_hs = out_hs;
        blk_state(k, NG, saved, rolling);
        cudaError_t e = launch_blk_fwd(k, NG, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "forward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(2);   // the regrouping of B and C, then the scan
        return CS2D_OK;
    }
    if (walk_fwd_ok(p, o)) {
        TileView tv;
        if ((rc = tile_view(p, 0, false, false, &tv))) return rc;   // the checkpoint layout is the tile kernels'
        Dev d;
        fill(d, &tv.q, tv.g);
        int swd, lr;
        walk_geometry(p->ncols, &swd, &lr);
        const int ct = walk_channels_per_cta(lr), dpg = p->dim / p->n_groups;
        d.ntiles = (dpg + ct - 1) / ct;
        d.out = out; d.o_bs = out_bs; d.o_ds = out_ds; d.o_hs = out_hs;
        d.saved = reinterpret_cast<float2 *>(saved);
        d.ck_roll = rolling;
        d.status = status;
        char *bc = reinterpret_cast<char *>(saved) + (rolling ? tv.adj_bytes : tv.saved_bytes);
        d.wbt = reinterpret_cast<float4 *>(bc);
        d.wct = reinterpret_cast<float4 *>(bc + walk_bc_bytes(p->batch, p->n_groups, p->nrows, p->ncols) / 2);
        cudaError_t e = launch_walk_fwd(d, p->batch * p->n_groups * d.ntiles, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "forward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(2);   // the regrouping of B and C, then the scan
        return CS2D_OK;
    }
    const int es = esize(p->io_dtype), eso = esize(p->out_dtype), nt = n_tiles(p->ncols);
    // saved = [checkpoints tile 0 | ... | checkpoints tile nt-1 | edge 0|1 | ... | edge nt-2|nt-1]
    size_t ck_total = 0;
    for (int t = 0; t < nt; ++t) {
        TileView tv;
        if ((rc = tile_view(p, t, false, false, &tv))) return rc;
        ck_total += rolling ? tv.adj_bytes : tv.saved_bytes;
    }
    size_t ck_off = 0;
    for (int t = 0; t < nt; ++t) {
        TileView tv;
        const bool bulk = nt == 1 && !dirs && bulk_ok1(p->u, es, p->ncols, p->u_bs, p->u_ds, p->u_hs) &&
                          bulk_ok1(p->delta, es, p->ncols, p->delta_bs, p->delta_ds, p->delta_hs);
        const bool serial = dirs_serial(o);   // a CTA walks all directions of its channel tile
        if ((rc = tile_view(p, t, false, bulk, &tv, serial))) return rc;
        Dev d;
        fill(d, &tv.q, tv.g);
        d.dir_serial = serial; d.merge_store = serial && nt == 1;
        d.out = const_cast<char *>(at(out, tv.c0, eso)); d.o_bs = out_bs; d.o_ds = out_ds; d.o_hs = out_hs;
        if (vec_ok(d.out, eso, tv.q.ncols, {out_bs, out_ds, out_hs})) d.vec |= VEC_OUT;
        d.saved = reinterpret_cast<float2 *>(reinterpret_cast<char *>(saved) + ck_off);
        ck_off += rolling ? tv.adj_bytes : tv.saved_bytes;
        d.ck_roll = rolling;
        d.status = status;
        d.tile_left = t > 0; d.tile_right = t + 1 < nt; d.Wout = p->ncols;
        const size_t eb = edge_bytes(p, tv.g.NPp);
        char *edges = reinterpret_cast<char *>(saved) + ck_total;
        d.edge_in = t > 0 ? reinterpret_cast<const float4 *>(edges + (size_t)(t - 1) * eb) : nullptr;
        d.edge_out = t + 1 < nt ? reinterpret_cast<float4 *>(edges + (size_t)t * eb) : nullptr;
        if (dirs) {
            d.flip_h = o->flip_rows_mask; d.flip_w = o->flip_cols_mask; d.u_shared = o->shared_input; d.mw = o->merge_w;
            tile_flip(d, p->ncols, tv.c0, tv.q.ncols, nt);
        }
        cudaError_t e = (serial ? launch_fwd_serial : launch_fwd)(d, tv.g.L, tv.g.grid, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "forward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
    }
    return CS2D_OK;
}

int cs2d_fwd(const cs2d_problem *p, void *out, int64_t out_bs, int64_t out_ds, int64_t out_hs, void *saved,
             void *stream) {
    return fwd_impl(p, nullptr, out, out_bs, out_ds, out_hs, saved, stream);
}

int cs2d_fwd_only(const cs2d_problem *p, const cs2d_dirs *dirs, void *out, int64_t out_bs, int64_t out_ds,
                  int64_t out_hs, void *scratch, void *stream) {
    return fwd_impl(p, dirs, out, out_bs, out_ds, out_hs, scratch, stream, true);
}

int cs2d_fwd_dir(const cs2d_problem *p, const cs2d_dirs *dirs, void *out, int64_t out_bs, int64_t out_ds,
                 int64_t out_hs, void *saved, void *stream) {
    return fwd_impl(p, dirs, out, out_bs, out_ds, out_hs, saved, stream);
}

// out[i] += part[i] + part[stride + i] + ... (count terms, in this order): the second step of the
// deterministic backward
__global__ void sum_slots(float *out, const float *part, int64_t n, int count, int64_t stride) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float v = 0.f;
        for (int t = 0; t < count; ++t) v += part[t * stride + i];
        out[i] += v;
    }
}

static cudaError_t launch_sum(float *out, const float *part, int64_t n, int count, int64_t stride, void *stream) {
    if (!out || n <= 0) return cudaSuccess;
    const int block = 256;
    const int64_t want = (n + block - 1) / block;
    sum_slots<<<(unsigned)(want < 8 * kSMs ? want : 8 * kSMs), block, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        out, part, n, count, stride);
    g_launches.fetch_add(1);
    return cudaGetLastError();
}

// layout of the deterministic backward's scratch, in floats
struct DetLayout { int64_t nB, dB, dC, dA, dD, dbias, ddecay, state, total; int ntiles, grid, zero; };
static int det_layout(const cs2d_problem *p, DetLayout *l, bool remake) {   // remake: room for the checkpoints, made again
    if (n_tiles(p->ncols) > 1)
        return fail(CS2D_ERR_UNSUPPORTED, "the deterministic backward covers ncols <= %d", kTileCols);
    TileView tv;
    int rc = tile_view(p, 0, true, false, &tv);
    if (rc) return rc;
    // Without the dB/dC tiles in shared memory the CTA adds to its plane row by row, which has a
    // single writer per element only when the CTA holds one channel group (see add_dbc).
    if (!tv.g.acc && tv.g.CG != 1)
        return fail(CS2D_ERR_UNSUPPORTED, "no deterministic backward for ncols=%d with dstate=%d "
                                          "(dB/dC tiles do not fit in shared memory and several channel groups share a CTA)",
                    p->ncols, p->dstate);
    l->zero = !tv.g.acc;
    l->ntiles = tv.g.ntiles; l->grid = tv.g.grid;
    l->nB = (int64_t)p->batch * p->n_groups * p->dstate * p->nrows * p->ncols;
    l->dB = 0; l->dC = l->dB + l->ntiles * l->nB; l->dA = l->dC + l->ntiles * l->nB;
    l->dD = l->dA + (int64_t)p->batch * p->dim * p->dstate; l->dbias = l->dD + (int64_t)p->batch * p->dim;
    l->ddecay = l->dbias + (int64_t)p->batch * p->dim; l->total = l->ddecay + l->grid;
    l->state = (l->total + 3) & ~int64_t(3);
    if (remake) l->total = l->state + (int64_t)(layout_bytes(p, SAVED, walk_shape(p)) / 4);
    return CS2D_OK;
}

// Fewer CTAs where the scratch is given and holds the rows of fewer teams (cs2d_bwd_noalloc).
static bool fit_grid(int *grid, int64_t items, int teams_per_cta, size_t row, size_t limit) {
    const int64_t teams = (int64_t)(limit / row);
    if (std::min(items, (int64_t)*grid * teams_per_cta) <= teams) return true;
    *grid = (int)(teams / teams_per_cta);
    if (*grid > 0) return true;
    fail(CS2D_ERR_UNSUPPORTED, "one row of the backward scratch is larger than the built-in buffer");
    return false;
}

static int bwd_impl(const cs2d_problem *p, const cs2d_dirs *o, const void *dout, int64_t dout_bs, int64_t dout_ds,
                    int64_t dout_hs, const void *saved, void *scratch, void *du, void *ddelta, float *dA, float *dB,
                    float *dC, float *dD, float *ddelta_bias, float *dA_decay, void *stream, float *det = nullptr,
                    size_t scratch_limit = SIZE_MAX) {
    int rc = validate(p);
    if (rc) return rc;
    if ((rc = check_dirs(p, o))) return rc;
    DetLayout dl = {};
    const Family fam = family(p, o);
    const bool remake = det && (fam == BLK || fam == PAIR);
    if (det && (rc = det_layout(p, &dl, remake))) return rc;
    const bool dirs = has_dirs(o);
    if (o && o->merge_w && (det || !(o->shared_input & 2)))
        return fail(CS2D_ERR_INVALID, "the direction merge needs the shared gradient image (shared_input bit 1) "
                                      "and is not combined with the deterministic backward");
    if (!dout || !saved || !scratch || !du || !ddelta || !dA || !dB || !dC)
        return fail(CS2D_ERR_INVALID, "dout, saved, scratch, du, ddelta, dA, dB, dC must be given");
    if ((reinterpret_cast<uintptr_t>(saved) | reinterpret_cast<uintptr_t>(scratch)) & 15)
        return fail(CS2D_ERR_INVALID, "saved and scratch must be 16-byte aligned");
    if (dA_decay && !p->A_decay) return fail(CS2D_ERR_INVALID, "dA_decay requested without A_decay");
    int *status = status_ptr();
    if (!status) return fail(CS2D_ERR_CUDA, "cannot locate the device status word");
    if (!det && fam == PAIR) {
        Pw k;
        pair_fill(k, p, o, true, dout, dout_bs, dout_ds, dout_hs);
        pair_state(k, saved);
        k.out = const_cast<void *>(dout); k.o_bs = dout_bs; k.o_ds = dout_ds; k.o_hs = dout_hs;
        const int es = esize(p->io_dtype);
        const int64_t W = p->ncols, HW = W * p->nrows;
        pair_out(k, es, std::min(pair_vout(k, du, es, HW, HW, W), pair_vout(k, ddelta, es, HW, HW, W)));
        k.v32 = move_bytes(du, {HW * 4, W * 4}) == 8;
        if (!fit_grid(&k.grid, k.items, PW_WARPS >> k.rwl, (size_t)k.wp * 32 * sizeof(float4), scratch_limit)) return CS2D_ERR_UNSUPPORTED;
        k.adj = reinterpret_cast<float4 *>(scratch);
        k.du = du; k.ddelta = ddelta; k.dA = dA; k.dB = dB; k.dC = dC; k.dD = dD; k.dbias = ddelta_bias;
        cudaError_t e = launch_pair_bwd(k, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "backward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
        return CS2D_OK;
    }
    if (!det && fam == BLK) {
        Blk k;
        int NG;
        blk_fill(k, NG, p, o, true);
        k.status = status;
        blk_state(k, NG, saved, false);
        k.out = const_cast<void *>(dout); k.o_bs = dout_bs; k.o_ds = dout_ds; k.o_hs = dout_hs;
        k.adj = reinterpret_cast<float4 *>(scratch);
        k.du = du; k.ddelta = ddelta; k.dA = dA; k.dB = dB; k.dC = dC; k.dD = dD; k.dbias = ddelta_bias; k.ddecay = dA_decay;
        k.vec_dbc = vec_ok(dB, 4, p->ncols, {}) && vec_ok(dC, 4, p->ncols, {});
        const int es = esize(p->io_dtype), eso = esize(p->out_dtype);
        k.vin = std::min(std::min(move_bytes(p->u, {p->u_bs * es, p->u_ds * es, p->u_hs * es, (int64_t)k.W * es}, 16),
                                  move_bytes(p->delta, {p->delta_bs * es, p->delta_ds * es, p->delta_hs * es, (int64_t)k.W * es}, 16)),
                         move_bytes(dout, {dout_bs * eso, dout_ds * eso, dout_hs * eso, (int64_t)k.W * eso}, 16));
        if (!fit_grid(&k.grid, k.items, k.warps >> k.rwl, blk_team_row(k), scratch_limit)) return CS2D_ERR_UNSUPPORTED;
        cudaError_t e = launch_blk_bwd(k, NG, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "backward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
        return CS2D_OK;
    }
    const cs2d_dirs tile = with_tile_state(o, true);
    if (remake) {
        // The deterministic backward is the tile kernels'; a forward that did not know of it (CS2D_DIRS_TILE_STATE) is made
        // again for the checkpoints (y goes to du, which is written later).
        cs2d_problem q = *p;
        q.out_dtype = p->io_dtype;
        void *st = det + dl.state;
        if ((rc = fwd_impl(&q, &tile, du, (int64_t)p->dim * p->nrows * p->ncols, (int64_t)p->nrows * p->ncols, p->ncols, st, stream)))
            return rc;
        saved = st;
    }
    const bool streamed = family(p, remake ? &tile : o) == STREAM;   // the checkpoints are the streaming kernel's
    if (streamed && !det) {
        Dev d;
        int L, grid;
        stream_fill(d, p, &L, &grid);
        d.out = const_cast<void *>(dout); d.o_bs = dout_bs; d.o_ds = dout_ds; d.o_hs = dout_hs;
        if (vec_ok(dout, esize(p->out_dtype), p->ncols, {dout_bs, dout_ds, dout_hs})) d.vec |= VEC_OUT;
        if (vec8_ok(dout, esize(p->out_dtype), p->ncols, {dout_bs, dout_ds, dout_hs})) d.vec8 |= VEC_OUT;
        if (word_ok(dout, esize(p->out_dtype), p->ncols, {dout_bs, dout_ds, dout_hs})) d.vec2 |= VEC_OUT;
        d.du = du; d.ddelta = ddelta;
        if (vec_ok(du, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}) &&
            vec_ok(ddelta, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}))
            d.vec |= VEC_DU;
        if (vec8_ok(du, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}) &&
            vec8_ok(ddelta, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}))
            d.vec8 |= VEC_DU;
        if (word_ok(du, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}) &&
            word_ok(ddelta, esize(p->io_dtype), p->ncols, {(int64_t)p->ncols}))
            d.vec2 |= VEC_DU;
        d.saved = reinterpret_cast<float2 *>(const_cast<void *>(saved));
        d.dA = dA; d.dB = dB; d.dC = dC; d.dD = dD; d.dbias = ddelta_bias;
        d.status = status;
        cudaError_t e = launch_stream_bwd(d, L, grid, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "backward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
        return CS2D_OK;
    }
    const int es = esize(p->io_dtype), eso = esize(p->out_dtype), nt = n_tiles(p->ncols);
    // saved as laid out by the forward; scratch = [adjoint rows tile 0 | ... | dh/ds edges]
    size_t ck_total = 0, adj_total = 0;
    size_t ck_offs[64], adj_offs[64];
    if (nt > 64) return fail(CS2D_ERR_UNSUPPORTED, "more than 64 column tiles");
    for (int t = 0; t < nt; ++t) {
        TileView tv;
        if ((rc = tile_view(p, t, true, false, &tv))) return rc;
        ck_offs[t] = ck_total; adj_offs[t] = adj_total;
        ck_total += tv.saved_bytes; adj_total += tv.adj_bytes;
    }
    for (int t = nt - 1; t >= 0; --t) {
        TileView tv;
        const bool bulk = nt == 1 && !dirs && bulk_ok1(p->u, es, p->ncols, p->u_bs, p->u_ds, p->u_hs) &&
                          bulk_ok1(p->delta, es, p->ncols, p->delta_bs, p->delta_ds, p->delta_hs) &&
                          bulk_ok1(dout, eso, p->ncols, dout_bs, dout_ds, dout_hs);
        const bool serial = dirs_serial(o);   // a CTA walks all directions of its channel tile
        if ((rc = tile_view(p, t, true, bulk, &tv, serial))) return rc;
        Dev d;
        fill(d, &tv.q, tv.g);
        d.dir_serial = serial; d.merge_store = serial && nt == 1;
        d.out = const_cast<char *>(at(dout, tv.c0, eso)); d.o_bs = dout_bs; d.o_ds = dout_ds; d.o_hs = dout_hs;
        if (vec_ok(d.out, eso, tv.q.ncols, {dout_bs, dout_ds, dout_hs})) d.vec |= VEC_OUT;
        d.du = const_cast<char *>(at(du, tv.c0, o && o->merge_w ? 4 : es));   // the merged du image is fp32
        d.ddelta = const_cast<char *>(at(ddelta, tv.c0, es));
        if (vec_ok(d.du, es, tv.q.ncols, {(int64_t)p->ncols}) && vec_ok(d.ddelta, es, tv.q.ncols, {(int64_t)p->ncols}))
            d.vec |= VEC_DU;
        if (serial && vec_ok(d.du, 4, tv.q.ncols, {(int64_t)p->ncols})) d.vec |= VEC_MDU;   // the merged du image is fp32
        d.saved = reinterpret_cast<float2 *>(const_cast<char *>(reinterpret_cast<const char *>(saved)) + ck_offs[t]);
        d.adj = reinterpret_cast<float2 *>(reinterpret_cast<char *>(scratch) + adj_offs[t]);
        d.dA = dA; d.dB = dB + tv.c0; d.dC = dC + tv.c0; d.dD = dD; d.dbias = ddelta_bias; d.ddecay = dA_decay;
        d.status = status;
        d.ck_pairs = streamed;   // deterministic backward of a streamed forward: read its checkpoint layout
        d.tile_left = t > 0; d.tile_right = t + 1 < nt; d.Wout = p->ncols;
        const size_t eb = edge_bytes(p, tv.g.NPp);
        const char *edges = reinterpret_cast<const char *>(saved) + ck_total;
        char *aedges = reinterpret_cast<char *>(scratch) + adj_total;
        d.edge_in = t > 0 ? reinterpret_cast<const float4 *>(edges + (size_t)(t - 1) * eb) : nullptr;
        d.adj_in = t + 1 < nt ? reinterpret_cast<const float4 *>(aedges + (size_t)t * eb) : nullptr;
        d.adj_out = t > 0 ? reinterpret_cast<float4 *>(aedges + (size_t)(t - 1) * eb) : nullptr;
        if (dirs) {
            d.flip_h = o->flip_rows_mask; d.flip_w = o->flip_cols_mask; d.u_shared = o->shared_input;
            d.mw = o->merge_w; d.dw = o->merge_dw;
            tile_flip(d, p->ncols, tv.c0, tv.q.ncols, nt);
        }
        if (det) {  // per-tile planes and per-batch slots instead of the results themselves
            if (dl.zero && cudaMemsetAsync(det + dl.dB, 0, (size_t)(2 * dl.ntiles * dl.nB) * sizeof(float),
                                           reinterpret_cast<cudaStream_t>(stream)) != cudaSuccess)
                return fail(CS2D_ERR_CUDA, "cannot clear the deterministic scratch");
            d.det = 1; d.det_ts = dl.nB;
            d.dB = det + dl.dB; d.dC = det + dl.dC; d.dA = det + dl.dA;
            d.dD = dD ? det + dl.dD : nullptr; d.dbias = ddelta_bias ? det + dl.dbias : nullptr;
            d.ddecay = dA_decay ? det + dl.ddecay : nullptr;
        }
        cudaError_t e = (serial ? launch_bwd_serial : launch_bwd)(d, tv.g.L, tv.g.grid, reinterpret_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "backward launch failed: %s", cudaGetErrorString(e));
        g_launches.fetch_add(1);
    }
    if (det) {
        const int64_t nA = (int64_t)p->dim * p->dstate;
        cudaError_t e = launch_sum(dB, det + dl.dB, dl.nB, dl.ntiles, dl.nB, stream);
        if (e == cudaSuccess) e = launch_sum(dC, det + dl.dC, dl.nB, dl.ntiles, dl.nB, stream);
        if (e == cudaSuccess) e = launch_sum(dA, det + dl.dA, nA, p->batch, nA, stream);
        if (e == cudaSuccess) e = launch_sum(dD, det + dl.dD, p->dim, p->batch, p->dim, stream);
        if (e == cudaSuccess) e = launch_sum(ddelta_bias, det + dl.dbias, p->dim, p->batch, p->dim, stream);
        if (e == cudaSuccess) e = launch_sum(dA_decay, det + dl.ddecay, 1, dl.grid, 1, stream);
        if (e != cudaSuccess) return fail(CS2D_ERR_CUDA, "deterministic reduction failed: %s", cudaGetErrorString(e));
    }
    return CS2D_OK;
}

size_t cs2d_bwd_det_scratch_bytes(const cs2d_problem *p) {
    DetLayout dl = {};
    if (validate(p) != CS2D_OK || det_layout(p, &dl, blk_shape(p) || pair_shape(p)) != CS2D_OK) return 0;
    return (size_t)dl.total * sizeof(float);
}
size_t cs2d_bwd_det_scratch_bytes_dir(const cs2d_problem *p, const cs2d_dirs *o) {
    DetLayout dl = {};
    if (validate(p) != CS2D_OK || check_dirs(p, o) != CS2D_OK) return 0;
    const Family f = family(p, o);
    if (det_layout(p, &dl, f == BLK || f == PAIR) != CS2D_OK) return 0;
    return (size_t)dl.total * sizeof(float);
}

int cs2d_bwd_det(const cs2d_problem *p, const cs2d_dirs *dirs, const void *dout, int64_t dout_bs, int64_t dout_ds,
                 int64_t dout_hs, const void *saved, void *scratch, void *det_scratch, void *du, void *ddelta,
                 float *dA, float *dB, float *dC, float *dD, float *ddelta_bias, float *dA_decay, void *stream) {
    if (!det_scratch || (reinterpret_cast<uintptr_t>(det_scratch) & 15))
        return fail(CS2D_ERR_INVALID, "det_scratch must be given and 16-byte aligned");
    return bwd_impl(p, dirs, dout, dout_bs, dout_ds, dout_hs, saved, scratch, du, ddelta, dA, dB, dC, dD, ddelta_bias,
                    dA_decay, stream, static_cast<float *>(det_scratch));
}

int cs2d_bwd(const cs2d_problem *p, const void *dout, int64_t dout_bs, int64_t dout_ds, int64_t dout_hs,
             const void *saved, void *scratch, void *du, void *ddelta, float *dA, float *dB, float *dC,
             float *dD, float *ddelta_bias, float *dA_decay, void *stream) {
    return bwd_impl(p, nullptr, dout, dout_bs, dout_ds, dout_hs, saved, scratch, du, ddelta, dA, dB, dC, dD,
                    ddelta_bias, dA_decay, stream);
}

int cs2d_bwd_dir(const cs2d_problem *p, const cs2d_dirs *dirs, const void *dout, int64_t dout_bs, int64_t dout_ds,
                 int64_t dout_hs, const void *saved, void *scratch, void *du, void *ddelta, float *dA, float *dB,
                 float *dC, float *dD, float *ddelta_bias, float *dA_decay, void *stream) {
    return bwd_impl(p, dirs, dout, dout_bs, dout_ds, dout_hs, saved, scratch, du, ddelta, dA, dB, dC, dD,
                    ddelta_bias, dA_decay, stream);
}

/*
 * Backward for callers that must not allocate.
 *
 * Some hosts of this library cannot call cudaMalloc at the point where they run
 * the backward: a serving or training runtime that hands every byte of device
 * memory to its own pool at start-up, a plugin called from inside somebody
 * else's allocator callback, or a binding (a JNI / cgo stub, say) that is only
 * given the tensors it was called with.  For them the adjoint-row scratch that
 * cs2d_bwd takes as an argument lives inside the library instead: a fixed
 * device array that every GPU loading the library carries until the process
 * exits.  In host code the array's name is only a handle, not a device address,
 * so the address is looked up with cudaGetSymbolAddress - once per device, with
 * that device current, on the first call there.  That first call should
 * therefore happen before any stream capture is started.
 *
 * Everything else is cs2d_bwd: same inputs, same caller-provided outputs, same
 * kernel.  Nothing in the array has to be cleared between calls (each row is
 * written before it is read), but all calls share it: two calls that can run
 * at the same time on one GPU would overwrite each other's rows.
 */
static __device__ __align__(256) unsigned char g_noalloc_scratch[CS2D_NOALLOC_SCRATCH_BYTES];

static void *noalloc_scratch_ptr() {
    static void *ptr[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!ptr[dev]) {
        void *q = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&q, g_noalloc_scratch);
        if (e != cudaSuccess || !q) {
            fail(CS2D_ERR_CUDA, "cudaGetSymbolAddress(built-in scratch) failed: %s", cudaGetErrorString(e));
            return nullptr;
        }
        ptr[dev] = q;
    }
    return ptr[dev];
}

int cs2d_bwd_noalloc(const cs2d_problem *p, const void *dout, int64_t dout_bs, int64_t dout_ds, int64_t dout_hs,
                     const void *saved, void *du, void *ddelta, float *dA, float *dB, float *dC, float *dD,
                     float *ddelta_bias, float *dA_decay, void *stream) {
    int rc = validate(p);
    if (rc) return rc;
    // The limit is on the tile kernels' rows, one per channel and state pair: the other families take as many CTAs as the array
    // has rows for.
    const size_t need = layout_bytes(p, SCRATCH, false);
    if (need == 0) return CS2D_ERR_UNSUPPORTED;  // message already set by the planner
    if (need > (size_t)CS2D_NOALLOC_SCRATCH_BYTES)
        return fail(CS2D_ERR_UNSUPPORTED,
                    "this problem needs %zu bytes of backward scratch but the built-in buffer holds %zu; "
                    "split the batch or call cs2d_bwd with your own scratch",
                    need, (size_t)CS2D_NOALLOC_SCRATCH_BYTES);
    void *scratch = noalloc_scratch_ptr();
    if (!scratch) return CS2D_ERR_CUDA;
    return bwd_impl(p, nullptr, dout, dout_bs, dout_ds, dout_hs, saved, scratch, du, ddelta, dA, dB, dC, dD, ddelta_bias,
                    dA_decay, stream, nullptr, CS2D_NOALLOC_SCRATCH_BYTES);
}

int cs2d_device_status(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_cs2d_status, sizeof(int)) != cudaSuccess) return CS2D_ERR_CUDA;
    if (v != 0) {
        cudaMemcpyToSymbol(g_cs2d_status, &zero, sizeof(int));
        status_text(g_err, sizeof(g_err), v);
    }
    return v;
}

const char *cs2d_last_error(void) { return g_err; }
int cs2d_abi_version(void) { return CS2D_ABI_VERSION; }
int64_t cs2d_launch_count(void) { return g_launches.load(); }

}  // extern "C"
