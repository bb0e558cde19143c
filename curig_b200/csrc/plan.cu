// Host orchestration of one ms2dirty / dirty2ms plan: set points (w range,
// sizing, tile binning), execute (spread -> cuFFT -> screen+correction, or the
// adjoint chain), destroy.  Mirrors the reference's plan life cycle
// (gridder_setting / gridder_execution / gridder_destroy, src/astro/cugridder.cu:105-328)
// with device memory from the stream-ordered pool and no host synchronisation
// inside execute.
#include "plan.h"

#include <cudaTypedefs.h>        // PFN_cuTensorMapEncodeTiled

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <tuple>

namespace curig {

#define CU_TRY(x)                                   \
    do {                                            \
        cudaError_t e_ = (x);                       \
        if (e_ != cudaSuccess) {                    \
            p->last_error = cudaGetErrorString(e_); \
            return e_ == cudaErrorMemoryAllocation ? ERR_NOMEM : ERR_CUDA; \
        }                                           \
    } while (0)

template <typename X>
static cudaError_t dalloc(X **ptr, size_t bytes, cudaStream_t st) {
    *ptr = nullptr;
    if (bytes == 0) bytes = 16;
    return alloc_async((void **)ptr, bytes, st);
}

template <typename X>
static void dfree(X *&ptr, cudaStream_t st) {
    if (ptr) cudaFreeAsync((void *)ptr, st);
    ptr = nullptr;
}

// A buffer of the plan: kept from the last set points where it is large enough
// and at most twice as large, else allocated anew.  (Freeing and allocating
// all buffers at every set points took 12-21 ms of a 66-73 ms step at 1.6e8
// visibilities and 4096^2 with several plans in turn: the pool splits freed
// blocks and maps new memory.)  A kept buffer's earlier use is stream-ordered
// before its next one, as a freed block's was.
template <typename X>
static cudaError_t kalloc(Plan *p, X **ptr, size_t bytes, cudaStream_t st) {
    size_t &cap = p->caps[ptr];
    if (*ptr && cap >= bytes && cap <= 2 * bytes + ((size_t)1 << 20)) return cudaSuccess;
    dfree(*ptr, st);
    cap = bytes;
    const cudaError_t e = dalloc(ptr, bytes, st);
    if (e != cudaSuccess) cap = 0;
    return e;
}

static void keep_pool_memory(int device) {
    static bool done[64] = {false};
    if (device < 0 || device >= 64 || done[device]) return;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
        unsigned long long thr = ULLONG_MAX;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr);
    }
    done[device] = true;
}

static int encode_grid_map(Plan *p);

// ------------------------------------------------------------------ cuFFT plan cache
// Rank-1 batched in-place plans keyed by (device, length, element stride,
// batch distance, batch, precision, stream, host thread).  Handles are made
// without a work area of their own (auto-allocation off): every transform pass
// takes one from the stream-ordered pool on the plan's stream and returns it,
// so cached handles hold no large buffers and the pool's memory serves all of
// them.  A handle's stream and work area are per-call state, hence one handle
// per stream and host thread.  Plans hold references to the handles they use;
// released handles stay cached for the next plan of the same shape, at most
// FFT_KEEP of them (least recently released destroyed first), and
// fft_cache_trim (called by curig_release_memory) destroys all of them.
namespace {
struct FftEntry {
    cufftHandle h;
    size_t work;
    int refs;
    unsigned long long released;   // release tick, for the least-recently-released eviction
};
using FftKey = std::tuple<int, int, int, int, int, int, uintptr_t, std::thread::id>;
std::mutex g_fft_mu;
std::map<FftKey, FftEntry> g_fft;
unsigned long long g_fft_tick = 0;
constexpr int FFT_KEEP = 16;
}

static int fft_plan1(Plan *p, int n, int stride, int dist, int batch, int prec, cufftHandle &out, size_t &work) {
    std::lock_guard<std::mutex> lk(g_fft_mu);
    FftKey key = std::make_tuple(p->device, n, stride, dist, batch, prec, (uintptr_t)p->st,
                                 std::this_thread::get_id());
    auto it = g_fft.find(key);
    if (it != g_fft.end()) {
        ++it->second.refs;
        p->fft_keys.push_back(key);
        out = it->second.h;
        work = it->second.work;
        return OK;
    }
    cufftHandle h;
    if (cufftCreate(&h) != CUFFT_SUCCESS) return ERR_CUFFT;
    int nn[1] = {n}, emb[1] = {n};
    size_t ws = 0;
    if (cufftSetAutoAllocation(h, 0) != CUFFT_SUCCESS ||
        cufftMakePlanMany(h, 1, nn, emb, stride, dist, emb, stride, dist, prec ? CUFFT_C2C : CUFFT_Z2Z, batch,
                          &ws) != CUFFT_SUCCESS) {
        cufftDestroy(h);
        return ERR_CUFFT;
    }
    g_fft[key] = FftEntry{h, ws, 1, 0};
    p->fft_keys.push_back(key);
    out = h;
    work = ws;
    return OK;
}

// Drop the plan's references; keep at most FFT_KEEP unreferenced handles.
static void fft_release(Plan *p) {
    std::lock_guard<std::mutex> lk(g_fft_mu);
    for (const FftKey &k : p->fft_keys) {
        auto it = g_fft.find(k);
        if (it != g_fft.end() && it->second.refs > 0 && --it->second.refs == 0) it->second.released = ++g_fft_tick;
    }
    p->fft_keys.clear();
    for (;;) {
        int idle = 0;
        auto oldest = g_fft.end();
        for (auto it = g_fft.begin(); it != g_fft.end(); ++it)
            if (it->second.refs == 0) {
                ++idle;
                if (oldest == g_fft.end() || it->second.released < oldest->second.released) oldest = it;
            }
        if (idle <= FFT_KEEP) break;
        cufftDestroy(oldest->second.h);
        g_fft.erase(oldest);
    }
}

int fft_cache_trim() {
    std::lock_guard<std::mutex> lk(g_fft_mu);
    int n = 0;
    for (auto it = g_fft.begin(); it != g_fft.end();) {
        if (it->second.refs == 0) {
            cufftDestroy(it->second.h);
            it = g_fft.erase(it);
            ++n;
        } else {
            ++it;
        }
    }
    return n;
}

int fft_cache_size() {
    std::lock_guard<std::mutex> lk(g_fft_mu);
    return (int)g_fft.size();
}

// ------------------------------------------------------------------ learned-window registry
namespace {
std::mutex g_win_mu;
std::vector<Window> g_windows;
}

// |k'| <= pi / sigma by the choice of gamma and h (set_nhg_type3), a little more for rounding.
static double psi_range(double sigma) { return PI_D / sigma * (1.0 + 1e-9); }

int registry_set_window(int kw, int degree, const double *coef, double eps_reached) {
    if (kw < 2 || kw > MAX_KW || degree < 1 || degree + 1 > MAX_POLY || !coef) return ERR_ARG;
    Window w;
    w.kind = 1;
    w.kw = kw;
    w.degree = degree;
    w.coef.assign(coef, coef + (size_t)kw * (degree + 1));
    w.eps_reached = eps_reached;
    if (degree <= TAB_DEG - 1) table_bounds(w.coef, kw, degree + 1, w.bound);
    {
        KernelParams kp;
        kp.kw = kw;
        double qx[MAX_QUAD], qg[MAX_QUAD];
        const int nq = quadrature_terms(kp, w, qx, qg);
        w.psi.resize(PSI_TERMS);
        w.psi.resize(psi_series(qx, qg, nq, psi_range(2.0), PSI_TERMS, w.psi.data()));
    }
    std::lock_guard<std::mutex> lk(g_win_mu);
    for (auto &x : g_windows)
        if (x.kw == kw) { x = w; return OK; }
    g_windows.push_back(w);
    return OK;
}

bool registry_pick_window(double eps, Window &out) {
    std::lock_guard<std::mutex> lk(g_win_mu);
    const Window *best = nullptr;
    for (auto &x : g_windows)
        if (x.eps_reached <= eps && (!best || x.kw < best->kw)) best = &x;
    if (best) out = *best;                       // a copy: the registry may grow meanwhile
    return best != nullptr;
}

bool registry_get_window(int kw, Window &out) {
    std::lock_guard<std::mutex> lk(g_win_mu);
    for (auto &x : g_windows)
        if (x.kw == kw) {
            out = x;
            return true;
        }
    return false;
}

void registry_clear() {
    std::lock_guard<std::mutex> lk(g_win_mu);
    g_windows.clear();
}

// ------------------------------------------------------------------ window tables
// The ES window's tables depend on its width and beta only; the most recent
// ones are kept (their samples took 0.1 ms of every set points on the host).
namespace {
std::mutex g_tab_mu;
std::map<std::tuple<int, double, bool>, std::shared_ptr<const WindowTable>> g_tabs;
constexpr size_t TABS_KEPT = 64;
}

static std::shared_ptr<const WindowTable> es_table(const KernelParams &kp, bool fp32) {
    const auto key = std::make_tuple(kp.kw, kp.beta, fp32);
    {
        std::lock_guard<std::mutex> lk(g_tab_mu);
        auto it = g_tabs.find(key);
        if (it != g_tabs.end()) return it->second;
    }
    auto t = std::make_shared<WindowTable>();
    if (fp32) {
        Window w;
        es_horner_window(kp, TAB_DEG - 1, w);
        t->c = w.coef;
        table_bounds(t->c, kp.kw, TAB_DEG, t->bound);
    } else {
        es_table64(kp, TAB64_DEG - 1, t->c);
    }
    std::lock_guard<std::mutex> lk(g_tab_mu);
    if (g_tabs.size() >= TABS_KEPT) g_tabs.clear();
    g_tabs[key] = t;
    return t;
}

// The series of the window's transform for the corrections (psi_series): a
// learned window's comes with it (sigma = 2), the ES window's most recent ones are kept.
static std::vector<double> psi_terms(const KernelParams &kp, const Window &win, const double *qx, const double *qg, int nq) {
    static std::mutex mu;
    static std::map<std::tuple<int, double, double>, std::vector<double>> kept;
    if (win.kind != 0 && kp.upsampfac == 2.0 && !win.psi.empty()) return win.psi;
    const auto key = std::make_tuple(kp.kw, kp.beta, kp.upsampfac);
    if (win.kind == 0) {
        std::lock_guard<std::mutex> lk(mu);
        auto it = kept.find(key);
        if (it != kept.end()) return it->second;
    }
    std::vector<double> t(PSI_TERMS);
    t.resize(psi_series(qx, qg, nq, psi_range(kp.upsampfac), PSI_TERMS, t.data()));
    if (win.kind == 0) {
        std::lock_guard<std::mutex> lk(mu);
        if (kept.size() >= TABS_KEPT) kept.clear();
        kept[key] = t;
    }
    return t;
}

// A learned window's table (degree <= TAB_DEG - 1), leading zeros up to TAB_DEG columns.
static std::shared_ptr<const WindowTable> learned_table(const Window &w) {
    auto t = std::make_shared<WindowTable>();
    t->c.assign((size_t)w.kw * TAB_DEG, 0.0);
    for (int d = 0; d < w.kw; ++d)
        for (int i = 0; i <= w.degree; ++i)
            t->c[d * TAB_DEG + (TAB_DEG - 1 - w.degree) + i] = w.coef[(size_t)d * (w.degree + 1) + i];
    if (w.bound.empty()) table_bounds(t->c, w.kw, TAB_DEG, t->bound);
    else t->bound = w.bound;
    return t;
}

// ------------------------------------------------------------------ instrumentation
namespace {
std::atomic<long long> g_launches{0};
std::atomic<bool> g_timing{false};
}

void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(); }
void set_timing(bool on) { g_timing.store(on); }

static void mark(Plan *p, int slot) {
    if (!g_timing.load()) return;
    if (!p->ev[slot]) cudaEventCreate(&p->ev[slot]);
    cudaEventRecord(p->ev[slot], p->st);
    p->ev_recorded[slot] = true;
}

int plan_timings(Plan *p, double *out, int n) {
    static const int pairs[11][2] = {{EV_SET_BEGIN, EV_SET_END}, {EV_SET_WRANGE, EV_SET_END},
                                     {EV_M2D_BEGIN, EV_M2D_PREP}, {EV_M2D_PREP, EV_M2D_ZERO},
                                     {EV_M2D_ZERO, EV_M2D_SPREAD}, {EV_M2D_SPREAD, EV_M2D_FFT},
                                     {EV_M2D_FFT, EV_M2D_END}, {EV_D2M_BEGIN, EV_D2M_CORRECT},
                                     {EV_D2M_CORRECT, EV_D2M_FFT}, {EV_D2M_FFT, EV_D2M_INTERP},
                                     {EV_D2M_INTERP, EV_D2M_END}};
    if (cudaStreamSynchronize(p->st) != cudaSuccess) return ERR_CUDA;
    for (int i = 0; i < n && i < 11; ++i) {
        out[i] = -1.0;
        int a = pairs[i][0], b = pairs[i][1];
        float ms = 0;
        if (p->ev_recorded[a] && p->ev_recorded[b] && cudaEventElapsedTime(&ms, p->ev[a], p->ev[b]) == cudaSuccess)
            out[i] = ms;
    }
    return OK;
}

// ------------------------------------------------------------------ tile-load wait
// Polls of the interpolator's tile-load barrier before it gives up (about a
// second at the default); a test can shorten it and suppress the load so that
// the wait runs out on purpose (nothing is in flight when the CTA leaves).
namespace {
std::atomic<long long> g_tma_polls{DEFAULT_TMA_POLLS};
std::atomic<int> g_tma_noissue{0};
}

void set_tile_wait(long long polls, int noissue) {
    g_tma_polls.store(polls > 0 ? polls : DEFAULT_TMA_POLLS);
    g_tma_noissue.store(noissue ? 1 : 0);
}

// The interpolator's sparse threshold (DEFAULT_SPARSE_I) is not an option of the
// calls; a test sets it (negative: the default).
namespace {
std::atomic<int> g_sparse_interp{-1};
}

void set_sparse_interp(int n) { g_sparse_interp.store(n); }

// The binning's limit, which a test lowers to bin a small call as a large one.
namespace {
std::atomic<long long> g_ranked_bytes{RANKED_BYTES};
}

void set_ranked_bytes(long long n) { g_ranked_bytes.store(n >= 0 ? n : RANKED_BYTES); }

// ms2dirty's weighted gather takes a scratch vis * wgt from the pool, or, when
// that allocation fails (or a test turns the scratch off), gathers vis and wgt
// in one pass.
namespace {
std::atomic<int> g_gather_scratch{1};
}

void set_gather_scratch(int on) { g_gather_scratch.store(on ? 1 : 0); }

// The transposed image columns' buffer serves where it is large enough (it is
// written by the plane transforms, after the gather); own: to be freed.
template <typename T>
static void *gather_scratch(Plan *p, const void *d_wgt, long long M, bool &own) {
    own = false;
    if (!d_wgt || !g_gather_scratch.load()) return nullptr;
    const size_t need = (size_t)M * 2 * sizeof(T);
    if ((size_t)p->gp.nf3 * p->ny * p->gp.nf2 * 2 * sizeof(T) >= need) return p->d_tgrid;
    void *vw = nullptr;
    own = dalloc(&vw, need, p->st) == cudaSuccess;
    return own ? vw : nullptr;
}

// ------------------------------------------------------------------ plan
int plan_create(int type, int nx, int ny, double psx, double psy, double eps, double sigma, int sign,
                const Options &opt, Plan **out) {
    *out = nullptr;
    if ((type != 1 && type != 2) || nx <= 0 || ny <= 0 || nx > (1 << 24) || ny > (1 << 24))
        return ERR_ARG;
    if (opt.precision != 0 && opt.precision != 1) return ERR_ARG;
    if (opt.smode < 0 || opt.smode > 3) return ERR_ARG;
    if (opt.w_term < 0 || opt.w_term > 1 || opt.grid_x < 0 || opt.grid_y < 0 || (opt.grid_x > 0) != (opt.grid_y > 0))
        return ERR_ARG;
    if (opt.bin_z < 0) return ERR_ARG;
    if (!std::isfinite(psx) || !std::isfinite(psy) || !(psx > 0) || !(psy > 0)) return ERR_ARG;
    KernelParams kp;
    int st = setup_kernel(eps, sigma, kp);
    if (st != OK) return st;
    Plan *p = new Plan();
    p->type = type;
    p->nx = nx;
    p->ny = ny;
    p->psx = psx;
    p->psy = psy;
    p->eps = eps;
    p->sigma = sigma;
    p->sign = sign >= 0 ? 1 : -1;
    p->opt = opt;
    p->st = opt.stream;
    if (cudaGetDevice(&p->device) != cudaSuccess) { delete p; return ERR_CUDA; }
    cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, p->device);
    keep_pool_memory(p->device);
    *out = p;
    return OK;
}

// Forgets the points and their sizes; the buffers stay.
static void plan_reset(Plan *p) {
    p->dg.cbin = nullptr;
    p->dg.ccls = nullptr;
    fft_release(p);
    p->fft_hx = p->fft_hx_rest = p->fft_hy = p->fft_hy_rest = 0;
    p->ready = false;
    p->geom_ready = false;
}

void plan_release_points(Plan *p) {
    cudaStream_t st = p->st;
    plan_reset(p);
    dfree(p->d_tab, st);
    p->d_foc = p->d_quad = p->d_psi1 = p->d_psi2 = p->d_psi3 = p->d_wcoef = nullptr;
    p->d_tw = p->d_twz = nullptr;
    dfree(p->d_bins, st);
    p->d_bin_start = p->d_bin_count = p->d_nsub = p->d_sub_end = p->d_bcur = p->d_scan = nullptr;
    p->d_keys_in = nullptr;
    p->d_tmp = nullptr;
    dfree(p->d_kcount, st);
    dfree(p->d_cbin, st); p->dg.cbin = nullptr; p->dg.ccls = nullptr;
    dfree(p->d_idx, st); dfree(p->d_keys, st);
    p->d_err = nullptr;
    dfree(p->d_rec, st); dfree(p->d_ph, st); dfree(p->d_cs, st); dfree(p->d_grid, st);
    dfree(p->d_tgrid, st);
    fft_release(p);
    p->fft_hx = p->fft_hx_rest = p->fft_hy = p->fft_hy_rest = 0;
    p->ready = false;
    p->geom_ready = false;
}

int plan_destroy(Plan *p) {
    if (!p) return OK;
    plan_release_points(p);
    cudaStreamSynchronize(p->st);
    for (auto &e : p->ev)
        if (e) cudaEventDestroy(e);
    delete p;
    return OK;
}

// Bin / tile geometry: among the xy bin sizes whose tile (bin + kw halo, all
// w-planes when the w support never wraps, else 8- or 4-plane slabs) fits the
// shared-memory budget, the one with the smallest tile/core cell ratio (the
// halo overhead of zeroing, staging and flushing a tile).
// FP32 tile accumulation of the spreader (kernel numbering: 0 two-word int32,
// 1 float atomics, 2 one-word int32).  Automatic: one word when the requested
// epsilon is at least 1e-5 (its rounding, about 1.5e-6 relative, stays well
// inside the error budget), else the exact two-word form.  FP64 tiles take the
// exact three-word int32 form in every mode but 1 (double atomics).
static int tile_mode(const Plan *p) {
    switch (p->opt.smode) {
    case 1: return 1;
    case 2: return 2;
    case 3: return 0;
    default: return p->eps >= 1e-5 ? 2 : 0;
    }
}

// Does the window fit the thread-per-visibility kernels' tables?  Wider ones and
// learned windows of a higher degree take the general kernels (k_spread, k_interp).
static bool tabulated(const Plan *p) {
    return p->gp.kp.kw <= TAB_KW && (p->win.kind == 0 || p->win.degree <= TAB_DEG - 1);
}

static int choose_tiles(Plan *p, int esize, bool force_slabs) {
    const GridParams &gp = p->gp;
    const int kw = gp.kp.kw;
    TileGeom &t = p->tg;
    // FP32 spreader: int32 fixed point, two words (exact) or one word per component;
    // FP64: three-word int32 fixed point (exact)
    const int mode = tile_mode(p);
    t.fix = !tabulated(p) ? 0 : esize == 4 ? (mode == 0 ? 1 : mode == 2 ? 2 : 0) : (mode != 1 ? 3 : 0);
    // FP32 tiles: two CTAs per SM (<= 112 KB each); FP64 fixed-point tiles: one
    // CTA per SM (its registers), so a larger tile with less halo
    size_t budget = p->opt.smem_budget ? p->opt.smem_budget
                    : (t.fix == 3 ? 200 * 1024 : t.fix ? 112 * 1024 : esize == 4 ? 72 * 1024 : 100 * 1024);
    int wdeg = p->win.kind ? p->win.degree : 0;
    // does the w support stay inside [0, nf3)?  (z grows monotonically with w;
    // same arithmetic as the binning kernel, which rejects any start outside)
    auto zstart = [&](double we) {
        double wp = (we - gp.i_center) / gp.gamma;
        double gz = (wp * INV_2PI + 0.5) * gp.nf3;
        return std::ceil(gz - 0.5 * kw);
    };
    double z0 = zstart(p->wmin_eff), z1 = zstart(p->wmax_eff);
    bool nowrap = gp.no_w || (!force_slabs && z0 >= 0.0 && z1 <= gp.nf3 - kw && gp.nf3 <= 4000);
    if (p->opt.n3 > 0) nowrap = false;                  // 3-D NUFFT: the third axis is periodic
    const int cand[] = {96, 64, 48, 32, 24, 20, 16, 12, 10, 8, 6, 4, 2};
    double best = 1e30;
    int bb = 0, bz_best = 0;
    auto consider = [&](int b, int bz, int tz) {
        if ((p->opt.bin_xy && b != p->opt.bin_xy) || b > gp.nf1 || b > gp.nf2) return;
        TileGeom q;
        q.tx = b + kw; q.ty = b + kw; q.tz = tz; q.fix = t.fix;
        if (q.tx > 1024 || tz > 4096 || tile_smem_bytes(q, esize, kw, wdeg) > budget) return;
        double ratio = (double)q.tx * q.ty * tz / ((double)b * b * bz);
        if (ratio < best - 1e-9) { best = ratio; bb = b; bz_best = bz; }
    };
    std::vector<int> edges(cand, cand + sizeof(cand) / sizeof(cand[0]));
    if (p->opt.bin_xy > 0) edges.assign(1, p->opt.bin_xy);   // a requested edge, any size
    if (p->opt.bin_z > 0 && !gp.no_w) {                 // requested slab depth
        if (p->opt.bin_z >= gp.nf3) return ERR_ARG;
        nowrap = false;
        for (int b : edges) consider(b, p->opt.bin_z, p->opt.bin_z + kw);
    } else {
        for (int b : edges) {
            if (nowrap) consider(b, gp.nf3, gp.nf3);
            for (int bz : {8, 4, 2}) if (bz < gp.nf3) consider(b, bz, bz + kw);
        }
    }
    if (!bb) return ERR_UNSUPPORTED;
    if (nowrap && bz_best == gp.nf3) {
        t.zpad = 0; t.bz = gp.nf3; t.tz = gp.nf3; t.nbz = 1;
    } else {
        t.zpad = 1; t.bz = bz_best; t.tz = bz_best + kw; t.nbz = (gp.nf3 + bz_best - 1) / bz_best;
    }
    t.bx = t.by = bb;
    t.tx = bb + kw; t.ty = bb + kw;
    t.nbx = (gp.nf1 + bb - 1) / bb;
    t.nby = (gp.nf2 + bb - 1) / bb;
    // visibilities per chunk: the two- and three-word tiles' per-cell headroom
    // assumes <= 4096; the one-word tiles bound their scale per chunk, so their
    // chunks may be larger: fewer tile flushes and reloads per bin (bench size,
    // 1.6e8 visibilities, ~4900 per bin: 67.4 ms per step at 4096, 66.2 at
    // 8192, 65.5-65.7 at 16384, no further change at 32768 or 65536).  Calls
    // with fewer visibilities cut their crowded bins smaller, so that no chunk
    // holds more than its share of the launch: an array's core puts most
    // visibilities into few bins, and whole chunks are what CTAs take turns
    // with.  At most a sixth of an SM's share (M / 16 of it also cut bins of
    // evenly spread points: 2-D NUFFT, 2e6 points, 1115 -> 1368 us), not below
    // the size whose taps outweigh its tile's zeroing and flush.  Spreader /
    // interpolator, us, uv tracks, chunks of 16384 (FP64 4096) against this
    // rule: FP32 80000 visibilities 384^2 216 / 191 -> 37 / 27, 2e5 512^2 160 /
    // 154 -> 49 / 31, 2e6 1500^2 852 / 653 -> 459 / 359; FP64 1.5e5 480 x 750
    // 997 / 681 -> 518 / 353.
    const int one_word = t.fix == 2;
    const long long vis = p->nrow * p->nchan / std::max(1, p->opt.slabs);
    const long long share = vis / ((long long)p->nsm * 6);
    const int least = esize == 4 ? 512 : 256;
    const int most = one_word ? 16384 : 4096;
    t.sub = p->opt.sub > 0 ? std::min(p->opt.sub, one_word ? 65536 : 4096)
                           : (int)std::min<long long>(most, std::max<long long>(least, share));
    t.smem_bytes = tile_smem_bytes(t, esize, kw, wdeg);
    if (t.nbins() > INT_MAX / 2) return ERR_UNSUPPORTED;
    return OK;
}

// Cells of one axis that points with coordinates in [lo, hi] (cycles per pixel
// times nf cells) can reach, two cells of margin beyond the taps, even bounds;
// the whole axis where the periodic wrap comes into play.
static void axis_window(double lo, double hi, int nf, int kw, int *win) {
    const double a = std::floor((lo + 0.5) * nf - 0.5 * kw) - 2.0, b = std::ceil((hi + 0.5) * nf + 0.5 * kw) + 3.0;
    win[0] = 0;
    win[1] = nf;
    if (!(a >= 0.0 && b <= nf)) return;
    win[0] = (int)a & ~1;
    win[1] = std::min(nf, ((int)b + 1) & ~1);
}

static double key_to_double(unsigned long long k) {
    unsigned long long b = (k & 0x8000000000000000ULL) ? (k & 0x7fffffffffffffffULL) : ~k;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}

int plan_setpts_geometry(Plan *p, long long nrow, int nchan, const double *du, const double *dv,
                         const double *dw, int stride, const double *h_freq) {
    if (!p) return ERR_ARG;
    if (nrow <= 0 || nchan <= 0 || !du || !dv || !dw || !h_freq || stride <= 0) return ERR_ARG;
    if (nrow * (long long)nchan >= INT_MAX) return ERR_ARG;
    for (int c = 0; c < nchan; ++c)
        if (!std::isfinite(h_freq[c]) || !(h_freq[c] > 0)) return ERR_NONFINITE;
    plan_reset(p);
    cudaStream_t st = p->st;
    p->nrow = nrow;
    p->nchan = nchan;
    p->freq.assign(h_freq, h_freq + nchan);
    p->du = du; p->dv = dv; p->dw = dw; p->stride = stride;
    const int esize = p->opt.precision ? 4 : 8;

    // 1. raw w range -> effective range over channels (precomp.cu:61-69, utils.cu:42-53);
    //    the u and v ranges give the window of the grid that the points reach
    mark(p, EV_SET_BEGIN);
    // ranges of w, u, v, then the error flags: one block, one copy each way
    unsigned long long hk[7] = {ULLONG_MAX, 0ULL, ULLONG_MAX, 0ULL, ULLONG_MAX, 0ULL, 0ULL};
    CU_TRY(kalloc(p, &p->d_keys, sizeof(hk), st));
    p->d_err = reinterpret_cast<int *>(p->d_keys + 6);
    CU_TRY(cudaMemcpyAsync(p->d_keys, hk, sizeof(hk), cudaMemcpyHostToDevice, st));
    launch_ranges(dw, du, dv, stride, nrow, p->d_keys, p->d_err, st);
    CU_TRY(cudaMemcpyAsync(hk, p->d_keys, sizeof(hk), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    CU_TRY(cudaGetLastError());
    if ((int)hk[6] & EF_NONFINITE) return ERR_NONFINITE;
    double wmin = key_to_double(hk[0]), wmax = key_to_double(hk[1]);
    double lo = INFINITY, hi = -INFINITY;
    std::vector<double> foc(nchan);
    for (int c = 0; c < nchan; ++c) {
        foc[c] = h_freq[c] / SPEEDOFLIGHT;
        double a = foc[c] * p->sign;
        for (double w : {wmin, wmax}) {
            double v = (w * a) * (2 * PI_D);
            lo = std::min(lo, v);
            hi = std::max(hi, v);
        }
    }
    p->wmin_eff = lo;
    p->wmax_eff = hi;

    // 2. sizes (cugridder.cu:29-101, 180-186) and window
    int kw_override = 0;
    p->win = Window();
    if (p->opt.window == 1) {
        if (!registry_pick_window(p->eps, p->win)) return ERR_WINDOW;
        kw_override = p->win.kw;
    }
    GridRequest req;
    req.grid_x = p->opt.grid_x;
    req.grid_y = p->opt.grid_y;
    req.no_w = p->opt.w_term == 1 || p->opt.n3 > 0;
    int s = grid_params(p->nx, p->ny, p->psx, p->psy, lo, hi, p->eps, p->sigma, p->sign, p->gp, kw_override, req);
    if (s != OK) return s;
    if (req.no_w && p->gp.kp.kw > TAB_KW) return ERR_UNSUPPORTED;   // no w-free mode at these widths
    if (p->opt.n3 > 0) {        // generic 3-D NUFFT: a periodic third axis of the NUFFT's own size
        GridParams &g3 = p->gp;
        g3.no_w = 0;
        g3.nf3 = get_num_cells(p->opt.n3, g3.kp);
        g3.gamma = 1.0;
        g3.i_center = g3.i_half = g3.o_center = g3.o_half = 0.0;
        g3.h = 2 * PI_D / g3.nf3;
    }
    p->win.kw = p->gp.kp.kw;
    // 3. correction tables (deconv.cu:60-197): psi1, psi2 on the grid, quadrature for psi3
    //    (psi1 / psi2 evaluated on the device from the quadrature: no host work
    //    while the GPU waits)
    const GridParams &gp = p->gp;
    double qx[MAX_QUAD], qg[MAX_QUAD];
    int nq = quadrature_terms(gp.kp, p->win, qx, qg);
    const int pr = p->opt.precision;
    fft_make_plan(gp.nf1, esize, p->fx);
    fft_make_plan(gp.nf2, esize, p->fy);
    p->fz = FftPlan();
    if (p->opt.n3 > 0 && gp.nf3 <= FFT_ZMAX) fft_make_plan(gp.nf3, 8, p->fz);
    // all tables in one block: what the host uploads in front (one copy), then
    // what the device fills in
    const bool learned = p->win.kind == 1;
    std::vector<double> up(foc);
    up.resize(nchan + 2 * MAX_QUAD, 0.0);
    std::copy(qx, qx + nq, up.begin() + nchan);
    std::copy(qg, qg + nq, up.begin() + nchan + MAX_QUAD);
    if (learned) up.insert(up.end(), p->win.coef.begin(), p->win.coef.end());
    const size_t n1 = gp.nf1 / 2 + 1, n2 = gp.nf2 / 2 + 1, n3 = p->opt.n3 > 0 ? gp.nf3 / 2 + 1 : 0;
    const size_t reals = (up.size() + n1 + n2 + n3 + 1) & ~(size_t)1;       // (twiddles: 16-byte aligned)
    const size_t tws = (size_t)(p->fx.tw_len + p->fy.tw_len) * 16, twz = (size_t)p->fz.tw_len * 16;
    CU_TRY(kalloc(p, &p->d_tab, reals * sizeof(double) + tws + twz, st));
    p->d_foc = p->d_tab;
    p->d_quad = p->d_foc + nchan;
    p->d_wcoef = learned ? p->d_quad + 2 * MAX_QUAD : nullptr;
    p->d_psi1 = p->d_tab + up.size();
    p->d_psi2 = p->d_psi1 + n1;
    p->d_psi3 = n3 ? p->d_psi2 + n2 : nullptr;
    p->d_tw = tws ? p->d_tab + reals : nullptr;
    p->d_twz = twz ? reinterpret_cast<char *>(p->d_tab + reals) + tws : nullptr;
    CU_TRY(cudaMemcpyAsync(p->d_tab, up.data(), up.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    launch_psi_grids((int)n1, (int)n2, (int)n3, nq, p->d_quad, p->d_quad + MAX_QUAD, p->d_psi1, st);
    if (tws && pr) launch_fft_tables<float>(p->fx, p->fy, p->d_tw, st);
    else if (tws) launch_fft_tables<double>(p->fx, p->fy, p->d_tw, st);
    if (twz) launch_fft_tables<double>(p->fz, FftPlan(), p->d_twz, st);
    DevCorr &cc = p->dc;
    cc.nx = p->nx; cc.ny = p->ny; cc.nf1 = gp.nf1; cc.nf2 = gp.nf2; cc.nf3 = gp.nf3;
    cc.psx = gp.pixsize_x; cc.psy = gp.pixsize_y; cc.o_center = gp.o_center; cc.i_center = gp.i_center;
    cc.gamma = gp.gamma; cc.h = gp.h; cc.nquad = nq; cc.no_w = gp.no_w;
    cc.npsi = 0;
    if (!gp.no_w && p->opt.n3 == 0) {
        const std::vector<double> t = psi_terms(gp.kp, p->win, qx, qg, nq);
        cc.npsi = (int)t.size();
        std::copy(t.begin(), t.end(), cc.psi);
        cc.kpmax = psi_range(gp.kp.upsampfac);
    }
    cc.qx = p->d_quad; cc.qg = p->d_quad + MAX_QUAD; cc.psi1 = p->d_psi1; cc.psi2 = p->d_psi2;
    cc.n3 = p->opt.n3; cc.psi3 = p->d_psi3; cc.dbg = p->d_err;

    // 4. fine grid and FFT plans
    size_t gbytes = (size_t)gp.nf1 * gp.nf2 * gp.nf3 * 2 * esize;
    CU_TRY(kalloc(p, &p->d_grid, gbytes, st));

    // 2-D transforms as two passes of contiguous rows: x rows of every plane
    // (length nf1), and y rows (length nf2) of the image's columns only, kept
    // transposed in d_tgrid [nf3][ny][nf2]
    CU_TRY(kalloc(p, &p->d_tgrid, (size_t)gp.nf3 * p->ny * gp.nf2 * 2 * esize, st));
    const long long nxrows = (long long)gp.nf2 * gp.nf3, nyrows = (long long)p->ny * gp.nf3;
    p->fft_hx_rest = p->fft_hy_rest = 0;
    p->fft_wx = p->fft_wx_rest = p->fft_wy = p->fft_wy_rest = 0;
    if (!p->fx.n) {
        p->fft_bx = (int)std::max(1LL, std::min(nxrows, (1LL << 28) / gp.nf1));
        p->fft_bx_rest = (int)(nxrows % p->fft_bx);
        if (fft_plan1(p, gp.nf1, 1, gp.nf1, p->fft_bx, pr, p->fft_hx, p->fft_wx)) return ERR_CUFFT;
        if (p->fft_bx_rest &&
            fft_plan1(p, gp.nf1, 1, gp.nf1, p->fft_bx_rest, pr, p->fft_hx_rest, p->fft_wx_rest))
            return ERR_CUFFT;
    }
    if (!p->fy.n) {
        p->fft_by = (int)std::max(1LL, std::min(nyrows, (1LL << 28) / gp.nf2));
        p->fft_by_rest = (int)(nyrows % p->fft_by);
        if (fft_plan1(p, gp.nf2, 1, gp.nf2, p->fft_by, pr, p->fft_hy, p->fft_wy)) return ERR_CUFFT;
        if (p->fft_by_rest &&
            fft_plan1(p, gp.nf2, 1, gp.nf2, p->fft_by_rest, pr, p->fft_hy_rest, p->fft_wy_rest))
            return ERR_CUFFT;
    }
    // only this library's passes know the window; the library's rows take whole planes
    p->win_x[0] = p->win_y[0] = 0;
    p->win_x[1] = gp.nf1;
    p->win_y[1] = gp.nf2;
    if (p->fx.n && p->fy.n) {
        double r[4] = {INFINITY, -INFINITY, INFINITY, -INFINITY};      // u, v in cycles per pixel, all channels
        for (int c = 0; c < nchan; ++c)
            for (int k = 0; k < 2; ++k) {
                const double u = key_to_double(hk[2 + k]) * foc[c] * p->psx, v = key_to_double(hk[4 + k]) * foc[c] * p->psy;
                r[0] = std::min(r[0], u);
                r[1] = std::max(r[1], u);
                r[2] = std::min(r[2], v);
                r[3] = std::max(r[3], v);
            }
        axis_window(r[0], r[1], gp.nf2, gp.kp.kw, p->win_y);
        axis_window(r[2], r[3], gp.nf1, gp.kp.kw, p->win_x);
    }
    p->geom_ready = true;
    return OK;
}

// Tiles, bins, the sort and the per-visibility records, on stream st (the
// plan's stream, or a second stream that the caller joins before executing).
int plan_setpts_bin(Plan *p, cudaStream_t st) {
    if (!p || !p->geom_ready) return ERR_ARG;
    const int esize = p->opt.precision ? 4 : 8;
    const long long nrow = p->nrow;
    const int nchan = p->nchan;
    const long long M = nrow * nchan;
    const double *du = p->du, *dv = p->dv, *dw = p->dw;
    const int stride = p->stride;
    int herr = 0, s;
    mark(p, EV_SET_WRANGE);
    bool force_slabs = false;
retry_tiles:
    s = choose_tiles(p, esize, force_slabs);
    if (s != OK) return s;
    const GridParams &gp = p->gp;
    const TileGeom &tg = p->tg;
    p->smem = tg.smem_bytes;
    {
        TileGeom ti = tg;
        ti.fix = 0;
        p->smem_interp = tile_smem_bytes(ti, esize, gp.kp.kw, p->win.kind ? p->win.degree : 0);
    }

    DevGeom &g = p->dg;
    g = DevGeom{};
    g.dbg = p->d_err;                                   // index checks of the bounds-checked build
    g.nf1 = gp.nf1; g.nf2 = gp.nf2; g.nf3 = gp.nf3;
    g.kw = gp.kp.kw; g.hkw = gp.kp.kw / 2;
    g.bx = tg.bx; g.by = tg.by; g.bz = tg.bz; g.nbx = tg.nbx; g.nby = tg.nby; g.nbz = tg.nbz;
    g.ibx = 1.0 / tg.bx; g.iby = 1.0 / tg.by; g.ibz = tg.bz > 0 ? 1.0 / tg.bz : 0.0;
    g.tx = tg.tx; g.ty = tg.ty; g.tz = tg.tz; g.zpad = tg.zpad; g.sub = tg.sub;
    const int sp = p->opt.sparse;
    g.sparse_n = sp < 0 ? 0 : sp > 0 ? sp : esize == 4 ? DEFAULT_SPARSE_N : DEFAULT_SPARSE_N64;
    const int si = g_sparse_interp.load();
    p->sparse_i = sp < 0 ? 0 : si >= 0 ? si : DEFAULT_SPARSE_I;   // (sp's positive values are the spreader's)
    g.tpitch = (tg.tx + 2) & ~1;
    g.use_tma = 0;                          // set once the grid's TMA descriptor exists
    g.tma_polls = g_tma_polls.load();
    g.tma_test_noissue = g_tma_noissue.load();
    // row slabs (tile kernels only): bins of slab k are k * nbins_slab + bin
    int nslab = std::max(1, std::min(p->opt.slabs, MAX_SLABS));
    const bool tab = tabulated(p);
    if (!tab || nrow < nslab || (long long)nslab * tg.nbins() > INT_MAX / 2) nslab = 1;
    p->nslab = nslab;
    g.nslab = nslab;
    g.nbins_slab = tg.nbins();
    g.nbins = nslab * tg.nbins();
    g.sub_lo = g.sub_hi = 0;
    p->slab_row.resize(nslab + 1);
    for (int k = 0; k <= nslab; ++k) p->slab_row[k] = slab_first_row(nrow, nslab, k);
    g.beta = gp.kp.beta; g.c = gp.kp.c;
    g.wkind = p->win.kind; g.wdeg = p->win.kind ? p->win.degree : 0;
    g.smode = tile_mode(p);
    g.no_w = gp.no_w;
    // window table for the thread-per-visibility kernels: the learned window, in
    // FP32 the ES window as degree-(TAB_DEG-1) Horner polynomials, in FP64 its
    // inner intervals at degree TAB64_DEG-1
    p->wtab.reset();
    if (tab) {
        if (p->win.kind == 1) p->wtab = learned_table(p->win);
        else p->wtab = es_table(gp.kp, p->opt.precision != 0);
        if (p->win.kind == 1 || p->opt.precision) g.wkind = 1;
    }
    // bounds on the window (sampled table maxima, 1% margin): per tap index d
    // over all offsets (wenv), of one tap's product (wmax3) and of the z factor;
    // they set the scale of the one-word fixed-point spreader
    g.wmax3 = 8.0f;
    g.wzmax = g.no_w ? 1.0f : 2.0f;
    for (int d = 0; d < TAB_KW; ++d) g.wenv[d] = 2.0f;
    if (p->wtab && !p->wtab->bound.empty()) {
        double wm = 0.0;
        for (int d = 0; d < g.kw; ++d) {
            g.wenv[d] = (float)(p->wtab->bound[d] * 1.01);
            wm = std::max(wm, p->wtab->bound[d]);
        }
        g.wmax3 = (float)(std::max(wm * wm, wm * wm * wm) * 1.01);   // 2-D: two factors
        if (!g.no_w) g.wzmax = (float)(wm * 1.01);
    }
    g.nrow = nrow; g.nchan = nchan; g.uvw_stride = stride;
    g.psx = gp.pixsize_x; g.psy = gp.pixsize_y; g.i_center = gp.i_center; g.gamma = gp.gamma;
    g.o_center = gp.o_center; g.sign = (double)gp.sign;

    // binning: key per visibility (bin, start-cell residue) and its count, a
    //    scan of the counts, per-bin bounds and sub-problems, the scatter of the
    //    input indices into bin order, then records in bin order (replaces the
    //    transpose and the unsorted point order of the reference)
    const long long nb = g.nbins;
    int binbits = 1;
    while ((1LL << binbits) < nb) ++binbits;
    // start-cell residue in the key: mod 16 for the FP32 tile kernels (their
    // class schedule needs it), mod 32 for the FP64 ones (bin-only keys beyond 31 bits)
    const bool f32tile = esize == 4 && tab;
    int cbits = f32tile ? 4 : (binbits + 5 <= 31 ? 5 : 0);
    if (binbits > 31 || binbits + cbits > 31) return ERR_UNSUPPORTED;
    g.cbits = cbits;
    const long long nkeys = nb << cbits;
    // the keys and the bin-ordered indices live in the amplitudes' buffer, which
    // the binning does not need (8 bytes per visibility at least)
    CU_TRY(kalloc(p, &p->d_cs, M * 2 * (size_t)esize, st));
    p->d_keys_in = static_cast<unsigned *>(p->d_cs);
    p->d_tmp = reinterpret_cast<int *>(p->d_keys_in + M);
    CU_TRY(kalloc(p, &p->d_kcount, nkeys * sizeof(int), st));
    CU_TRY(kalloc(p, &p->d_bins, (5 * nb + std::max(scan_temp_ints(nkeys), scan_temp_ints(nb))) * sizeof(int), st));
    p->d_bin_start = p->d_bins;
    p->d_bin_count = p->d_bin_start + nb;
    p->d_nsub = p->d_bin_count + nb;
    p->d_sub_end = p->d_nsub + nb;
    p->d_bcur = p->d_sub_end + nb;
    p->d_scan = p->d_bcur + nb;
    CU_TRY(cudaMemsetAsync(p->d_kcount, 0, nkeys * sizeof(int), st));
    // few visibilities: their ranks now, records straight from input order later
    const bool ranked = M * (7LL * esize) <= g_ranked_bytes.load();
    launch_bin_count(g, du, dv, dw, p->d_foc, p->d_keys_in, ranked ? p->d_tmp : nullptr, p->d_kcount, p->d_err, st);
    scan_ints(p->d_kcount, p->d_kcount, nkeys, false, p->d_scan, st);          // in place: first position per key
    launch_bins_from_keys(p->d_kcount, p->d_scan, nb, cbits, g.sub, p->d_bin_start, p->d_bin_count, p->d_nsub,
                          p->d_bcur, st);
    if (!ranked) launch_bin_scatter(M, p->d_keys_in, cbits, p->d_bcur, p->d_tmp, st);
    scan_ints(p->d_nsub, p->d_sub_end, nb, true, p->d_scan, st);
    p->slab_sub_end.assign(nslab, 0);               // last sub-problem end of every slab
    for (int k = 0; k < nslab; ++k)
        CU_TRY(cudaMemcpyAsync(&p->slab_sub_end[k], p->d_sub_end + (k + 1) * g.nbins_slab - 1, sizeof(int),
                               cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaMemcpyAsync(&herr, p->d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    CU_TRY(cudaGetLastError());
    if (herr & EF_NONFINITE) return ERR_NONFINITE;
    if (herr & EF_BOUNDS) {
        p->last_error = "an index left its buffer (bounds-checked build)";
        return ERR_GENERIC;
    }
    if (herr & EF_RANGE) {
        if (p->tg.zpad == 0 && !force_slabs) {          // a w support reached the grid edge: use z slabs
            force_slabs = true;
            herr = 0;
            CU_TRY(cudaMemsetAsync(p->d_err, 0, sizeof(int), st));
            goto retry_tiles;
        }
        return ERR_GENERIC;
    }
    CU_TRY(kalloc(p, &p->d_rec, M * 4 * (size_t)esize, st));
    CU_TRY(kalloc(p, &p->d_ph, M * 2 * (size_t)esize, st));
    CU_TRY(kalloc(p, &p->d_idx, M * sizeof(int), st));
    // each bin's visibilities (tmp) placed by residue; the key cursors start at
    // the scanned key counts
    if (ranked && p->opt.precision)
        launch_records_ranked<float>(g, du, dv, dw, p->d_foc, p->d_keys_in, p->d_tmp, p->d_kcount, M, p->d_rec,
                                     p->d_ph, p->d_idx, st);
    else if (ranked)
        launch_records_ranked<double>(g, du, dv, dw, p->d_foc, p->d_keys_in, p->d_tmp, p->d_kcount, M, p->d_rec,
                                      p->d_ph, p->d_idx, st);
    else if (p->opt.precision)
        launch_records<float>(g, du, dv, dw, p->d_foc, p->d_tmp, M, p->d_kcount, p->d_rec, p->d_ph, p->d_idx, st);
    else
        launch_records<double>(g, du, dv, dw, p->d_foc, p->d_tmp, M, p->d_kcount, p->d_rec, p->d_ph, p->d_idx, st);
    p->d_keys_in = nullptr;
    p->d_tmp = nullptr;
    // the key cursors now hold the end of every (bin, residue) run: the class
    // boundaries of the FP32 tile kernels; every sub-problem's bin
    // (ranked: the array still holds every run's start, the next run's end)
    g.ccls = f32tile ? p->d_kcount + (ranked ? 1 : 0) : nullptr;
    const int nsubs = p->slab_sub_end.empty() ? 0 : p->slab_sub_end.back();
    g.cbin = nullptr;
    if (nsubs > 0) {
        CU_TRY(kalloc(p, &p->d_cbin, ((size_t)nsubs + nsubs / 8) * sizeof(int), st));   // (other points: about as many)
        launch_chunk_bins(nb, p->d_sub_end, p->d_cbin, st);
        g.cbin = p->d_cbin;
    }
    // TMA descriptor of the grid for the interpolator's interior tile boxes
    // ({tpitch, ty, tz} cells in 8-byte elements: one per FP32 cell, two per
    // FP64 cell; box edges <= 256 elements, x starts 16-byte aligned)
    if (g.tpitch * (p->opt.precision ? 1 : 2) <= 256 && g.ty <= 256 && g.tz <= 256)
        g.use_tma = encode_grid_map(p) == OK ? 1 : 0;
    mark(p, EV_SET_END);
    p->ready = true;
    return OK;
}

int plan_setpts(Plan *p, long long nrow, int nchan, const double *du, const double *dv,
                const double *dw, int stride, const double *h_freq) {
    auto both = [&] {
        const int s = plan_setpts_geometry(p, nrow, nchan, du, dv, dw, stride, h_freq);
        return s != OK ? s : plan_setpts_bin(p, p->st);
    };
    const bool held = p && p->d_grid;
    int s = both();
    if (s == ERR_NOMEM && held) {                  // without what the last points left behind
        plan_release_points(p);
        s = both();
    }
    // without points (unless the arguments were refused, which leaves the last
    // ones) the plan holds no memory either
    if (s != OK && p && !p->ready) plan_release_points(p);
    return s;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no -lcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void *f = nullptr;                            // initialised once, thread-safe
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
        return nullptr;
    }();
    return fn;
}

static int encode_grid_map(Plan *p) {
    auto enc = tensor_map_encoder();
    if (!enc) return ERR_UNSUPPORTED;
    const GridParams &gp = p->gp;
    const DevGeom &g = p->dg;
    // 8-byte elements: one complex cell in FP32, one component in FP64 (a cell = 2 elements)
    const int per = p->opt.precision ? 1 : 2;
    cuuint64_t dims[3] = {(cuuint64_t)gp.nf1 * per, (cuuint64_t)gp.nf2, (cuuint64_t)gp.nf3};
    cuuint64_t strides[2] = {(cuuint64_t)gp.nf1 * per * 8, (cuuint64_t)gp.nf1 * gp.nf2 * per * 8};
    cuuint32_t box[3] = {(cuuint32_t)(g.tpitch * per), (cuuint32_t)g.ty, (cuuint32_t)g.tz};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(&p->tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, p->d_grid, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? OK : ERR_UNSUPPORTED;
}

static int fft_exec(Plan *p, cufftHandle h, void *base, long long offset, int dir) {
    if (cufftSetStream(h, p->st) != CUFFT_SUCCESS) return ERR_CUFFT;
    cufftResult r;
    if (p->opt.precision) {
        cufftComplex *d = reinterpret_cast<cufftComplex *>(base) + offset;
        r = cufftExecC2C(h, d, d, dir);
    } else {
        cufftDoubleComplex *d = reinterpret_cast<cufftDoubleComplex *>(base) + offset;
        r = cufftExecZ2Z(h, d, d, dir);
    }
    return r == CUFFT_SUCCESS ? OK : ERR_CUFFT;
}

// Batched contiguous row transforms of length n over nrows rows of buf, with
// one work area from the stream-ordered pool for the pass.
static int fft_rows(Plan *p, void *buf, long long nrows, int n, cufftHandle h, size_t wh, int b,
                    cufftHandle h_rest, size_t wr, int b_rest, int dir) {
    const size_t ws = std::max(wh, h_rest ? wr : (size_t)0);
    void *work = nullptr;
    if (ws) CU_TRY(alloc_async(&work, ws, p->st));
    int s = OK;
    if (cufftSetWorkArea(h, work) != CUFFT_SUCCESS || (h_rest && cufftSetWorkArea(h_rest, work) != CUFFT_SUCCESS))
        s = ERR_CUFFT;
    for (long long r = 0; s == OK && r < nrows;) {
        const bool full = nrows - r >= b;
        s = fft_exec(p, full ? h : h_rest, buf, r * n, dir);
        r += full ? b : b_rest;
    }
    if (work) cudaFreeAsync(work, p->st);
    return s;
}

// 2-D transform of every plane (cuft.cu:127-143) restricted to what the image
// needs.  ms2dirty: x rows of the grid, their image columns transposed into
// d_tgrid, y rows there (the correction reads the image rows).  dirty2ms: the
// correction writes the image rows of d_tgrid, y rows are transformed (zeros
// outside the image rows), the columns go back into the grid's rows (zeros
// outside the image columns), which are transformed along x.  A length without
// a row pass of its own (fft_make_plan) takes cuFFT rows, separate transposes
// and stored zeros.
template <typename T>
static int plane_fft(Plan *p, int dir, bool m2d) {
    const GridParams &gp = p->gp;
    const long long nx_rows = (long long)gp.nf2 * gp.nf3, ny_rows = (long long)p->ny * gp.nf3;
    FftGeom fg{p->nx, p->ny, gp.nf1, gp.nf2, gp.nf3, p->win_x[0], p->win_x[1], p->win_y[0], p->win_y[1]};
#ifdef CURIG_BOUNDS_CHECK
    fg.dbg = p->d_err;
#endif
    const char *twx = static_cast<const char *>(p->d_tw);
    const char *twy = twx ? twx + (size_t)p->fx.tw_len * 16 : nullptr;
    auto lib_x = [&] {
        return fft_rows(p, p->d_grid, nx_rows, gp.nf1, p->fft_hx, p->fft_wx, p->fft_bx, p->fft_hx_rest, p->fft_wx_rest,
                        p->fft_bx_rest, dir);
    };
    auto lib_y = [&] {
        return fft_rows(p, p->d_tgrid, ny_rows, gp.nf2, p->fft_hy, p->fft_wy, p->fft_by, p->fft_hy_rest, p->fft_wy_rest,
                        p->fft_by_rest, dir);
    };
    int s = OK;
    if (m2d) {
        if (p->fx.n) {
            s = launch_fft_pass<T>(X_M2D, p->fx, fg, twx, p->d_grid, p->d_tgrid, p->st);
        } else if ((s = lib_x()) == OK) {
            launch_cols_to_t<T>(p->ny, gp.nf1, gp.nf2, gp.nf3, p->d_grid, p->d_tgrid, p->st);
        }
        if (s) return s;
        return p->fy.n ? launch_fft_pass<T>(Y_M2D, p->fy, fg, twy, p->d_tgrid, p->d_tgrid, p->st) : lib_y();
    }
    s = p->fy.n ? launch_fft_pass<T>(Y_D2M, p->fy, fg, twy, p->d_tgrid, p->d_tgrid, p->st) : lib_y();
    if (s) return s;
    if (p->fx.n) return launch_fft_pass<T>(X_D2M, p->fx, fg, twx, p->d_tgrid, p->d_grid, p->st);
    launch_t_to_grid<T>(p->ny, gp.nf1, gp.nf2, gp.nf3, p->d_tgrid, p->d_grid, p->st);
    return lib_x();
}

// Zeroes the grid's window.  One fill of the whole grid beats rows of a window
// that is most of it (eight 2048^2 grids, 0.94 of each side: 566 against 624 us).
template <typename T>
static cudaError_t zero_grid(Plan *p) {
    const GridParams &gp = p->gp;
    const double part = (double)(p->win_x[1] - p->win_x[0]) * (p->win_y[1] - p->win_y[0]) / ((double)gp.nf1 * gp.nf2);
    if (part > 0.85)
        return cudaMemsetAsync(p->d_grid, 0, (size_t)gp.nf1 * gp.nf2 * gp.nf3 * 2 * sizeof(T), p->st);
    launch_zero_window<T>(gp.nf1, gp.nf2, gp.nf3, p->win_x[0], p->win_x[1], p->win_y[0], p->win_y[1], p->d_grid, p->d_err,
                          p->st);
    return cudaSuccess;
}

template <typename T>
static int execute_t(Plan *p, int type, void *d_vis, const void *d_wgt, void *d_dirty) {
    cudaStream_t st = p->st;
    const DevGeom &g = p->dg;
    const GridParams &gp = p->gp;
    const long long M = p->nrow * p->nchan;
    int s;
    if (type == 1) {
        mark(p, EV_M2D_BEGIN);
        bool own;
        void *vw = gather_scratch<T>(p, d_wgt, M, own);   // vis * wgt in input order
        launch_vis_prep<T>(0, M, p->d_idx, p->d_ph, d_vis, d_wgt, vw, p->d_cs, st);
        if (own) dfree(vw, st);
        mark(p, EV_M2D_PREP);
        CU_TRY(zero_grid<T>(p));
        mark(p, EV_M2D_ZERO);
        const VisIO io{p->d_idx, p->d_ph, d_wgt, d_vis};
        s = launch_spread<T>(g, p->smem, p->d_bin_start, p->d_bin_count, p->d_sub_end, p->d_rec, p->d_cs,
                             p->d_grid, p->d_wcoef, p->wtab ? p->wtab->c.data() : nullptr, io, M, p->nsm,
                             st);
        if (s) return s;
        mark(p, EV_M2D_SPREAD);
        s = plane_fft<T>(p, CUFFT_INVERSE, true);    // +1, cuft.cu:127-143
        if (s) return s;
        mark(p, EV_M2D_FFT);
        if (p->fz.n) {
            if ((s = launch_fft_z<T>(true, p->fz, p->dc, p->d_twz, p->d_tgrid, d_dirty, st))) return s;
        } else if (p->opt.n3 > 0) launch_correct3_m2d<T>(p->dc, p->d_tgrid, d_dirty, st);
        else launch_correct_m2d<T>(p->dc, p->d_tgrid, d_dirty, st);
        mark(p, EV_M2D_END);
    } else {
        mark(p, EV_D2M_BEGIN);
        if (!p->fy.n) launch_zero_tpad<T>(p->nx, p->ny, gp.nf2, gp.nf3, p->d_tgrid, st);
        if (p->fz.n) {
            if ((s = launch_fft_z<T>(false, p->fz, p->dc, p->d_twz, d_dirty, p->d_tgrid, st))) return s;
        } else if (p->opt.n3 > 0) launch_correct3_d2m<T>(p->dc, d_dirty, p->d_tgrid, st);
        else launch_correct_d2m<T>(p->dc, d_dirty, p->d_tgrid, st);
        mark(p, EV_D2M_CORRECT);
        s = plane_fft<T>(p, CUFFT_FORWARD, false);   // -1
        if (s) return s;
        mark(p, EV_D2M_FFT);
        const VisIO io{p->d_idx, p->d_ph, nullptr, d_vis};   // weights applied after the scatter
        DevGeom gi = g;
        gi.sparse_n = p->sparse_i;
        s = launch_interp<T>(gi, p->smem_interp, p->d_bin_start, p->d_bin_count, p->d_sub_end, p->d_rec, p->d_grid,
                             p->d_cs, p->d_wcoef, p->wtab ? p->wtab->c.data() : nullptr, io, M, &p->tmap,
                             p->d_err, p->nsm, st);
        if (s) return s;
        mark(p, EV_D2M_INTERP);                  // the scatter runs inside the interpolator
        launch_vis_scale<T>(0, M, d_vis, d_wgt, st);
        mark(p, EV_D2M_END);
    }
    CU_TRY(cudaGetLastError());
    return OK;
}

template <typename T>
static int execute_slabs_t(Plan *p, int type, void *d_vis, const void *d_wgt, void *d_dirty,
                           const cudaEvent_t *ready, const cudaEvent_t *done, int nev, bool prologue_done) {
    cudaStream_t st = p->st;
    const GridParams &gp = p->gp;
    const int ns = p->nslab;
    if (nev != ns && !(ns == 1 && nev > 0)) return ERR_ARG;
    auto wait_slab = [&](int k) {
        if (!ready) return cudaSuccess;
        if (ns == nev) return cudaStreamWaitEvent(st, ready[k], 0);
        for (int e = 0; e < nev; ++e) {               // one plan slab: every upload
            cudaError_t r = cudaStreamWaitEvent(st, ready[e], 0);
            if (r != cudaSuccess) return r;
        }
        return cudaSuccess;
    };
    auto done_slab = [&](int k) {
        if (!done) return cudaSuccess;
        if (ns == nev) return cudaEventRecord(done[k], st);
        for (int e = 0; e < nev; ++e) {
            cudaError_t r = cudaEventRecord(done[e], st);
            if (r != cudaSuccess) return r;
        }
        return cudaSuccess;
    };
    // launch geometry of slab k: its sub-problem window
    auto slab_geom = [&](int k, DevGeom &gk) {
        gk = p->dg;
        gk.sub_lo = k ? p->slab_sub_end[k - 1] : 0;
        gk.sub_hi = p->slab_sub_end[k];
        return gk.sub_hi > gk.sub_lo;
    };
    const VisIO io{p->d_idx, p->d_ph, d_wgt, d_vis};
    const double *ht = p->wtab ? p->wtab->c.data() : nullptr;
    int s;
    if (type == 1) {
        CU_TRY(zero_grid<T>(p));
        bool own;
        void *vw = gather_scratch<T>(p, d_wgt, p->nrow * p->nchan, own);   // vis * wgt in input order
        for (int k = 0; k < ns; ++k) {
            if (cudaError_t e = wait_slab(k)) {
                if (own) dfree(vw, st);
                CU_TRY(e);
            }
            const long long i0 = p->slab_row[k] * p->nchan, i1 = p->slab_row[k + 1] * p->nchan;
            launch_vis_prep<T>(i0, i1 - i0, p->d_idx, p->d_ph, d_vis, d_wgt, vw, p->d_cs, st);
            DevGeom gk;
            if (slab_geom(k, gk) &&
                (s = launch_spread<T>(gk, p->smem, p->d_bin_start, p->d_bin_count, p->d_sub_end, p->d_rec, p->d_cs,
                                      p->d_grid, p->d_wcoef, ht, io, p->nrow * p->nchan, p->nsm, st))) {
                if (own) dfree(vw, st);
                return s;
            }
        }
        if (own) dfree(vw, st);
        if ((s = plane_fft<T>(p, CUFFT_INVERSE, true))) return s;
        launch_correct_m2d<T>(p->dc, p->d_tgrid, d_dirty, st);
    } else {
        if (!prologue_done) {
            if (!p->fy.n) launch_zero_tpad<T>(p->nx, p->ny, gp.nf2, gp.nf3, p->d_tgrid, st);
            launch_correct_d2m<T>(p->dc, d_dirty, p->d_tgrid, st);
            if ((s = plane_fft<T>(p, CUFFT_FORWARD, false))) return s;
        }
        const VisIO io_out{p->d_idx, p->d_ph, nullptr, d_vis};   // weights applied after the scatter
        for (int k = 0; k < ns; ++k) {
            CU_TRY(wait_slab(k));
            DevGeom gk;
            const bool some = slab_geom(k, gk);
            gk.sparse_n = p->sparse_i;
            if (some &&
                (s = launch_interp<T>(gk, p->smem_interp, p->d_bin_start, p->d_bin_count, p->d_sub_end, p->d_rec,
                                      p->d_grid, p->d_cs, p->d_wcoef, ht, io_out, p->nrow * p->nchan, &p->tmap,
                                      p->d_err, p->nsm, st)))
                return s;
            const long long i0 = p->slab_row[k] * p->nchan, i1 = p->slab_row[k + 1] * p->nchan;
            launch_vis_scale<T>(i0, i1 - i0, d_vis, d_wgt, st);
            CU_TRY(done_slab(k));
        }
    }
    CU_TRY(cudaGetLastError());
    return OK;
}

int plan_execute_slabs(Plan *p, int type, void *d_vis, const void *d_wgt, void *d_dirty,
                       const cudaEvent_t *ready, const cudaEvent_t *done, int nev, bool prologue_done) {
    if (!p || !p->ready || !d_vis || !d_dirty || (type != 1 && type != 2)) return ERR_ARG;
    return p->opt.precision
               ? execute_slabs_t<float>(p, type, d_vis, d_wgt, d_dirty, ready, done, nev, prologue_done)
               : execute_slabs_t<double>(p, type, d_vis, d_wgt, d_dirty, ready, done, nev, prologue_done);
}

template <typename T>
static int d2m_prologue_t(Plan *p, const void *d_dirty, cudaEvent_t image_ready) {
    const GridParams &gp = p->gp;
    if (!p->fy.n) launch_zero_tpad<T>(p->nx, p->ny, gp.nf2, gp.nf3, p->d_tgrid, p->st);   // needs no image
    if (image_ready) CU_TRY(cudaStreamWaitEvent(p->st, image_ready, 0));
    launch_correct_d2m<T>(p->dc, d_dirty, p->d_tgrid, p->st);
    int s = plane_fft<T>(p, CUFFT_FORWARD, false);
    if (s) return s;
    CU_TRY(cudaGetLastError());
    return OK;
}

int plan_d2m_prologue(Plan *p, const void *d_dirty, cudaEvent_t image_ready) {
    if (!p || !p->geom_ready || !d_dirty) return ERR_ARG;
    return p->opt.precision ? d2m_prologue_t<float>(p, d_dirty, image_ready)
                            : d2m_prologue_t<double>(p, d_dirty, image_ready);
}

// Error flags raised by kernels of earlier executes (an interpolator tile load
// that never completed); waits for the plan's stream.
int plan_device_status(Plan *p) {
    if (!p || !p->d_err) return OK;
    int herr = 0;
    CU_TRY(cudaMemcpyAsync(&herr, p->d_err, sizeof(int), cudaMemcpyDeviceToHost, p->st));
    CU_TRY(cudaStreamSynchronize(p->st));
    if (herr & EF_TIMEOUT) {
        p->last_error = "a tile load did not complete (timed out)";
        return ERR_CUDA;
    }
    if (herr & EF_BOUNDS) {
        p->last_error = "an index left its buffer (bounds-checked build)";
        return ERR_GENERIC;
    }
    return OK;
}

int plan_execute(Plan *p, void *d_vis, const void *d_wgt, void *d_dirty, int type) {
    if (!p || !p->ready || !d_vis || !d_dirty) return ERR_ARG;
    if (type == 0) type = p->type;
    if (type != 1 && type != 2) return ERR_ARG;
    return p->opt.precision ? execute_t<float>(p, type, d_vis, d_wgt, d_dirty)
                            : execute_t<double>(p, type, d_vis, d_wgt, d_dirty);
}

}  // namespace curig
