// ymkh_capi.cu — the extern "C" boundary of include/ymkh.h: context
// lifetime, state binding, the step sequence and the diagnostics.
//
// The step keeps the reference's stage order (ymgpu2d/main_ym.cu:324-455):
//   FCT x+z sweeps of both beams, density floor   -> fct_strip_kernel / fct_fused_kernel
//   currents, Ampère, potential, Faraday          -> maxwell_fused_kernel
//   sponge, xi_cut                                -> sponge_xicut_kernel
//   z-mean removal and colour-1 EM zeroing        -> zmean_p2_kernel / zmean_kernel
//   DFT kz bands on the 21 filtered arrays        -> band_coef / band_apply
//   z-hyperdiffusion                              -> hyperdiff_kernel
// (the stages from the sponge on in one launch of column_kernel, where
// col_fused_alone and the batch say so).
// The sources of stage 7 are recomputed inside the next FCT launch.
//
// The stencil kernels read start-of-step values of neighbouring tiles, so
// the state alternates between two 24-array buffers: buffer 0 is the state
// the caller binds; buffer 1 is either a second caller-bound set
// (ymkh_bind_state2, zero copy) or allocated here once.  With a library
// buffer, ymkh_step copies back when it ends on buffer 1, so the caller's
// arrays always hold the current state after the call.

#include <cstdio>
#include <cstring>
#include <cstdarg>
#include <atomic>
#include <exception>
#include <memory>
#include <mutex>
#include <vector>
#include <algorithm>
#include "ymkh_common.cuh"

#include <cuda.h>
#include <nvtx3/nvToolsExt.h>


using namespace ymkh;

namespace {

thread_local int t_err_code = 0;
thread_local char t_err_msg[512] = "";
std::atomic<long long> g_launches{0};

int set_err(int code, const char* fmt, ...) {
  t_err_code = code;
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(t_err_msg, sizeof t_err_msg, fmt, ap);
  va_end(ap);
  return code;
}

// NVTX range for the host timeline of a profiler (header-only NVTX 3: a
// no-op unless a tool is attached).
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
};

#define CK(call, what)                                                                    \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess) return set_err(YMKH_ECUDA, "%s: %s", what, cudaGetErrorString(e_)); \
  } while (0)

// Ends an entry point written as a function-try-block: no exception (a host
// allocation that fails) leaves the C boundary.
#define YMKH_CATCH                                                                          \
  catch (const std::exception& e_) { return set_err(YMKH_ENOMEM, "host: %s", e_.what()); } \
  catch (...) { return set_err(YMKH_ENOMEM, "host exception"); }

constexpr int MAX_BANDS = kMaxBands;
constexpr int kMaxFctCtas = 512;

// Pages of pinned host memory that the diagnostics' last kernels write their
// results to, one slot of 32 doubles per context: reading a result back is
// then the stream's synchronisation alone, where a copy to the caller's
// pageable memory is staged and synchronised by itself.  Slots come from
// 64 KiB slabs shared by all contexts of the process (any device, any
// thread); a slab whose slots are all given back is freed, but for one kept.
class HostSlots {
 public:
  static constexpr int kDoubles = 32, kPerSlab = 256;
  double* take() try {
    std::lock_guard<std::mutex> lock(mu_);
    for (Slab& s : slabs_)
      if (s.used < kPerSlab)
        for (int i = 0; i < kPerSlab; ++i)
          if (!s.taken[i]) return give_out(s, i);
    void* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(double) * kDoubles * kPerSlab, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
      return nullptr;
    struct Free {
      void operator()(void* q) const { cudaFreeHost(q); }
    };
    std::unique_ptr<void, Free> hold(p);
    slabs_.push_back(Slab{static_cast<double*>(p), 0, std::vector<char>(kPerSlab, 0)});
    hold.release();
    return give_out(slabs_.back(), 0);
  } catch (const std::bad_alloc&) {
    return nullptr;
  }
  void give_back(double* slot) {
    std::lock_guard<std::mutex> lock(mu_);
    int empty = 0;
    for (size_t k = 0; k < slabs_.size(); ++k) {
      Slab& s = slabs_[k];
      if (slot >= s.base && slot < s.base + kDoubles * kPerSlab) {
        s.taken[(slot - s.base) / kDoubles] = 0;
        --s.used;
      }
      if (!s.used && empty++) {
        cudaFreeHost(s.base);
        slabs_.erase(slabs_.begin() + k--);
      }
    }
  }

 private:
  struct Slab {
    double* base;
    int used;
    std::vector<char> taken;
  };
  double* give_out(Slab& s, int i) {
    s.taken[i] = 1;
    ++s.used;
    return s.base + (size_t)i * kDoubles;
  }
  std::mutex mu_;
  std::vector<Slab> slabs_;
};
HostSlots& host_slots() {
  static HostSlots* p = new HostSlots();  // not destroyed: contexts may outlive static objects
  return *p;
}

}  // namespace

struct ymkh_ctx {
  int device = 0;
  int nx = 0, nz = 0;
  size_t N = 0;
  ymkh_params prm{};
  StepParams sp{};
  State buf[2]{};
  bool bound = false;
  bool dual = false;         // second buffer bound by the caller
  double* own = nullptr;     // library second buffer (24*N doubles)
  int cur = 0;
  int nb = 0, lo[MAX_BANDS]{}, hi[MAX_BANDS]{}, J[MAX_BANDS]{};
  double* W[MAX_BANDS]{};
  double* coef = nullptr;    // band coefficients [21][J][nx]
  Tf32BandImages tfb[MAX_BANDS]{};  // TF32 engine: twiddle tile images per band
  Tf32Scratch tfs{};                // TF32 engine: G and C^T tile images
  double* zmeans = nullptr;         // TF32 engine with suppress_kz0: z-means the first band takes off
  double* epart = nullptr;   // energy partials
  double* hres = nullptr;    // results of the diagnostics: a slot of pinned host memory
  double* mcol = nullptr;    // mode amplitude partial sums
  double* mweight = nullptr; // x weights of ymkh_circ_amp (NX doubles, allocated on first use)
  double* gpart = nullptr;   // Gauss residual partials (allocated on first use)
  SnapshotQueue* snaps = nullptr;  // snapshot writers (created on first use)
  int fct_tx = 64, fct_seg = 16, fct_grid = 296;  // FCT threads per beam, segment rows, persistent CTAs
  int mx_seg = 16, mx_grid = 148;                   // Maxwell segment rows, persistent CTAs
  int sms = 148;
  bool aligned16 = false;   // every bound array 16-byte aligned: TMA bulk row copies allowed
  unsigned* derr = nullptr; // device error word of the bounded in-kernel waits
  // Tables of the kernels, uploaded in stream order by the next step call.
  struct Tables {
    TensorMap maps[2 * kMaps];     // kMaps of buffer 0, then of buffer 1
    RunDesc desc[2];               // run descriptors for start buffer 0 and 1
    ColDesc col[2];                // column stages writing buffer 0 and buffer 1
    int fct_first[kMaxFctCtas + 1];  // items of the fused FCT's CTAs
  };
  Tables host{};              // host copy
  Tables* dev = nullptr;      // device copy
  bool boxed = false;         // the maps encoded: evenly spaced, 16-byte aligned arrays, nx even
  bool col_ok = false;        // the column stages can run as one kernel (ymkh_colfused.cu)
  bool col_fused = false;     // and do, in a lone run
  int col_items = 0;
  size_t col_smem = 0;
  unsigned version = 0;       // of the descriptors: a batch rebuilds its tables when a member's changed
  int fct_items = 0, mx_items = 0, fx_items = 0, fz_items = 0;
  bool desc_ok = false;
  bool desc_pending = false; // host tables not yet uploaded
  int fct_mode = YMKH_FCT_FUSED;  // YMKH_FCT_FUSED or YMKH_FCT_SPLIT
  double* xscratch = nullptr;     // 12 x-swept fluid arrays of the split form
  int fz_seg = 128;
  int fx_grid = 0, fz_grid = 0;
  // CUDA graphs of `graph_steps` steps, one per starting buffer
  int graph_steps = 4;
  cudaGraphExec_t gexec[2]{nullptr, nullptr};
  cudaStream_t gstream[2]{nullptr, nullptr};
  long long glaunches[2]{0, 0};  // kernels per captured graph
  // optional per-stage event timing (ymkh_stage_times)
  cudaEvent_t ev[16]{};
  int nev = 0;
  bool timing = false;
};

namespace {

void fill_step_params(ymkh_ctx* c) {
  const ymkh_params& p = c->prm;
  StepParams& s = c->sp;
  s.nx = c->nx; s.nz = c->nz;
  s.dx = p.dx; s.dz = p.dz; s.dt = p.dt_step;
  s.rdx = 1.0 / p.dx; s.rdz = 1.0 / p.dz;  // IEEE division: correctly rounded
  s.c2 = p.c * p.c; s.eps0 = p.eps_0; s.alpha = p.alpha_YM;
  s.freeze_az1 = p.freeze_az1; s.periodic_x = p.periodic_x;
  s.epsilon = p.epsilon; s.xi_sponge = p.xi_sponge; s.sigma_sponge = p.sigma_sponge;
  s.xi_cut = p.xi_cut; s.warm_T = p.warm_T; s.suppress_kz0 = p.suppress_kz0;
  s.hyp_diff = p.hyp_diff_coeff;
}

int band_list(const ymkh_params& p, int* lo, int* hi) {
  int n = 0;
  if (p.kz_suppress_max >= 1) { lo[n] = 1; hi[n] = p.kz_suppress_max; ++n; }
  if (p.kz_suppress_hi > p.kz_suppress_max + 1) { lo[n] = p.kz_suppress_max + 2; hi[n] = p.kz_suppress_hi; ++n; }
  for (int i = 0; i < p.n_extra_bands && i < YMKH_MAX_EXTRA_BANDS; ++i) {
    lo[n] = p.extra_band_lo[i]; hi[n] = p.extra_band_hi[i]; ++n;
  }
  return n;
}

void drop_graphs(ymkh_ctx* c) {
  for (int k = 0; k < 2; ++k)
    if (c->gexec[k]) { cudaGraphExecDestroy(c->gexec[k]); c->gexec[k] = nullptr; c->gstream[k] = nullptr; }
}

void free_bands(ymkh_ctx* c) {
  for (int b = 0; b < MAX_BANDS; ++b) {
    if (c->W[b]) { cudaFree(c->W[b]); c->W[b] = nullptr; }
    for (float** q : {&c->tfb[b].a1h, &c->tfb[b].a1l, &c->tfb[b].a2h, &c->tfb[b].a2l})
      if (*q) { cudaFree(*q); *q = nullptr; }
  }
  for (float** q : {&c->tfs.gh, &c->tfs.gl, &c->tfs.ch, &c->tfs.cl})
    if (*q) { cudaFree(*q); *q = nullptr; }
  if (c->coef) { cudaFree(c->coef); c->coef = nullptr; }
  if (c->zmeans) { cudaFree(c->zmeans); c->zmeans = nullptr; }
  c->nb = 0;
}

// TF32 engine set-up: twiddle tile images per band and the shared scratch.
int setup_tf32(ymkh_ctx* c) {
  CK(prepare_tf32(), "TF32 GEMM shared-memory attribute");
  const size_t zp = (size_t)tf32_zpad(c->nz);
  const size_t tf = tf32_tile_floats();
  const size_t nt = (size_t)tf32_ntiles(c->nx);
  int maxJp = 0;
  for (int b = 0; b < c->nb; ++b) {
    Tf32BandImages& t = c->tfb[b];
    t.J = c->J[b];
    t.Jp = tf32_jpad(c->J[b]);
    maxJp = std::max(maxJp, t.Jp);
    const size_t n = (size_t)t.Jp * zp;  // floats per image
    for (float** q : {&t.a1h, &t.a1l, &t.a2h, &t.a2l}) CK(cudaMalloc(q, n * sizeof(float)), "cudaMalloc TF32 twiddle images");
    CK(launch_tf32_w_images(c->W[b], c->J[b], c->J[b], c->nz, t, 0), "TF32 twiddle images");
    g_launches++;
  }
  const size_t ng = 21 * nt * (zp / 32) * tf, nc = 21 * nt * (size_t)(maxJp / 32) * tf;
  CK(cudaMalloc(&c->tfs.gh, ng * sizeof(float)), "cudaMalloc TF32 G images");
  CK(cudaMalloc(&c->tfs.gl, ng * sizeof(float)), "cudaMalloc TF32 G images");
  CK(cudaMalloc(&c->tfs.ch, nc * sizeof(float)), "cudaMalloc TF32 coefficient images");
  CK(cudaMalloc(&c->tfs.cl, nc * sizeof(float)), "cudaMalloc TF32 coefficient images");
  if (c->prm.suppress_kz0) CK(cudaMalloc(&c->zmeans, (size_t)12 * c->nx * sizeof(double)), "cudaMalloc z-means");
  return 0;
}

// Twiddles and scratch of the bands of c->prm.
int setup_bands(ymkh_ctx* c, int nb, const int* lo, const int* hi) {
  size_t maxJ = 0;
  for (int b = 0; b < nb; ++b) {
    c->lo[b] = lo[b]; c->hi[b] = hi[b]; c->J[b] = 2 * (hi[b] - lo[b] + 1);
    CK(cudaMalloc(&c->W[b], (size_t)c->nz * c->J[b] * sizeof(double)), "cudaMalloc twiddles");
    CK(launch_twiddles(c->W[b], c->nz, lo[b], hi[b], c->J[b], 0), "twiddle kernel");
    g_launches++;
    maxJ = std::max(maxJ, (size_t)c->J[b]);
  }
  c->nb = nb;
  if (nb && c->prm.filter_engine == YMKH_FILTER_TF32X3) {
    int rc = setup_tf32(c);
    if (rc) return rc;
  } else if (nb) {
    CK(cudaMalloc(&c->coef, 21 * maxJ * (size_t)c->nx * sizeof(double)), "cudaMalloc band coefficients");
  }
  // the twiddle tables and images are built on the legacy default stream:
  // wait for that stream only, not for other streams' work in flight (a
  // server creates runs while others step)
  CK(cudaStreamSynchronize(0), "twiddle setup");
  return 0;
}

int setup_params(ymkh_ctx* c, const ymkh_params* p) {
  if (p->dt_step <= 0 || p->dx <= 0 || p->dz <= 0) return set_err(YMKH_EINVAL, "dx, dz, dt_step must be > 0");
  if (p->filter_engine != YMKH_FILTER_DFT && p->filter_engine != YMKH_FILTER_TF32X3)
    return set_err(YMKH_EINVAL, "unknown filter_engine %d", p->filter_engine);
  if (p->suppress_kz0 && (c->nz & (c->nz - 1)) != 0)
    return set_err(YMKH_EINVAL, "suppress_kz0 requires NZ a power of 2 (got %d)", c->nz);
  if (p->n_extra_bands < 0 || p->n_extra_bands > YMKH_MAX_EXTRA_BANDS)
    return set_err(YMKH_EINVAL, "n_extra_bands out of range");
  int lo[MAX_BANDS], hi[MAX_BANDS];
  const int nb = band_list(*p, lo, hi);
  for (int b = 0; b < nb; ++b)
    if (lo[b] < 0 || hi[b] < lo[b] || hi[b] > 1 << 20) return set_err(YMKH_EINVAL, "bad band [%d, %d]", lo[b], hi[b]);
  drop_graphs(c);
  free_bands(c);
  // The tables of the column stages, this run's and those of a batch that it is
  // in, point at the bands just freed: they are built again before the next
  // step, also when the new bands cannot be had.
  c->desc_ok = false;
  ++c->version;
  c->prm = *p;
  fill_step_params(c);
  const int rc = setup_bands(c, nb, lo, hi);
  if (rc) {
    free_bands(c);       // no half of a band list: the run goes on without bands
    cudaGetLastError();  // reported here, not by the next launch
  }
  return rc;
}

// Maxwell's segment rows for persistent CTAs taking (strip, segment) items
// round-robin: the length whose busiest CTA has the least to do, each item
// paying kMxStart rows of start-up besides its own (two rows staged ahead, the
// pipeline's fill and the item's set-up; 2, 4 and 8 measured alike).  A row
// costs a CTA about 2 us whatever the grid, so short segments over every SM
// are what a small grid needs: against segments of at least 16 rows, 64 x 96
// took 13 us instead of 49, 256 x 512 21 instead of 37; against 128 rows in
// batches, 16 uneven runs 2.20 ms a step instead of 2.42.
constexpr int kMxStart = 4;
struct MxGrid {
  int nz, nstrips;
};
int pick_mx_segment(const MxGrid* g, int n, int grid) {
  int nz_max = 1;
  for (int i = 0; i < n; ++i) nz_max = std::max(nz_max, g[i].nz);
  int best = 1;
  long long best_cost = 1ll << 60;
  for (int nseg = 1; nseg <= nz_max; ++nseg) {
    const int seg = (nz_max + nseg - 1) / nseg;
    if (nseg > 1 && seg == (nz_max + nseg - 2) / (nseg - 1)) continue;
    long long items = 0;
    for (int i = 0; i < n; ++i) items += (long long)g[i].nstrips * ((g[i].nz + seg - 1) / seg);
    const long long rounds = (items + grid - 1) / grid, cost = rounds * (seg + kMxStart);
    if (cost < best_cost) { best_cost = cost; best = seg; }
  }
  return best;
}

// One-row segments: a CTA's contiguous block then ends at any row, so the
// blocks differ by at most one row.
constexpr int kFctSegment = 1;

void choose_launch_shape(ymkh_ctx* c) {
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->device);
  // Strip width: 128 from NX = 128 up, and from NX = 64 up with 128 rows or more;
  // below 32, where the 128-wide form's start-up shows and on narrow grids its
  // empty lanes and the many short copies of a wrapped row (FCT us, NZ x NX, 128-
  // against the better of 64- and 32-wide strips: 64 x 128 23 / 28, 256 x 512 37
  // / 52, 128 x 96 25 / 26, 512 x 96 33 / 38, 2048 x 64 73 / 80, but 64 x 96 27 /
  // 25, 32 x 48 29 / 23, 512 x 48 36 / 36, 2048 x 48 78 / 63, 2048 x 16 107 / 46,
  // 128 x 4 90 / 27; from 53 to 63 columns within a tenth of each other; element
  // copies, walls 64 x 200 28 / 31, 243 x 371 47 / 58, 1000 x 300 87 / 118, 64 x
  // 96 29 / 29, 2048 x 64 81 / 91, 2048 x 48 85 / 70, odd periodic 243 x 371 47 /
  // 53, 33 x 47 29 / 24).
  c->fct_tx = c->nx >= 128 || (c->nx >= 64 && c->nz >= 128) ? 128 : 32;
  const int fct_per_sm = std::max(1, fct_ctas_per_sm(c->fct_tx));
  c->fct_grid = c->sms * fct_per_sm;
  // segments are the FCT's unit of load balance: each CTA runs a contiguous
  // block of them, a strip's part as one piece (ymkh_fct.cu)
  c->fct_seg = std::min(c->nz, kFctSegment);
  const int mx_per_sm = std::max(1, maxwell_ctas_per_sm());
  c->mx_grid = c->sms * mx_per_sm;
  const MxGrid mg{c->nz, maxwell_nstrips(c->nx)};
  c->mx_seg = pick_mx_segment(&mg, 1, c->mx_grid);
  c->fx_grid = c->sms * std::max(1, fct_split_ctas_per_sm(0)) * 4;
  c->fz_grid = c->sms * std::max(1, fct_split_ctas_per_sm(1)) * 4;
}

// Row staging of the fused kernels when every bound array is 16-byte aligned
// and x is periodic with nx even: TMA bulk row copies issued one per thread
// across all warps (RowLoad).
constexpr int kAlignedRowLoad = LOAD_BULK_ALL;

RunDesc make_desc(const ymkh_ctx* c, int start, int tb, int fct_item0, int mx_item0) {
  RunDesc d{};
  d.in = c->buf[start];
  d.out = c->buf[1 - start];
  d.p = c->sp;
  d.fct_nstrips = fct_nstrips(c->nx, tb);
  d.fct_seg = c->fct_seg;
  d.fct_item0 = fct_item0;
  d.fct_bulk = (c->aligned16 && fct_bulk_ok(c->sp, tb)) ? kAlignedRowLoad : (int)LOAD_ELEM;
  if (tb == 128 && d.fct_bulk != LOAD_ELEM && c->boxed) {
    d.fct_bulk = LOAD_BOX;
    d.maps = c->dev->maps + kMaps * start;
  }
  d.mx_nstrips = maxwell_nstrips(c->nx);
  d.mx_seg = c->mx_seg;
  d.mx_item0 = mx_item0;
  d.mx_bulk = (c->aligned16 && maxwell_bulk_ok(c->sp)) ? kAlignedRowLoad : (int)LOAD_ELEM;
  if (d.mx_bulk != LOAD_ELEM && c->boxed) {
    d.mx_bulk = LOAD_BOX;
    d.mx_fluid = c->dev->maps + kMaps * (1 - start) + kFctMaps;
    d.mx_field = c->dev->maps + kMaps * start + kFctMaps;
  }
  if (c->xscratch)
    for (int i = 0; i < 6; ++i) {
      d.xsw.a[i] = c->xscratch + (size_t)i * c->N;
      d.xsw.b[i] = c->xscratch + (size_t)(6 + i) * c->N;
    }
  d.fx_nstrips = fctx_nstrips(c->nx);
  d.fz_ncols = fctz_ncols(c->nx);
  d.fz_seg = std::min(c->nz, c->fz_seg);
  return d;
}

int items_fx(const RunDesc& d, int nz) { return d.fx_nstrips * nz * 2; }
int items_fz(const RunDesc& d, int nz) { return d.fz_ncols * ((nz + d.fz_seg - 1) / d.fz_seg); }

// The split FCT form needs a 12-array scratch for the x-swept fluid.
int ensure_xscratch(ymkh_ctx* c) {
  if (c->fct_mode != YMKH_FCT_SPLIT || c->xscratch) return 0;
  if (cudaMalloc(&c->xscratch, (size_t)12 * c->N * sizeof(double)) != cudaSuccess)
    return set_err(YMKH_ENOMEM, "cudaMalloc x-sweep scratch (%zu bytes)", (size_t)12 * c->N * sizeof(double));
  return 0;
}

// CTAs of an FCT launch (launch_fct_table).
int fct_ctas(int items, int grid) { return std::max(1, std::min(std::min(items, grid), kMaxFctCtas)); }
int items_fct(const RunDesc& d, int nz) { return d.fct_nstrips * ((nz + d.fct_seg - 1) / d.fct_seg); }
int items_mx(const RunDesc& d, int nz) { return d.mx_nstrips * ((nz + d.mx_seg - 1) / d.mx_seg); }

// Tensor maps of both buffers for the kernels' TMA boxes: [array][z][x] with the
// distance between arrays as the outer stride, which needs the 24 arrays of a
// buffer evenly spaced in the state's order (a [24, NZ, NX] tensor, or the
// library's own buffer).  Other layouts, odd NX and unaligned arrays keep the
// per-array row copies.
bool encode_box(TensorMap* out, const State& s, int nx, int nz, int arrays, int width) {
  const double* p[24];
  for (int i = 0; i < 12; ++i) p[i] = s.f[i];
  for (int i = 0; i < 6; ++i) { p[12 + i] = s.a[i]; p[18 + i] = s.b[i]; }
  const ptrdiff_t d = p[1] - p[0];
  if (d < (ptrdiff_t)nx * nz) return false;
  for (int i = 2; i < 24; ++i) if (p[i] - p[i - 1] != d) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)nz, 24};
  const cuuint64_t strides[2] = {(cuuint64_t)nx * sizeof(double), (cuuint64_t)d * sizeof(double)};
  if (strides[0] % 16 || strides[1] % 16 || strides[1] >= (1ull << 40)) return false;
  const cuuint32_t box[3] = {(cuuint32_t)width, 1, (cuuint32_t)arrays}, es[3] = {1, 1, 1};
  static const auto encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn);
  }();
  static_assert(sizeof(CUtensorMap) == sizeof(TensorMap) && alignof(CUtensorMap) <= alignof(TensorMap), "tensor map");
  if (!encode) return false;
  return encode(reinterpret_cast<CUtensorMap*>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(p[0]), dims,
                strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The list l without its first k arrays.
ArrayList drop_front(const ArrayList& l, int k) {
  ArrayList r{};
  for (int i = 0; i + k < 24; ++i) r.p[i] = l.p[i + k];
  return r;
}

ArrayList list21(const State& s) {
  ArrayList l{};
  double* v[21] = {s.f[BY1], s.f[EX1], s.f[EZ1], s.f[BY2], s.f[BY3], s.f[EX2], s.f[EX3],
                   s.f[EZ2], s.f[EZ3], s.f[AZ2], s.f[AZ3], s.a[FQ2], s.a[FQ3], s.b[FQ2],
                   s.b[FQ3], s.a[FPZ], s.b[FPZ], s.a[FPX], s.b[FPX], s.a[FN], s.b[FN]};
  for (int i = 0; i < 21; ++i) l.p[i] = v[i];
  return l;
}
ArrayList list12(const State& s) {
  ArrayList l{};
  double* v[12] = {s.f[BY2], s.f[BY3], s.f[EX2], s.f[EX3], s.f[EZ2], s.f[EZ3],
                   s.f[AZ2], s.f[AZ3], s.a[FQ2], s.a[FQ3], s.b[FQ2], s.b[FQ3]};
  for (int i = 0; i < 12; ++i) l.p[i] = v[i];
  return l;
}

// The fused column stages' table for the run writing buffer `to`.
ColDesc make_col(const ymkh_ctx* c, int to) {
  ColDesc d{};
  const ArrayList l = list21(c->buf[to]);
  for (int i = 0; i < 21; ++i) d.arr[i] = l.p[i];
  const ymkh_params& p = c->prm;
  d.nx = c->nx; d.nz = c->nz; d.nb = c->nb;
  for (int b = 0; b < c->nb; ++b) { d.W[b] = c->W[b]; d.M[b] = c->J[b] / 2; }
  d.ncb = (c->nx + 31) / 32;
  d.sponge = p.xi_sponge > 0.0; d.cut = p.xi_cut > 0.0; d.kz0 = p.suppress_kz0 != 0; d.hyper = p.hyp_diff_coeff > 0.0;
  d.k0 = (c->nb || d.kz0) ? 0 : 3;
  d.dx = c->sp.dx; d.dt = c->sp.dt; d.epsilon = c->sp.epsilon; d.xi_sponge = c->sp.xi_sponge;
  d.sigma_sponge = c->sp.sigma_sponge; d.xi_cut = c->sp.xi_cut; d.hyp_diff = c->sp.hyp_diff;
  d.inv2 = (double)(2.0f / (float)c->nz);
  return d;
}

// Arrays the fused column stages visit: all 21 with bands, else colours 2 and
// 3 (and colour 1, to zero it, with suppress_kz0).
int col_arrays(const ColDesc& d) { return d.nb ? 21 : (d.kz0 ? 15 : 12); }

int band_modes(const ymkh_ctx* c) {  // of the widest band
  int m = 0;
  for (int b = 0; b < c->nb; ++b) m = std::max(m, c->J[b] / 2);
  return m;
}

// Whether the column stages can run as one kernel (ymkh_colfused.cu).
bool col_fused_ok(const ymkh_ctx* c) {
  const ymkh_params& p = c->prm;
  if (c->nz % 32 || c->nz > kColumnFusedMaxNz) return false;
  if (c->nb && p.filter_engine != YMKH_FILTER_DFT) return false;
  if (!c->nb && !p.suppress_kz0 && p.xi_sponge <= 0.0 && p.xi_cut <= 0.0 && p.hyp_diff_coeff <= 0.0) return false;
  return column_fused_smem(c->nz, band_modes(c), p.suppress_kz0) <= kColumnFusedSmemMax;
}

int col_stages(const ymkh_ctx* c) {
  const ymkh_params& p = c->prm;
  return (p.xi_sponge > 0.0 || p.xi_cut > 0.0) + (p.suppress_kz0 != 0) + (c->nb > 0) + (p.hyp_diff_coeff > 0.0);
}
int col_modes(const ymkh_ctx* c) {
  int m = 0;
  for (int b = 0; b < c->nb; ++b) m += c->J[b] / 2;
  return m;
}

// Whether a lone run takes that kernel: with two stages or more, or with band
// filters alone up to 128 rows.  Step us, one kernel against separate ones:
// all stages and 14 modes 64 x 768 53 / 63, 256 x 768 106 / 127, 512 x 1024 241
// / 263; bands alone 64 x 192 36 / 37, 128 x 512 57 / 63, but 256 x 512 of 43
// modes 158 / 136, 512 x 512 of 86 471 / 375 (its CTAs have a column tile each
// and end unevenly); z-mean alone 256 x 256 43 / 41, 512 x 1024 134 / 127.
// Above 48 modes and 256 rows a CTA lasts so long that what counts is how well
// its turns fill the SMs: it is taken where they nearly do (z-mean and 86 modes
// at 512 rows: 192 columns, 108 CTAs 182 / 187, 256 columns, 144 CTAs 192 / 203;
// but 40 columns, 36 CTAs 178 / 102; hyperdiffusion and 86 modes 256 columns,
// 168 CTAs 321 / 229, 1024 columns, 672 CTAs 782 / 706).
constexpr int kColWideModes = 48;
bool col_fused_alone(const ymkh_ctx* c) {
  const int stages = col_stages(c);
  if (c->nz > 256 && col_modes(c) > kColWideModes) {
    const int tiles = (c->nx + 31) / 32 * (c->prm.suppress_kz0 ? 18 : 21), turns = (tiles + c->sms - 1) / c->sms;
    return stages >= 2 && tiles * 20 >= turns * c->sms * (turns == 1 ? 14 : 19);
  }
  return stages >= 2 || (c->nb && c->nz <= 128);
}

// Whether a member of a batch does, where the launch is shared by all members of
// its NZ and its turns fill better: always with three stages or more, with two
// but for more than 48 modes on large grids, with bands alone up to a number of
// modes that falls with the columns, and with another stage alone on small
// grids.  Step us of 4 and 12 runs, one kernel against separate ones: 512 x 512
// z-mean and hyperdiffusion 280 / 299, 793 / 856, all stages with 40 modes 780 /
// 776, 2273 / 2294; z-mean with 86 modes 512 x 512 1317 / 1188, 3888 / 3486, 512 x
// 40 216 / 248, 583 / 666, with 40 modes 512 x 128 255 / 281, 713 / 779; bands
// alone 512 x 512 14 modes 508 / 446, 1427 / 1283, 256 x 512 20 modes 300 / 282,
// 815 / 788, 512 x 256 28 modes 394 / 355, 1081 / 991, 256 x 128 28 modes 145 /
// 150, 332 / 381, 64 modes 224 / 196, 511 / 513; z-mean alone 64 x 512 58 / 63,
// 132 / 153, 512 x 512 273 / 260, 777 / 743, sponge alone 128 x 40 50 / 52, 76 /
// 85, 512 x 512 257 / 238, 731 / 681.
bool col_fused_batch(const ymkh_ctx* c) {
  if (!c->col_ok) return false;
  const int stages = col_stages(c), modes = col_modes(c);
  if (stages >= 3) return true;
  if (stages == 2) return c->nz <= 256 || c->nx < 128 || modes <= kColWideModes;
  if (!modes) return c->nz <= 64 || c->nx < 512;
  return c->nz <= 128 || modes <= (c->nx >= 512 ? 10 : c->nx >= 256 ? 24 : kColWideModes);
}

// How the fused FCT's items (strip-major segments) are cut into one contiguous
// block per CTA.  The launch lasts as long as its slowest CTA, so the cut is
// the one whose costliest block is cheapest: in units of a fifth of an inner
// strip's row, a row of a strip whose window wraps takes 6 (its wrapped columns
// are put in place separately: 480 against 400 thousand cycles for 131 rows),
// and every strip that a block enters kFctEntry more (six rows of warm-up and
// the pipeline's fill).  So on a large grid the blocks even out (against equal
// rows 3.42 -> 3.12 ms at 4096 x 8192, 252 -> 227 us at 1024 x 2048), and on a
// small one none runs on into a second strip for a few rows (FCT us, against
// equal rows there: 128 x 256 38 -> 27, 256 x 512 48 -> 37, 256 x 768 56 -> 42,
// walls of 64-wide strips 243 x 371 71 -> 61; entry 25: 45 at 256 x 768, 60 as
// 40).
struct StripRun {
  int nstrips, nseg, seg;
  bool box;
};
constexpr int kFctEntry = 40, kFctEdgeRow = 6, kFctInnerRow = 5;
// Cuts the items into blocks of cost `most` or less; returns how many that
// takes, and with `first` writes where each starts.
int cut_fct_at(const std::vector<StripRun>& runs, long long most, int* first) {
  int n = 0, item = 0;
  long long left = 0;
  for (const StripRun& r : runs)
    for (int s = 0; s < r.nstrips; ++s) {
      const long long unit = (long long)r.seg * (r.box && (s == 0 || s == r.nstrips - 1) ? kFctEdgeRow : kFctInnerRow);
      for (int rem = r.nseg; rem > 0;) {
        if (left < kFctEntry + unit) {
          if (first) first[n] = item;
          ++n;
          left = most;
        }
        const int take = (int)std::min<long long>(rem, std::max<long long>(1, (left - kFctEntry) / unit));
        left -= kFctEntry + take * unit;
        rem -= take;
        item += take;
      }
    }
  return n;
}
void cut_fct(const std::vector<StripRun>& runs, int grid, int* first) {
  long long lo = 1, hi = 0;  // the cheapest `most` lies in [lo, hi]
  int items = 0;
  for (const StripRun& r : runs) {
    items += r.nstrips * r.nseg;
    hi += r.nstrips * (kFctEntry + (long long)r.nseg * r.seg * kFctEdgeRow);
    lo = std::max(lo, kFctEntry + (long long)r.seg * kFctEdgeRow);
  }
  while (lo < hi) {
    const long long mid = lo + (hi - lo) / 2;
    if (cut_fct_at(runs, mid, nullptr) <= grid) hi = mid;
    else lo = mid + 1;
  }
  const int n = cut_fct_at(runs, lo, first);
  for (int b = n; b <= grid; ++b) first[b] = items;
}
StripRun strip_run(const RunDesc& d, int nz) {
  return {d.fct_nstrips, (nz + d.fct_seg - 1) / d.fct_seg, d.fct_seg, d.fct_bulk == LOAD_BOX};
}

// Device descriptors of this run for both start buffers (single-run tables).
int upload_desc(ymkh_ctx* c) {
  c->desc_ok = false;
  if (!c->bound) return 0;
  if (!c->dev) CK(cudaMalloc(&c->dev, sizeof(ymkh_ctx::Tables)), "cudaMalloc run tables");
  { int rc = ensure_xscratch(c); if (rc) return rc; }
  c->boxed = c->aligned16 && c->nx >= kFctBoxWidth;
  const int arrays[kMaps] = {12, 9, 1, 12, 9, 12};
  const int width[kMaps] = {kFctBoxWidth, kFctBoxWidth, kFctBoxWidth, 4, 4, maxwell_box_width()};
  for (int k = 0; k < 2 * kMaps && c->boxed; ++k)
    c->boxed = encode_box(&c->host.maps[k], c->buf[k / kMaps], c->nx, c->nz, arrays[k % kMaps], width[k % kMaps]);
  RunDesc* h = c->host.desc;
  h[0] = make_desc(c, 0, c->fct_tx, 0, 0);
  h[1] = make_desc(c, 1, c->fct_tx, 0, 0);
  for (int i = 0; i < 2; ++i) h[i].fx_item0 = h[i].fz_item0 = 0;
  c->fct_items = items_fct(h[0], c->nz);
  cut_fct({strip_run(h[0], c->nz)}, fct_ctas(c->fct_items, c->fct_grid), c->host.fct_first);
  c->mx_items = items_mx(h[0], c->nz);
  c->fx_items = items_fx(h[0], c->nz);
  c->fz_items = items_fz(h[0], c->nz);
  c->col_ok = col_fused_ok(c);
  c->col_fused = c->col_ok && col_fused_alone(c);
  if (c->col_ok) {
    for (int i = 0; i < 2; ++i) c->host.col[i] = make_col(c, i);
    c->col_smem = column_fused_smem(c->nz, band_modes(c), c->prm.suppress_kz0);
    c->col_items = c->host.col[0].ncb * col_arrays(c->host.col[0]);
  }
  ++c->version;
  c->desc_pending = true;  // uploaded by the next step call, on its stream
  c->desc_ok = true;
  return 0;
}

// Table uploads are ordered on the stream of the step call that follows a
// change, after the steps already queued there, so a table is never
// rewritten under a kernel in flight on that stream.  Inside a stream
// capture (where a pageable copy cannot be captured) the copy is synchronous.
cudaError_t upload_table(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (s) cudaStreamIsCapturing(s, &cs);
  if (cs != cudaStreamCaptureStatusNone) return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
}

int flush_desc(ymkh_ctx* c, cudaStream_t s) {
  if (!c->desc_ok) { int rc = upload_desc(c); if (rc) return rc; }
  if (c->desc_pending) {
    CK(upload_table(c->dev, &c->host, sizeof c->host, s), "upload run tables");
    c->desc_pending = false;
  }
  return 0;
}

// One reference iteration from buffer c->cur into buffer 1 - c->cur.
enum Stage { ST_FCT = 0, ST_MAXWELL, ST_POINTWISE, ST_ZMEAN, ST_BANDS, ST_HYPER, ST_ZERO, ST_COUNT };

void mark(ymkh_ctx* c, int stage, cudaStream_t s) {
  if (c->timing) cudaEventRecord(c->ev[stage], s);
}

// Stages after the fused FCT and Maxwell launches, on the run's new buffer: as
// one kernel (fused) or one by one.
int post_stages(ymkh_ctx* c, bool fused, cudaStream_t s) {
  const State& out = c->buf[1 - c->cur];
  mark(c, ST_POINTWISE, s);
  if (fused) {
    mark(c, ST_ZMEAN, s);
    mark(c, ST_BANDS, s);
    CK(launch_column_fused(c->dev->col + (1 - c->cur), 1, c->col_items, c->nz, c->col_smem, s), "column stages");
    g_launches++;
    mark(c, ST_HYPER, s);
    mark(c, ST_ZERO, s);
    mark(c, ST_COUNT, s);
    return 0;
  }
  if (c->prm.xi_sponge > 0.0) { CK(launch_sponge_xicut(list12(out), c->sp, 0, s), "sponge"); g_launches++; }
  if (c->prm.xi_cut > 0.0) { CK(launch_sponge_xicut(list12(out), c->sp, 1, s), "xi_cut"); g_launches++; }
  // With suppress_kz0 the step ends by zeroing By1, Ex1 and Ez1, the first
  // three arrays of list21 (main_ym.cu:443-447).  The z-mean and the band
  // filters treat every array on its own and hyperdiffusion does not touch
  // colour 1, so the z-mean launch zeroes those three and the later stages
  // skip them: the state after the step is the same bit for bit.
  const int skip = c->prm.suppress_kz0 ? 3 : 0;
  const ArrayList l21 = list21(out);
  const ArrayList filt = drop_front(l21, skip);
  mark(c, ST_ZMEAN, s);
  if (c->prm.suppress_kz0) {
    ArrayList zl = filt;  // 12 arrays lose their z-mean, then By1, Ex1, Ez1 are zeroed
    for (int i = 0; i < 3; ++i) zl.p[12 + i] = l21.p[i];
    CK(launch_zmean(zl, 12, 3, c->nx, c->nz, c->zmeans, s), "zmean");
    g_launches++;
  }
  mark(c, ST_BANDS, s);
  const double inv2 = (double)(2.0f / (float)c->nz);
  for (int b = 0; b < c->nb; ++b) {
    if (c->prm.filter_engine == YMKH_FILTER_TF32X3) {
      // the first band also takes off the z-means (filt's first 12 arrays)
      CK(launch_band_tf32(filt, 21 - skip, c->tfb[b], c->tfs, c->nx, c->nz, 2.0f / (float)c->nz, c->zmeans,
                          c->zmeans && b == 0 ? 12 : 0, c->derr, s),
         "band filter (TF32 tensor cores)");
      g_launches += 3;
    } else {
      CK(launch_band(filt, 21 - skip, c->W[b], c->J[b], c->J[b], c->coef, c->nx, c->nz, inv2, s), "band filter");
      g_launches += 2;
    }
  }
  mark(c, ST_HYPER, s);
  if (c->prm.hyp_diff_coeff > 0.0) {
    CK(launch_hyperdiff(list12(out), c->nx, c->nz, c->prm.hyp_diff_coeff, s), "hyperdiffusion");
    g_launches++;
  }
  mark(c, ST_ZERO, s);  // colour-1 zeroing: done by the z-mean launch above
  mark(c, ST_COUNT, s);
  return 0;
}

bool has_column_stages(const ymkh_ctx* c) {
  const ymkh_params& p = c->prm;
  return c->nb || p.suppress_kz0 || p.xi_sponge > 0.0 || p.xi_cut > 0.0 || p.hyp_diff_coeff > 0.0;
}

// One reference iteration from buffer c->cur into buffer 1 - c->cur.
int step_once(ymkh_ctx* c, cudaStream_t s) {
  { int rc = flush_desc(c, s); if (rc) return rc; }
  RunTable T{c->dev->desc + c->cur, 1, c->fct_items, c->mx_items, c->derr, c->fx_items, c->fz_items, c->dev->fct_first};
  mark(c, ST_FCT, s);
  {
    NvtxRange r("ymkh fct");
    if (c->fct_mode == YMKH_FCT_SPLIT) {
      CK(launch_fct_split_table(T, c->fx_grid, c->fz_grid, s), "fct_x/fct_z kernels");
      g_launches++;
    } else {
      CK(launch_fct_table(T, c->fct_tx, fct_ctas(c->fct_items, c->fct_grid), s), "fct_fused_kernel");
    }
  }
  mark(c, ST_MAXWELL, s);
  {
    NvtxRange r("ymkh maxwell");
    CK(launch_maxwell_table(T, c->mx_grid, s), "maxwell_fused_kernel");
  }
  g_launches += 2;
  NvtxRange r("ymkh column stages");
  int rc = post_stages(c, c->col_fused, s);
  if (rc) return rc;
  c->cur = 1 - c->cur;
  return 0;
}

int copy_back(ymkh_ctx* c, cudaStream_t s) {
  const size_t bytes = c->N * sizeof(double);
  const State& a = c->buf[1];
  const State& b = c->buf[0];
  for (int i = 0; i < 12; ++i) CK(cudaMemcpyAsync(b.f[i], a.f[i], bytes, cudaMemcpyDeviceToDevice, s), "copy back");
  for (int i = 0; i < 6; ++i) {
    CK(cudaMemcpyAsync(b.a[i], a.a[i], bytes, cudaMemcpyDeviceToDevice, s), "copy back");
    CK(cudaMemcpyAsync(b.b[i], a.b[i], bytes, cudaMemcpyDeviceToDevice, s), "copy back");
  }
  c->cur = 0;
  return 0;
}

int run_graph(ymkh_ctx* c, cudaStream_t s) {
  const int start = c->cur;
  if (!c->gexec[start] || c->gstream[start] != s) {
    if (c->gexec[start]) { cudaGraphExecDestroy(c->gexec[start]); c->gexec[start] = nullptr; }
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "begin capture");
    int rc = 0;
    const long long l0 = g_launches.load();
    for (int k = 0; k < c->graph_steps && !rc; ++k) rc = step_once(c, s);
    c->glaunches[start] = g_launches.load() - l0;
    g_launches -= c->glaunches[start];  // counted when the graph runs
    cudaError_t ec = cudaStreamEndCapture(s, &g);
    c->cur = start;  // capture did not execute anything
    if (rc) { if (g) cudaGraphDestroy(g); return rc; }
    CK(ec, "end capture");
    cudaError_t ei = cudaGraphInstantiate(&c->gexec[start], g, 0);
    cudaGraphDestroy(g);
    CK(ei, "graph instantiate");
    c->gstream[start] = s;
  }
  CK(cudaGraphLaunch(c->gexec[start], s), "graph launch");
  g_launches += c->glaunches[start];
  // graph_steps is even: the state ends in the buffer it started from
  return 0;
}

}  // namespace

extern "C" {

int ymkh_last_error(char* buf, size_t n) {
  if (buf && n) {
    strncpy(buf, t_err_msg, n - 1);
    buf[n - 1] = 0;
  }
  return t_err_code;
}

long long ymkh_launch_count(void) { return g_launches.load(); }

int ymkh_build_flags(void) { return YMKH_DEBUG ? YMKH_BUILD_DEBUG : 0; }

int ymkh_create(const ymkh_grid* grid, const ymkh_params* params, ymkh_ctx** out) try {
  if (!grid || !params || !out) return set_err(YMKH_EINVAL, "null argument");
  if (grid->nx < 4 || grid->nz < 4) return set_err(YMKH_EINVAL, "grid too small (%d x %d)", grid->nx, grid->nz);
  if ((size_t)grid->nx * grid->nz > ((size_t)1 << 34)) return set_err(YMKH_EINVAL, "grid too large");
  ymkh_ctx* c = new ymkh_ctx();
  // failures after this point release the context and what it holds
#define CK_CREATE(call, what)                                                                 \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) {                                                                  \
      const int rc_ = set_err(YMKH_ECUDA, "%s: %s", what, cudaGetErrorString(e_));            \
      ymkh_destroy(c);                                                                        \
      return rc_;                                                                             \
    }                                                                                         \
  } while (0)
  CK_CREATE(cudaGetDevice(&c->device), "cudaGetDevice");
  c->nx = grid->nx; c->nz = grid->nz; c->N = (size_t)grid->nx * grid->nz;
  int rc = setup_params(c, params);
  if (rc) { free_bands(c); delete c; return rc; }
  CK_CREATE(prepare_fct(32), "FCT kernel attributes");
  CK_CREATE(prepare_fct(64), "FCT kernel attributes");
  CK_CREATE(prepare_fct(128), "FCT kernel attributes");
  CK_CREATE(prepare_maxwell(), "Maxwell kernel attributes");
  CK_CREATE(prepare_fct_split(), "split FCT kernel attributes");
  CK_CREATE(prepare_column_fused(), "column kernel attributes");
  choose_launch_shape(c);
  CK_CREATE(prepare_column(c->nz), "column kernel attributes");
#undef CK_CREATE
  // everything that energy and amplitude calls need, so that a first one in the
  // middle of a campaign that fills the memory cannot fail for the want of it
  const int np = energy_nparts(c->N);
  if (!(c->hres = host_slots().take()) || cudaMalloc(&c->epart, (size_t)2 * np * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&c->mcol, mode_amp_scratch(c->nx, c->nz) * sizeof(double)) != cudaSuccess ||
      cudaMalloc(&c->derr, sizeof(unsigned)) != cudaSuccess || cudaMemset(c->derr, 0, sizeof(unsigned)) != cudaSuccess) {
    ymkh_destroy(c);
    return set_err(YMKH_ENOMEM, "cudaMalloc diagnostics");
  }
  *out = c;
  return 0;
} YMKH_CATCH

int ymkh_set_params(ymkh_ctx* c, const ymkh_params* p) try {
  if (!c || !p) return set_err(YMKH_EINVAL, "null argument");
  int rc = setup_params(c, p);
  if (rc) return rc;
  return upload_desc(c);
} YMKH_CATCH

static State make_state(double* const f[12], double* const a[6], double* const b[6]) {
  State s{};
  for (int i = 0; i < 12; ++i) s.f[i] = f[i];
  for (int i = 0; i < 6; ++i) { s.a[i] = a[i]; s.b[i] = b[i]; }
  return s;
}

static bool aligned16(const State& s) {
  for (int i = 0; i < 12; ++i) if (reinterpret_cast<uintptr_t>(s.f[i]) % 16) return false;
  for (int i = 0; i < 6; ++i)
    if (reinterpret_cast<uintptr_t>(s.a[i]) % 16 || reinterpret_cast<uintptr_t>(s.b[i]) % 16) return false;
  return true;
}

static bool state_ok(const State& s) {
  for (int i = 0; i < 12; ++i) if (!s.f[i]) return false;
  for (int i = 0; i < 6; ++i) if (!s.a[i] || !s.b[i]) return false;
  return true;
}

int ymkh_bind_state(ymkh_ctx* c, double* const fields[YMKH_NFIELDS], double* const fluidA[YMKH_NFLUID],
                    double* const fluidB[YMKH_NFLUID]) try {
  if (!c || !fields || !fluidA || !fluidB) return set_err(YMKH_EINVAL, "null argument");
  State s = make_state(fields, fluidA, fluidB);
  if (!state_ok(s)) return set_err(YMKH_EINVAL, "null state array");
  drop_graphs(c);
  c->buf[0] = s;
  if (!c->own) {
    if (cudaMalloc(&c->own, 24 * c->N * sizeof(double)) != cudaSuccess)
      return set_err(YMKH_ENOMEM, "cudaMalloc second state buffer (%zu bytes)", 24 * c->N * sizeof(double));
  }
  for (int i = 0; i < 12; ++i) c->buf[1].f[i] = c->own + (size_t)i * c->N;
  for (int i = 0; i < 6; ++i) {
    c->buf[1].a[i] = c->own + (size_t)(12 + i) * c->N;
    c->buf[1].b[i] = c->own + (size_t)(18 + i) * c->N;
  }
  c->dual = false;
  c->cur = 0;
  c->bound = true;
  c->aligned16 = aligned16(c->buf[0]) && aligned16(c->buf[1]);
  return upload_desc(c);
} YMKH_CATCH

// Zero-copy form: the caller provides both buffers; after ymkh_step the
// current state is in buffer ymkh_current_buffer().
int ymkh_bind_state2(ymkh_ctx* c, double* const* state0, double* const* state1) try {
  if (!c || !state0 || !state1) return set_err(YMKH_EINVAL, "null argument");
  State s0 = make_state(state0, state0 + 12, state0 + 18);
  State s1 = make_state(state1, state1 + 12, state1 + 18);
  if (!state_ok(s0) || !state_ok(s1)) return set_err(YMKH_EINVAL, "null state array");
  drop_graphs(c);
  if (c->own) { cudaFree(c->own); c->own = nullptr; }
  c->buf[0] = s0;
  c->buf[1] = s1;
  c->dual = true;
  c->cur = 0;
  c->bound = true;
  c->aligned16 = aligned16(s0) && aligned16(s1);
  return upload_desc(c);
} YMKH_CATCH

// Reads (and clears) the device error word set by in-kernel waits that ran
// out of polls; synchronises the stream.
int ymkh_check(ymkh_ctx* c, void* stream) try {
  if (!c) return set_err(YMKH_EINVAL, "null context");
  unsigned h = 0;
  CK(cudaMemcpyAsync(&h, c->derr, sizeof h, cudaMemcpyDeviceToHost, (cudaStream_t)stream), "error word D2H");
  CK(cudaStreamSynchronize((cudaStream_t)stream), "error word sync");
  if (h) {
    cudaMemsetAsync(c->derr, 0, sizeof(unsigned), (cudaStream_t)stream);
    return set_err(YMKH_ECUDA, "%s (error word %u); results of that step are invalid",
                   (h & ERR_BOUNDS) ? "a checked access was out of range and skipped" : "a bounded in-kernel wait timed out",
                   h);
  }
  return 0;
} YMKH_CATCH

int ymkh_current_buffer(ymkh_ctx* c) { return c ? c->cur : -1; }

int ymkh_set_current_buffer(ymkh_ctx* c, int which) try {
  if (!c || (which != 0 && which != 1)) return set_err(YMKH_EINVAL, "bad buffer index");
  if (!c->dual && which == 1) return set_err(YMKH_ESTATE, "buffer 1 is library-owned");
  c->cur = which;
  return 0;
} YMKH_CATCH

int ymkh_init(ymkh_ctx* c, const ymkh_init_params* ip, void* stream) try {
  if (!c || !ip) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  cudaStream_t s = (cudaStream_t)stream;
  InitArgs a{};
  a.nx = c->nx; a.nz = c->nz; a.dx = c->prm.dx; a.dz = c->prm.dz;
  a.k_mode = ip->k_mode; a.perturb_amp = ip->perturb_amp; a.V0 = ip->V0; a.epsilon = ip->epsilon;
  a.run_mode = ip->run_mode; a.alpha_YM = (double)(float)ip->alpha_YM;
  a.init_by1_eq = ip->init_by1_eq; a.vz_edge_taper = ip->vz_edge_taper;
  const double* hs[6] = {ip->seed_by, ip->seed_ex, ip->seed_ez, ip->seed_az, ip->seed_qA, ip->seed_qB};
  const double** ds[6] = {&a.by, &a.ex, &a.ez, &a.az, &a.qA, &a.qB};
  double* seedbuf = nullptr;
  int nseed = 0;
  for (int k = 0; k < 6; ++k) if (hs[k]) ++nseed;
  if (nseed) {
    CK(cudaMalloc(&seedbuf, (size_t)6 * c->nx * sizeof(double)), "cudaMalloc seed");
    for (int k = 0; k < 6; ++k) {
      if (!hs[k]) continue;
      double* d = seedbuf + (size_t)k * c->nx;
      CK(cudaMemcpyAsync(d, hs[k], c->nx * sizeof(double), cudaMemcpyHostToDevice, s), "seed upload");
      *ds[k] = d;
    }
  }
  c->cur = 0;
  cudaError_t e = launch_init(c->buf[0], a, s);
  g_launches++;
  if (seedbuf) {
    cudaStreamSynchronize(s);
    cudaFree(seedbuf);
  }
  CK(e, "init kernel");
  return 0;
} YMKH_CATCH

int ymkh_step(ymkh_ctx* c, int nsteps, void* stream) try {
  if (!c) return set_err(YMKH_EINVAL, "null context");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  if (nsteps < 0) return set_err(YMKH_EINVAL, "negative step count");
  NvtxRange range("ymkh_step");
  cudaStream_t s = (cudaStream_t)stream;
  { int rc = flush_desc(c, s); if (rc) return rc; }  // before any capture of the steps
  int done = 0;
  const bool graphs = s != nullptr && c->graph_steps >= 2 && (c->graph_steps % 2) == 0;
  if (graphs) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cs);
    if (cs == cudaStreamCaptureStatusNone) {
      while (nsteps - done >= c->graph_steps) {
        int rc = run_graph(c, s);
        if (rc) return rc;
        done += c->graph_steps;
      }
    }
  }
  for (; done < nsteps; ++done) {
    int rc = step_once(c, s);
    if (rc) return rc;
  }
  if (!c->dual && c->cur == 1) return copy_back(c, s);
  return 0;
} YMKH_CATCH

int ymkh_set_graph_steps(ymkh_ctx* c, int n) try {
  if (!c || n < 0 || (n % 2) != 0) return set_err(YMKH_EINVAL, "graph step count must be even and >= 0");
  drop_graphs(c);
  c->graph_steps = n;
  return 0;
} YMKH_CATCH

int ymkh_set_fct_shape(ymkh_ctx* c, int tx, int seg) try {
  if (!c || (tx != 32 && tx != 64 && tx != 128) || seg < 1) return set_err(YMKH_EINVAL, "bad FCT launch shape");
  drop_graphs(c);
  c->fct_tx = tx;
  c->fct_seg = seg;
  c->fct_grid = c->sms * std::max(1, fct_ctas_per_sm(tx));
  return upload_desc(c);
} YMKH_CATCH

int ymkh_set_fct_mode(ymkh_ctx* c, int mode) try {
  if (!c || (mode != YMKH_FCT_FUSED && mode != YMKH_FCT_SPLIT)) return set_err(YMKH_EINVAL, "bad FCT mode");
  drop_graphs(c);
  c->fct_mode = mode;
  return upload_desc(c);
} YMKH_CATCH

int ymkh_get_fct_shape(ymkh_ctx* c, int* tx, int* seg) try {
  if (!c) return set_err(YMKH_EINVAL, "null context");
  if (tx) *tx = c->fct_tx;
  if (seg) *seg = c->fct_seg;
  return 0;
} YMKH_CATCH

// Runs nsteps plain (uncaptured) steps with an event between stages and
// accumulates the device time of each stage into out_ms[0..ST_COUNT).
int ymkh_stage_times(ymkh_ctx* c, int nsteps, void* stream, float* out_ms, int nout) try {
  if (!c || !out_ms || nout < ST_COUNT) return set_err(YMKH_EINVAL, "bad arguments");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  cudaStream_t s = (cudaStream_t)stream;
  for (int i = 0; i <= ST_COUNT; ++i) CK(cudaEventCreate(&c->ev[i]), "cudaEventCreate");
  for (int i = 0; i < ST_COUNT; ++i) out_ms[i] = 0.f;
  c->timing = true;
  int rc = 0;
  for (int k = 0; k < nsteps && !rc; ++k) {
    rc = step_once(c, s);
    if (rc) break;
    cudaError_t e = cudaEventSynchronize(c->ev[ST_COUNT]);
    if (e != cudaSuccess) { rc = set_err(YMKH_ECUDA, "stage timing: %s", cudaGetErrorString(e)); break; }
    for (int i = 0; i < ST_COUNT; ++i) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, c->ev[i], c->ev[i + 1]);
      out_ms[i] += ms;
    }
  }
  c->timing = false;
  for (int i = 0; i <= ST_COUNT; ++i) cudaEventDestroy(c->ev[i]);
  if (!rc && !c->dual && c->cur == 1) rc = copy_back(c, s);
  return rc;
} YMKH_CATCH

int ymkh_energy_async(ymkh_ctx* c, double* dev_out, void* stream) try {
  if (!c || !dev_out) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  CK(launch_energy(c->buf[c->cur], c->N, c->epart, dev_out, nullptr, (cudaStream_t)stream), "energy kernels");
  g_launches += 2;
  return 0;
} YMKH_CATCH

int ymkh_energy(ymkh_ctx* c, double* host_out, void* stream) try {
  if (!host_out) return set_err(YMKH_EINVAL, "null argument");
  if (!c) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  cudaStream_t s = (cudaStream_t)stream;
  CK(launch_energy(c->buf[c->cur], c->N, c->epart, c->hres, c->derr, s), "energy kernels");
  g_launches += 2;
  CK(cudaStreamSynchronize(s), "energy sync");
  *host_out = c->hres[0];
  return c->hres[1] != 0.0 ? ymkh_check(c, stream) : 0;  // reports and clears the error word
} YMKH_CATCH

int ymkh_mode_amp(ymkh_ctx* c, int k, double* host_out2, void* stream) try {
  return ymkh_circ_amp(c, YMKH_PAIR_AZ, k, nullptr, host_out2, stream);
} YMKH_CATCH

int ymkh_circ_amp(ymkh_ctx* c, int pair, int k, const double* host_weight, double* host_out2, void* stream) try {
  if (!c || !host_out2) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  static const int re_of[4] = {AZ2, BY2, EX2, EZ2};
  if (pair < 0 || pair > 3) return set_err(YMKH_EINVAL, "pair %d not in 0..3", pair);
  cudaStream_t s = (cudaStream_t)stream;
  const State& st = c->buf[c->cur];
  const double* w = nullptr;
  if (host_weight) {
    if (!c->mweight && cudaMalloc(&c->mweight, (size_t)c->nx * sizeof(double)) != cudaSuccess)
      return set_err(YMKH_ENOMEM, "cudaMalloc mode weights");
    CK(cudaMemcpyAsync(c->mweight, host_weight, (size_t)c->nx * sizeof(double), cudaMemcpyHostToDevice, s),
       "mode weights H2D");
    w = c->mweight;
  }
  CK(launch_mode_amp(st.f[re_of[pair]], st.f[re_of[pair] + 1], c->nx, c->nz, k, c->mcol, w, c->hres, s),
     "mode amplitude kernels");
  g_launches += 2;
  CK(cudaStreamSynchronize(s), "mode amp sync");
  host_out2[0] = c->hres[0];
  host_out2[1] = c->hres[1];
  return 0;
} YMKH_CATCH

int ymkh_gauss(ymkh_ctx* c, double* host_out, void* stream) try {
  if (!c || !host_out) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  const int np = gauss_nparts(c->N);
  const size_t n = (size_t)np * YMKH_GAUSS_NOUT * 2;
  if (!c->gpart && cudaMalloc(&c->gpart, n * sizeof(double)) != cudaSuccess)
    return set_err(YMKH_ENOMEM, "cudaMalloc Gauss partials");
  cudaStream_t s = (cudaStream_t)stream;
  CK(launch_gauss(c->buf[c->cur], c->nx, c->nz, c->prm.dx, c->prm.dz, c->prm.alpha_YM, c->gpart, c->hres, s),
     "Gauss residual kernels");
  g_launches += 2;
  CK(cudaStreamSynchronize(s), "Gauss sync");
  for (int i = 0; i < YMKH_GAUSS_NOUT; ++i) host_out[i] = c->hres[i];
  return 0;
} YMKH_CATCH

int ymkh_snapshot(ymkh_ctx* c, const char* path, int format, void* stream) try {
  if (!c || !path) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "state not bound");
  if (format != YMKH_SNAP_CSV && format != YMKH_SNAP_FP64) return set_err(YMKH_EINVAL, "snapshot format %d", format);
  if (!c->snaps) c->snaps = snapshot_queue_create(c->device);
  std::string err;
  const int rc = snapshot_submit(c->snaps, c->buf[c->cur], c->nx, c->nz, c->prm.dx, c->prm.dz, path, format,
                                 (cudaStream_t)stream, err);
  return rc ? set_err(rc, "%s", err.c_str()) : 0;
} YMKH_CATCH

int ymkh_snapshot_wait(ymkh_ctx* c) try {
  if (!c) return set_err(YMKH_EINVAL, "null context");
  if (!c->snaps) return 0;
  std::string err;
  const int rc = snapshot_wait(c->snaps, err);
  return rc ? set_err(rc, "%s", err.c_str()) : 0;
} YMKH_CATCH

int ymkh_destroy(ymkh_ctx* c) try {
  if (!c) return 0;
  if (c->snaps) snapshot_queue_destroy(c->snaps);  // waits for its writers
  drop_graphs(c);
  free_bands(c);
  if (c->own) cudaFree(c->own);
  if (c->epart) cudaFree(c->epart);
  if (c->hres) host_slots().give_back(c->hres);
  if (c->mcol) cudaFree(c->mcol);
  if (c->mweight) cudaFree(c->mweight);
  if (c->gpart) cudaFree(c->gpart);
  if (c->derr) cudaFree(c->derr);
  if (c->dev) cudaFree(c->dev);
  if (c->xscratch) cudaFree(c->xscratch);
  delete c;
  return 0;
} YMKH_CATCH

int ymkh_twiddles(int nz, int m_lo, int m_hi, float* cos_out, float* sin_out) try {
  if (nz < 1 || m_lo < 0 || m_hi < m_lo || !cos_out || !sin_out) return set_err(YMKH_EINVAL, "bad arguments");
  const size_t n = (size_t)(m_hi - m_lo + 1) * nz;
  float *dc = nullptr, *ds = nullptr;
  CK(cudaMalloc(&dc, n * sizeof(float)), "cudaMalloc");
  CK(cudaMalloc(&ds, n * sizeof(float)), "cudaMalloc");
  cudaError_t e = launch_twiddles_f32(dc, ds, nz, m_lo, m_hi, 0);
  g_launches++;
  if (e == cudaSuccess) e = cudaMemcpy(cos_out, dc, n * sizeof(float), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(sin_out, ds, n * sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(dc);
  cudaFree(ds);
  CK(e, "twiddle table");
  return 0;
} YMKH_CATCH

// ------------------------------------------------------------------ batches
// Runs of any sizes advance together: one FCT and one Maxwell launch per step
// cover the (run, strip, segment) items of every member; one launch per NZ the
// column stages of the members that share column_kernel (col_fused_batch), and
// the others' stages are launched per member on auxiliary streams.  Steps can be
// captured as CUDA graphs.

struct ymkh_batch {
  std::vector<ymkh_ctx*> runs;
  RunDesc* ddesc = nullptr;  // [2][cap]: tables for the members' current / next buffers
  int cap = 0;
  // members whose column stages run fused, grouped by NZ (one launch a group)
  struct ColGroup { int nz, first, n, items; size_t smem; };
  ColDesc* dcol = nullptr;   // [2][cap]
  int* dfirst = nullptr;     // items of the fused FCT's CTAs
  std::vector<ColGroup> col;
  std::vector<char> col_member;    // whether the member is in one of the groups
  // of each member when the tables were built: its descriptors' version and the
  // buffer it stepped from
  std::vector<unsigned> versions;
  std::vector<int> cur0;
  int fct_items = 0, mx_items = 0, fx_items = 0, fz_items = 0;
  int tb = 128, fct_grid = 0, mx_grid = 0, fx_grid = 0, fz_grid = 0;
  int fct_grids[3] = {0, 0, 0};    // CTAs of each strip width (kBatchWidth)
  int fct_mode = YMKH_FCT_FUSED;
  unsigned* derr = nullptr;
  bool dirty = true;
  int parity = 0;            // steps taken since the tables were built, mod 2
  int graph_steps = 4;
  cudaGraphExec_t gexec = nullptr;
  cudaStream_t gstream = nullptr;
  long long glaunches = 0;
  // The members' column stages (z-mean, band filters, ...) are independent
  // run to run: they fork onto auxiliary streams after the fused launches
  // and join back before the next step (also inside a captured graph).
  static constexpr int kAux = 8;
  cudaStream_t aux[kAux]{};
  cudaEvent_t fork_ev = nullptr;
  cudaEvent_t join_ev[kAux]{};
};

namespace {

void batch_drop_graph(ymkh_batch* b) {
  if (b->gexec) { cudaGraphExecDestroy(b->gexec); b->gexec = nullptr; b->gstream = nullptr; }
}

// Strip width of a batch: the one whose strips take least time over all rows of
// its members.  A strip's row costs about as 4, 6 and 9 in 32-, 64- and 128-wide
// strips (305, 450 and 690 us for 16 runs of 2048 rows), and in the last form
// one more for every copy past two that fills the window of a narrow grid.  So
// 128 but for grids of up to 58 columns (step of 16 runs, 32-, 64- and 128-wide:
// 2048 x 8 692, 826, 2013 us; 2048 x 48 984, 834, 1133; 2048 x 64 1285, 1292,
// 1070; 64 x 96 73, -, 56; 64 x 48 54, 57, 60).
constexpr int kBatchWidth[3] = {32, 64, 128}, kBatchRow[3] = {4, 6, 9};
int pick_batch_width(const std::vector<ymkh_ctx*>& runs) {
  int best = 2;
  long long best_cost = 0;
  for (int k = 2; k >= 0; --k) {
    long long cost = 0;
    for (const ymkh_ctx* c : runs) {
      const int row = kBatchRow[k] + (k == 2 ? std::max(0, kBatchWidth[k] / c->nx - 2) : 0);
      cost += (long long)row * fct_nstrips(c->nx, kBatchWidth[k]) * c->nz;
    }
    if (k == 2 || cost < best_cost) { best = k; best_cost = cost; }
  }
  return best;
}

int batch_build(ymkh_batch* b, cudaStream_t s) {
  const int n = (int)b->runs.size();
  if (n > b->cap) {
    const int cap = std::max(n, 2 * b->cap);
    if (b->ddesc) cudaFree(b->ddesc);
    if (b->dcol) cudaFree(b->dcol);
    b->ddesc = nullptr;
    b->dcol = nullptr;
    b->cap = 0;
    CK(cudaMalloc(&b->dcol, 2 * (size_t)cap * sizeof(ColDesc)), "cudaMalloc batch column tables");
    CK(cudaMalloc(&b->ddesc, 2 * (size_t)cap * sizeof(RunDesc)), "cudaMalloc batch descriptors");
    b->cap = cap;
  }
  const int width = pick_batch_width(b->runs);
  b->tb = kBatchWidth[width];
  b->fct_grid = b->fct_grids[width];
  std::vector<RunDesc> h(2 * (size_t)std::max(n, 1));
  std::vector<StripRun> strips;
  std::vector<MxGrid> mg;
  for (const ymkh_ctx* c : b->runs) mg.push_back({c->nz, maxwell_nstrips(c->nx)});
  const int mx_seg = pick_mx_segment(mg.data(), n, b->mx_grid);
  int f0 = 0, m0 = 0, x0 = 0, z0 = 0;
  for (int i = 0; i < n; ++i) {
    ymkh_ctx* c = b->runs[i];
    if (b->fct_mode == YMKH_FCT_SPLIT && !c->xscratch) {
      const int keep = c->fct_mode;
      c->fct_mode = YMKH_FCT_SPLIT;
      int rc = ensure_xscratch(c);
      c->fct_mode = keep;
      if (rc) return rc;
    }
    { int rc = flush_desc(c, s); if (rc) return rc; }  // the member's tensor maps
    RunDesc d0 = make_desc(c, c->cur, b->tb, f0, m0);
    RunDesc d1 = make_desc(c, 1 - c->cur, b->tb, f0, m0);
    d0.fx_item0 = d1.fx_item0 = x0;
    d0.fz_item0 = d1.fz_item0 = z0;
    x0 += items_fx(d0, c->nz);
    z0 += items_fz(d0, c->nz);
    // one-row FCT segments in contiguous blocks, as a lone run's (at 16 uneven
    // runs of 128..1024 x 256..2048, the step took 2422 us against 2453 with
    // 128-row segments round-robin; at 24 runs of 64 x 768, 820 against 905)
    d0.fct_seg = d1.fct_seg = kFctSegment;
    d0.mx_seg = d1.mx_seg = std::min(c->nz, mx_seg);
    d0.fct_item0 = d1.fct_item0 = f0;
    d0.mx_item0 = d1.mx_item0 = m0;
    h[i] = d0;
    h[n + i] = d1;
    strips.push_back(strip_run(d0, c->nz));
    f0 += items_fct(d0, c->nz);
    m0 += items_mx(d0, c->nz);
  }
  b->fct_items = f0;
  b->mx_items = m0;
  b->fx_items = x0;
  b->fz_items = z0;
  if (n) {
    // in stream order after the steps already queued on s (a pageable
    // source is staged before the call returns)
    CK(upload_table(b->ddesc, h.data(), (size_t)n * sizeof(RunDesc), s), "upload batch table");
    CK(upload_table(b->ddesc + b->cap, h.data() + n, (size_t)n * sizeof(RunDesc), s), "upload batch table");
  }
  // fused column stages: members sorted by NZ, one table range and launch per NZ
  b->col.clear();
  b->versions.clear();
  b->cur0.clear();
  std::vector<int> order;
  int n_ok = 0;
  for (int i = 0; i < n; ++i) {
    b->versions.push_back(b->runs[i]->version);
    b->cur0.push_back(b->runs[i]->cur);
    n_ok += b->runs[i]->col_ok;
  }
  // up to three members that can go by what each does alone
  b->col_member.assign(n, 0);
  for (int i = 0; i < n; ++i)
    if (n_ok >= 4 ? col_fused_batch(b->runs[i]) : b->runs[i]->col_fused) {
      b->col_member[i] = 1;
      order.push_back(i);
    }
  std::stable_sort(order.begin(), order.end(), [&](int i, int j) { return b->runs[i]->nz < b->runs[j]->nz; });
  std::vector<ColDesc> hc[2];
  for (int i : order) {
    ymkh_ctx* c = b->runs[i];
    if (b->col.empty() || b->col.back().nz != c->nz) b->col.push_back({c->nz, (int)hc[0].size(), 0, 0, 0});
    ymkh_batch::ColGroup& g = b->col.back();
    for (int p = 0; p < 2; ++p) {
      hc[p].push_back(c->host.col[p ? c->cur : 1 - c->cur]);
      hc[p].back().item0 = g.items;
    }
    g.n++;
    g.items += c->col_items;
    g.smem = std::max(g.smem, c->col_smem);
  }
  for (int p = 0; p < 2 && !order.empty(); ++p)
    CK(upload_table(b->dcol + (size_t)p * b->cap, hc[p].data(), hc[p].size() * sizeof(ColDesc), s), "upload batch column table");
  if (n) {
    std::vector<int> first(kMaxFctCtas + 1);
    cut_fct(strips, fct_ctas(b->fct_items, b->fct_grid), first.data());
    if (!b->dfirst) CK(cudaMalloc(&b->dfirst, first.size() * sizeof(int)), "cudaMalloc batch FCT blocks");
    CK(upload_table(b->dfirst, first.data(), first.size() * sizeof(int), s), "upload batch FCT blocks");
  }
  b->parity = 0;
  b->dirty = false;
  batch_drop_graph(b);
  return 0;
}

int batch_step_once(ymkh_batch* b, cudaStream_t s) {
  const int n = (int)b->runs.size();
  if (!n) return 0;
  RunTable T{b->ddesc + (size_t)b->parity * b->cap, n, b->fct_items, b->mx_items, b->derr, b->fx_items, b->fz_items, b->dfirst};
  if (b->fct_mode == YMKH_FCT_SPLIT)
    CK(launch_fct_split_table(T, b->fx_grid, b->fz_grid, s), "fct_x/fct_z kernels (batch)");
  else
    CK(launch_fct_table(T, b->tb, fct_ctas(b->fct_items, b->fct_grid), s), "fct_fused_kernel (batch)");
  CK(launch_maxwell_table(T, b->mx_grid, s), "maxwell_fused_kernel (batch)");
  g_launches += 2;
  // column stages: one launch per NZ of the fused ones, the others per member;
  // all independent of each other, spread over the auxiliary streams
  auto separate = [&](int i) { return !b->col_member[i] && has_column_stages(b->runs[i]); };
  int nsep = 0;
  for (int i = 0; i < n; ++i) nsep += separate(i);
  const int jobs = (int)b->col.size() + nsep;
  const int na = b->aux[0] ? std::min(jobs, (int)ymkh_batch::kAux) : 1;
  if (na > 1) {
    CK(cudaEventRecord(b->fork_ev, s), "batch fork");
    for (int i = 0; i < na; ++i) CK(cudaStreamWaitEvent(b->aux[i], b->fork_ev, 0), "batch fork");
  }
  int job = 0;
  for (const ymkh_batch::ColGroup& g : b->col) {
    CK(launch_column_fused(b->dcol + (size_t)b->parity * b->cap + g.first, g.n, g.items, g.nz, g.smem,
                           na > 1 ? b->aux[job % na] : s), "column stages (batch)");
    g_launches++;
    ++job;
  }
  for (int i = 0; i < n; ++i) {
    ymkh_ctx* c = b->runs[i];
    if (separate(i)) {
      int rc = post_stages(c, false, na > 1 ? b->aux[job % na] : s);
      if (rc) return rc;
      ++job;
    }
    c->cur = 1 - c->cur;
  }
  if (na > 1) {
    for (int i = 0; i < na; ++i) {
      CK(cudaEventRecord(b->join_ev[i], b->aux[i]), "batch join");
      CK(cudaStreamWaitEvent(s, b->join_ev[i], 0), "batch join");
    }
  }
  b->parity ^= 1;
  return 0;
}

}  // namespace

int ymkh_batch_create(ymkh_batch** out) try {
  if (!out) return set_err(YMKH_EINVAL, "null argument");
  ymkh_batch* b = new ymkh_batch();
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  for (int tb : {32, 64, 128}) prepare_fct(tb);
  prepare_maxwell();
  prepare_fct_split();
  for (int k = 0; k < 3; ++k) b->fct_grids[k] = sms * std::max(1, fct_ctas_per_sm(kBatchWidth[k]));
  b->mx_grid = sms * std::max(1, maxwell_ctas_per_sm());
  b->fx_grid = sms * std::max(1, fct_split_ctas_per_sm(0)) * 4;
  b->fz_grid = sms * std::max(1, fct_split_ctas_per_sm(1)) * 4;
  bool ok = cudaEventCreateWithFlags(&b->fork_ev, cudaEventDisableTiming) == cudaSuccess;
  for (int i = 0; ok && i < ymkh_batch::kAux; ++i)
    ok = cudaStreamCreateWithFlags(&b->aux[i], cudaStreamNonBlocking) == cudaSuccess &&
         cudaEventCreateWithFlags(&b->join_ev[i], cudaEventDisableTiming) == cudaSuccess;
  if (!ok || cudaMalloc(&b->derr, sizeof(unsigned)) != cudaSuccess ||
      cudaMemset(b->derr, 0, sizeof(unsigned)) != cudaSuccess) {
    for (int i = 0; i < ymkh_batch::kAux; ++i) {
      if (b->aux[i]) cudaStreamDestroy(b->aux[i]);
      if (b->join_ev[i]) cudaEventDestroy(b->join_ev[i]);
    }
    if (b->fork_ev) cudaEventDestroy(b->fork_ev);
    delete b;
    return set_err(YMKH_ENOMEM, "batch streams, events or error word");
  }
  *out = b;
  return 0;
} YMKH_CATCH

int ymkh_batch_add(ymkh_batch* b, ymkh_ctx* c) try {
  if (!b || !c) return set_err(YMKH_EINVAL, "null argument");
  if (!c->bound) return set_err(YMKH_ESTATE, "run state not bound");
  for (ymkh_ctx* r : b->runs) if (r == c) return set_err(YMKH_EINVAL, "run already in the batch");
  b->runs.push_back(c);
  b->dirty = true;
  return 0;
} YMKH_CATCH

int ymkh_batch_remove(ymkh_batch* b, ymkh_ctx* c) try {
  if (!b || !c) return set_err(YMKH_EINVAL, "null argument");
  auto it = std::find(b->runs.begin(), b->runs.end(), c);
  if (it == b->runs.end()) return set_err(YMKH_EINVAL, "run not in the batch");
  b->runs.erase(it);
  b->dirty = true;
  return 0;
} YMKH_CATCH

int ymkh_batch_size(ymkh_batch* b) { return b ? (int)b->runs.size() : -1; }

int ymkh_batch_set_graph_steps(ymkh_batch* b, int n) try {
  if (!b || n < 0 || (n % 2) != 0) return set_err(YMKH_EINVAL, "graph step count must be even and >= 0");
  batch_drop_graph(b);
  b->graph_steps = n;
  return 0;
} YMKH_CATCH

int ymkh_batch_step(ymkh_batch* b, int nsteps, void* stream) try {
  if (!b) return set_err(YMKH_EINVAL, "null batch");
  if (nsteps < 0) return set_err(YMKH_EINVAL, "negative step count");
  NvtxRange range("ymkh_batch_step");
  cudaStream_t s = (cudaStream_t)stream;
  // the tables no longer hold for a member with new parameters or arrays, or one
  // whose state was put into the other buffer (set anew, or stepped alone)
  for (size_t i = 0; i < b->versions.size() && !b->dirty; ++i)
    b->dirty = b->versions[i] != b->runs[i]->version || b->runs[i]->cur != (b->cur0[i] ^ b->parity);
  if (b->dirty) { int rc = batch_build(b, s); if (rc) return rc; }
  int done = 0;
  const bool graphs = s != nullptr && b->graph_steps >= 2 && !b->runs.empty();
  if (graphs) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(s, &cs);
    if (cs == cudaStreamCaptureStatusNone) {
      // the captured graph starts from the tables' first parity
      if (b->parity != 0 && nsteps - done > b->graph_steps) {
        int rc = batch_step_once(b, s);
        if (rc) return rc;
        ++done;
      }
      while (b->parity == 0 && nsteps - done >= b->graph_steps) {
        if (!b->gexec || b->gstream != s) {
          batch_drop_graph(b);
          std::vector<int> cur0;
          for (ymkh_ctx* c : b->runs) cur0.push_back(c->cur);
          cudaGraph_t g = nullptr;
          CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal), "begin capture");
          const long long l0 = g_launches.load();
          int rc = 0;
          for (int k = 0; k < b->graph_steps && !rc; ++k) rc = batch_step_once(b, s);
          b->glaunches = g_launches.load() - l0;
          g_launches -= b->glaunches;
          cudaError_t ec = cudaStreamEndCapture(s, &g);
          for (size_t i = 0; i < b->runs.size(); ++i) b->runs[i]->cur = cur0[i];  // nothing ran yet
          b->parity = 0;
          if (rc) { if (g) cudaGraphDestroy(g); return rc; }
          CK(ec, "end capture");
          cudaError_t ei = cudaGraphInstantiate(&b->gexec, g, 0);
          cudaGraphDestroy(g);
          CK(ei, "graph instantiate");
          b->gstream = s;
        }
        CK(cudaGraphLaunch(b->gexec, s), "graph launch");
        g_launches += b->glaunches;
        done += b->graph_steps;  // even: every member ends in the buffer it started from
      }
    }
  }
  for (; done < nsteps; ++done) {
    int rc = batch_step_once(b, s);
    if (rc) return rc;
  }
  bool moved = false;
  for (ymkh_ctx* c : b->runs)
    if (!c->dual && c->cur == 1) { int rc = copy_back(c, s); if (rc) return rc; moved = true; }
  // A member moved back to buffer 0 no longer matches the tables of the
  // current parity (built for it starting in buffer 1): rebuild them from
  // every member's current buffer before the next step.
  if (moved) b->dirty = true;
  return 0;
} YMKH_CATCH

int ymkh_batch_check(ymkh_batch* b, void* stream) try {
  if (!b) return set_err(YMKH_EINVAL, "null batch");
  unsigned h = 0;
  CK(cudaMemcpyAsync(&h, b->derr, sizeof h, cudaMemcpyDeviceToHost, (cudaStream_t)stream), "error word D2H");
  CK(cudaStreamSynchronize((cudaStream_t)stream), "error word sync");
  if (h) {
    cudaMemsetAsync(b->derr, 0, sizeof(unsigned), (cudaStream_t)stream);
    return set_err(YMKH_ECUDA, "%s (error word %u)",
                   (h & ERR_BOUNDS) ? "a checked access was out of range and skipped" : "a bounded in-kernel wait timed out",
                   h);
  }
  return 0;
} YMKH_CATCH

int ymkh_batch_set_fct_mode(ymkh_batch* b, int mode) try {
  if (!b || (mode != YMKH_FCT_FUSED && mode != YMKH_FCT_SPLIT)) return set_err(YMKH_EINVAL, "bad FCT mode");
  b->fct_mode = mode;
  b->dirty = true;
  return 0;
} YMKH_CATCH

int ymkh_batch_destroy(ymkh_batch* b) try {
  if (!b) return 0;
  batch_drop_graph(b);
  if (b->ddesc) cudaFree(b->ddesc);
  if (b->dcol) cudaFree(b->dcol);
  if (b->dfirst) cudaFree(b->dfirst);
  if (b->derr) cudaFree(b->derr);
  for (int i = 0; i < ymkh_batch::kAux; ++i) {
    if (b->aux[i]) cudaStreamDestroy(b->aux[i]);
    if (b->join_ev[i]) cudaEventDestroy(b->join_ev[i]);
  }
  if (b->fork_ev) cudaEventDestroy(b->fork_ev);
  delete b;
  return 0;
} YMKH_CATCH

}  // extern "C"

namespace ymkh {
// Error reporting and launch counting for entry points defined in other
// translation units (ymkh_noalloc.cu).
int capi_error(int code, const char* msg) { return set_err(code, "%s", msg); }
void capi_count_launches(int n) { g_launches += n; }
}  // namespace ymkh
