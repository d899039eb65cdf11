// engine.cu -- host side of the C ABI declared in include/nspt_b200.h.
//
// One context = one lattice on one device with its own stream.  nspt_step
// mirrors NsptEvolve (nspt.cc:953-1039) with the reference's Jacobi option:
//   sweep (U -> F, observables, per-link log F)   gauge_wilson
//   swap U <-> F                                  Umu = Fmu   (nspt.cc:992)
//   zero-mode reduction + subtraction             zero_modes_subtraction
//   Fourier-accelerated gauge fixing              FAstochastic_gauge_fixing
// Twisted boundaries are applied inside every neighbour read.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/nspt_b200.h"
#include "kernels.cuh"
#include "fft.cuh"
#include "loops.cuh"
#include "hostcopy.cuh"

using namespace nspt;

struct nspt_ctx {
  int L[4];
  int N;
  unsigned flags;
  double alpha;
  long V;
  int dev, nsm;
  size_t smem_optin;
  cudaStream_t st;
  cudaEvent_t ev0, ev1;
  float last_ms;
  // CUDA events around the first KEV sweep-kernel launches of a call
  static constexpr int KEV = 64;
  cudaEvent_t kev[2 * KEV];
  int kcount;
  double last_kernel_ms;  // average sweep-kernel launch of the last call
  Geo geo;
  int SS;  // slot stride (double2)
  double2 *U, *F;    // link records (kernels.cuh)
  bool unit_flags;   // every link's flag is 1 (false after an upload that says otherwise)
  double2 *plaq[2];  // plaquette records of two slabs of the Jacobi sweep, or none
  size_t plaq_bytes;
  int slab;          // planes of direction 0 per slab
  // held by every call that launches sweeps or a graph of them: another context's
  // creation may take the records back in between (release_records)
  std::recursive_mutex use;
  double2 *Lg;       // per-link logs (zero modes, FA)
  bool snap_valid;   // on the fly, twisted: F holds the step's start field, which reads
                     // across a twisted face see until twist_boundary
  bool lg_current;   // Lg holds log U of the current field (after a sweep with
                     // zero modes and after the zero-mode subtraction)
  double2 *Wg, *Gx;  // FA work planes, gauge transformation records
  double *obs, *obs_tr;  // SweepArgs
  // column sums: obs [12N], obs_tr [<= 8(N+1)], obs_tr2 [8(N+1)], Lg [8(1+9N)]
  double *red;
  double *red_part;  // [COLSUM_CHUNKS][widest row]
  int tr_rows;       // rows of the last sweep's traces per site: 6 (plaquettes) or 4 (links)
  double2 *meas;     // plaquette_measure: per-CTA rows
  double *p2;     // lattice momenta p2hat[4][128] of this context's extents
  double2 *ftw;   // FFT twiddles exp(-2 pi i t / L_d), [4][128] (FA only)
  int gf_grid[4]; // local gauge fixing: the reference's thread grid (ntt, ntx, nty, ntz)
  int gf_form;    // form of the grid-ordered kernels: NSPT_LGF_AUTO, _GROUP or _TEAM
  unsigned long long *dcounter;  // Philox step counter on the device (advanced by k_inc)
  int sweep_warps;               // warps per CTA at most, 0 = as many as fit (nspt_batch_tune_shape)
  double c1;                     // improved action weight (0: Wilson), c0 = 1 - 8 c1
  double *obs_tr2;               // rectangle traces (improved actions)
  int *ff_e;                     // float-float scale exponent used by the sweep (device)
  unsigned long long *ff_mx;     // [N] per-order max |U_k| (bit patterns)
  bool ff_auto;                  // fit the exponent each sweep
  double timeout_s;              // host-side limit on waiting for a call's device work (0: none)
  bool busy;                     // a call returned NSPT_ERR_TIMEOUT; its work may still run
  double2 *loop_part;            // Wilson loops: per-CTA rows and the summed row
  size_t loop_part_n;
  double *noise;  // injected noise
  bool noise_pending;
  bool have_obs;
  uint64_t seed, counter;
  // bumped by every setter that changes what a step launches or the values
  // its kernels take by argument (seed, gauge-fixing grid, sweep shape,
  // float-float scale mode); a CUDA graph captured under another value is
  // stale (batch.cuh)
  std::atomic<uint64_t> launch_gen;
  std::atomic<size_t> bytes;
  std::string err;
};

static const char *kErr[] = {"ok",
                             "invalid argument",
                             "perturbative order outside the supported range",
                             "allocation failed",
                             "CUDA runtime error",
                             "no CUDA device",
                             "call out of sequence",
                             "file I/O error",
                             "device work still running at the time limit"};

extern "C" const char *nspt_error_string(int code) {
  if (code < 0 || code > 8) return "unknown error";
  return kErr[code];
}

extern "C" const char *nspt_last_error(nspt_ctx *ctx) {
  return ctx ? ctx->err.c_str() : "null context";
}

#define CK(call)                                                              \
  do {                                                                        \
    cudaError_t e_ = (call);                                                  \
    if (e_ != cudaSuccess) {                                                  \
      if (ctx) ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_); \
      return NSPT_ERR_CUDA;                                                   \
    }                                                                         \
  } while (0)

// ---------------- memory ----------------

// Every context of the process, so that one that cannot have the memory it needs
// is given the plaquette records of the others, which they can do without.
static struct Contexts {
  std::mutex mu;
  std::vector<nspt_ctx *> all;
} g_ctx;

static void free_records(nspt_ctx *ctx) {
  for (double2 *&p : ctx->plaq) {
    if (p) cudaFree(p);
    p = nullptr;
  }
  ctx->bytes -= ctx->plaq_bytes;
  ctx->plaq_bytes = 0;
}

// The records of all contexts on a device that are in no call back to the driver.
// Their next sweeps form each link's plaquettes anew or find memory again; a graph
// that held the records is captured again (launch_gen).
static bool release_records(int dev) {
  bool any = false;
  std::lock_guard<std::mutex> lock(g_ctx.mu);
  for (nspt_ctx *c : g_ctx.all) {
    std::unique_lock<std::recursive_mutex> use(c->use, std::try_to_lock);
    if (!use || c->dev != dev || !c->plaq_bytes) continue;
    cudaStreamSynchronize(c->st);  // what a call past its time limit left
    free_records(c);
    c->launch_gen++;
    any = true;
  }
  return any;
}

// Device memory that a context on `dev` cannot do without, whatever device is current
static cudaError_t dev_alloc(void **p, size_t n, int dev) {
  const OnDevice current(dev);
  cudaError_t e = cudaMalloc(p, n);
  if (e == cudaErrorMemoryAllocation && release_records(dev)) {
    cudaGetLastError();
    e = cudaMalloc(p, n);
  }
  return e;
}

// ---------------- kernel shapes ----------------

// CTAs (partial rows) of plaquette_measure
constexpr int MEASURE_CTAS = 592;
// sites per slab of the Jacobi sweep at least: 24 k plaquettes, ten rounds of
// the 2368 warps that the GPU holds
constexpr long SLAB_SITES = 4096;

// Lanes of a link's group (wseries.cuh) in a launch of `units` groups: 9 where
// the SMs then have enough warps, 32 where they have not -- because shared
// memory holds few links (sweep of 16 x 16 x 16 x 8, ms with 9 / 32 lanes: 2.2 /
// 2.9 at 8 orders, 5.3 / 5.6 at 14, 6.7 / 6.1 at 16, 13.7 / 11.2 at 24) or
// because the launch is small (1296 links of an on-the-fly step of 12^4 x 8: 5.1
// / 4.0 ms per sweep; 1024 links of 4^4: 67 / 51 us).  Float-float products follow
// the same line; their own would lie lower (12^4, ms with 9 / 32 lanes: 1.44 / 1.83
// at 4 orders, 3.36 / 3.06 at 8, 8.99 / 6.73 at 12).
static int form_lanes(const nspt_ctx *ctx, long units) {
  return ctx->N > 14 || units < 24L * ctx->nsm ? 32 : 9;
}
// Runs with logarithms (zero modes, Fourier-accelerated gauge fixing) at high
// order keep the order of every sum (wseries.cuh, ORDERED).  The difference of
// two orders of summation is 1e-10 of the field's largest entries after 40 steps
// at 13 orders and 4e-7 after 20 steps at 20.
static bool ordered(const nspt_ctx *ctx) {
  return ctx->N > 14 && (ctx->flags & (NSPT_ZEROMODE | NSPT_GF_FA));
}
// Run fn with the form as a constant: for what enters the field, and (measure_form)
// for what has no order to keep.
template <class Fn>
static void measure_form(const nspt_ctx *ctx, long units, Fn fn) {
  if (form_lanes(ctx, units) == 9)
    fn(std::integral_constant<int, 9>());
  else
    fn(std::integral_constant<int, 32>());
}
template <class Fn>
static void with_form(const nspt_ctx *ctx, long units, Fn fn) {
  if (ordered(ctx))
    fn(std::integral_constant<int, ORDERED>());
  else
    measure_form(ctx, units, fn);
}
// Groups per CTA: as many as give an SM the most groups, with 228 KB of shared
// memory per SM, 1 KB of it taken by each CTA, at most ctas_max CTAs per SM
// (registers) of CTA_WARPS warps of 32 / lanes groups; among equals the
// larger CTA.  cap: warps per CTA at most.  gpc 0 when not even one group fits.
struct Shape {
  int warps, gpc;
  size_t smem;
};
static Shape group_shape(int lanes, int ctas_max, int slots, int SS, size_t smem_optin, int cap = CTA_WARPS) {
  const size_t lead = LEAD * sizeof(double2);
  const size_t per = group_stride(slots, SS) * sizeof(double2);
  cap = std::min(cap, CTA_WARPS);
  Shape k = {0, 0, 0};
  long most = 0;
  for (int ctas = 1; ctas <= ctas_max; ctas++) {
    const size_t room = std::min<size_t>(smem_optin, (size_t)228 * 1024 / ctas - 1024);
    const long g = std::min<long>(32L / lanes * cap, room > lead ? (long)((room - lead) / per) : 0);
    if (g * ctas > most) most = g * ctas, k.gpc = (int)g;
  }
  k.warps = std::min(cap, k.gpc);
  k.smem = lead + k.gpc * per;
  return k;
}

// Launch a kernel of a group per unit with `slots` series per group; units too
// few to fill the GPU are spread over the SMs.
template <int G, class... P, class... A>
static int wlaunch(nspt_ctx *ctx, std::integral_constant<int, G>, void (*kernel)(P...), int slots,
                   long units, const char *what, A... args) {
  Shape k = group_shape(glanes<G>(), sm_ctas<G>(), slots, ctx->SS, ctx->smem_optin,
                        ctx->sweep_warps > 0 ? ctx->sweep_warps : CTA_WARPS);
  if (k.gpc < 1) return NSPT_ERR_ORDER;
  k.gpc = (int)std::max<long>(1, std::min<long>(k.gpc, (units + ctx->nsm - 1) / ctx->nsm));
  k.warps = std::min(k.warps, k.gpc);
  k.smem = (LEAD + (size_t)k.gpc * group_stride(slots, ctx->SS)) * sizeof(double2);
  cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)ctx->smem_optin);
  kernel<<<(unsigned)((units + k.gpc - 1) / k.gpc), 32 * k.warps, k.smem, ctx->st>>>(args..., k.gpc);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->err = std::string(what) + ": " + cudaGetErrorString(e);
    return NSPT_ERR_CUDA;
  }
  return NSPT_OK;
}

// ---------------- reductions ----------------

// Column sums (k_colsum) in a fixed order that depends on the sizes alone.
constexpr int COLSUM_CHUNKS = 296;

static int colsum(nspt_ctx *ctx, const double *in, long rows, int width, double *out) {
  const long chunk = std::max<long>(32, (rows + COLSUM_CHUNKS - 1) / COLSUM_CHUNKS);
  const long n = (rows + chunk - 1) / chunk;
  const unsigned cols = (unsigned)((width + 31) / 32);
  k_colsum<<<dim3(cols, (unsigned)n), 256, 0, ctx->st>>>(in, rows, width, chunk, ctx->red_part);
  k_colsum<<<cols, 256, 0, ctx->st>>>(ctx->red_part, n, width, n, out);
  CK(cudaGetLastError());
  return NSPT_OK;
}

// the areas of red
static size_t red_tr(const nspt_ctx *ctx) { return 12 * (size_t)ctx->N; }
static size_t red_tr2(const nspt_ctx *ctx) { return red_tr(ctx) + 8 * (size_t)(ctx->N + 1); }
static size_t red_mm(const nspt_ctx *ctx) { return red_tr2(ctx) + 8 * (size_t)(ctx->N + 1); }
static size_t red_size(const nspt_ctx *ctx) { return red_mm(ctx) + 8 * link_rec(ctx->N); }

static int reduce_sweep_obs(nspt_ctx *ctx) {
  const int N = ctx->N;
  int rc = colsum(ctx, ctx->obs, ctx->V, 12 * N, ctx->red);
  const int w = ctx->tr_rows == 6 ? 6 * (N + 1) : 8 * (N + 1);
  if (!rc) rc = colsum(ctx, ctx->obs_tr, ctx->V, w, ctx->red + red_tr(ctx));
  if (!rc && ctx->c1 != 0.0)
    rc = colsum(ctx, ctx->obs_tr2, ctx->V, 8 * (N + 1), ctx->red + red_tr2(ctx));
  return rc;
}

// The reference's OpenMP thread grid (the context's gf_grid) as the kernels
// walk it: steps = the number of barrier steps.
static LgfGrid thread_grid(const nspt_ctx *ctx, long &steps) {
  LgfGrid gr;
  gr.dmax = -1;
  gr.nthr = 1;
  gr.seg = 1;
  for (int d = 0; d < 4; d++) {
    gr.n[d] = ctx->gf_grid[d];
    gr.bs[d] = ctx->L[d] / gr.n[d];
    gr.nthr *= gr.n[d];
    if (gr.n[d] > 1) gr.dmax = d;
  }
  steps = 1;
  for (int d = 0; d < 4; d++) {
    if (d <= gr.dmax)
      steps *= gr.bs[d];
    else
      gr.seg *= ctx->L[d];
  }
  return gr;
}

// Whether the on-the-fly sweep takes a site's staples ahead of its links
// (k_otf_parts): periodic fields, whose F is free (a twisted one holds the step's
// start field there) and large enough, with no extent of 1 (no link of the site
// is then its own neighbour).  The ORDERED form keeps its order of sums.  Steps
// of many threads at low orders have warps enough to hide a link's chain, and the
// parts' way through memory costs more: in one launch and in parts, 16^4 (4096
// threads) N=6 4.5 and 5.1 ms, N=9 7.1 and 6.5, 24^4 (20736) N=8 19.6 and 20.5,
// N=10 32.4 and 31.6; 12^4 (1296) N=8 3.03 and 2.16, 16*14^3 (2744) N=4 5.4 and
// 3.4, 8^4 (256) N=11 3.9 and 2.1.
// Two launches per site of the walk are also bounded: a call returns at its time
// limit (nspt_set_timeout) only if its launches fit the stream's queue, some 1000,
// and a graph of the step holds a node for each.  So a walk of several sites is
// taken in parts up to OTF_WALK sites in a sweep, although a longer one is twice
// as fast that way (5^4 N=8, one thread: 88 ms in one launch, 50 in 1250; 9^4 925
// and 524, but with a limit of 20 ms the call came back after 503); steps of one
// site each took four launches in the engine's first kernels and take two.
constexpr long OTF_WALK = 256;
static bool otf_in_parts(const nspt_ctx *ctx, const LgfGrid &gr) {
  if (gr.seg > 1 && ctx->V > OTF_WALK * gr.nthr) return false;
  for (int d = 0; d < 4; d++)
    if (ctx->L[d] < 2) return false;
  return ctx->c1 == 0.0 && !ctx->geo.twist && !ordered(ctx) &&
         (gr.nthr < 24L * ctx->nsm || ctx->N > BLK) && (long)OTF_PARTS * gr.nthr <= 4L * ctx->V;
}

// The order in which an ORDERED on-the-fly sweep adds up a link's six staples:
// plane by plane where a barrier step has one site per thread and few threads,
// else one by one.  The engine's first kernels gave such a step a group of lanes
// per plane, on grids that filled 8 warps an SM at most (11 at 16 orders, of 3 x 3
// slots each, would fit), unless told to take a group per thread; a run with
// logarithms at high order keeps what it was begun with (ordered).
static bool otf_by_planes(const nspt_ctx *ctx, const LgfGrid &gr) {
  if (!ordered(ctx) || gr.seg != 1 || ctx->gf_form == NSPT_LGF_GROUP) return false;
  if (ctx->gf_form == NSPT_LGF_TEAM) return true;
  const long slot = ((long)link_rec(ctx->N) + 4) / 8 * 8 + 3;  // 3 (mod 8)
  return gr.nthr <= std::min<long>(228 * 1024 / (9 * slot * (long)sizeof(double2)), 8) * ctx->nsm;
}

// gauge_wilson on the fly (UPDATE_ONTHEFLY, nspt.cc:355-460): one launch per
// barrier step of the thread grid, or two per site of its walk; one group per
// reference thread.
static int launch_sweep_otf(nspt_ctx *ctx, const SweepArgs &a) {
  long steps;
  const LgfGrid gr = thread_grid(ctx, steps);
  int rc = NSPT_OK;
  if (otf_in_parts(ctx, gr)) {
    const long parts = (long)OTF_PARTS * gr.nthr;
    // all of a link's operands at once where every group then still has its place
    const bool wide = gr.nthr * (long)(group_stride(OTF_LINK_SLOTS_WIDE, ctx->SS) * sizeof(double2)) <=
                      ctx->nsm * 200L * 1024;
    for (long p = 0; p < steps; p++)
      for (long r = 0; r < gr.seg && !rc; r++) {
        measure_form(ctx, parts, [&](auto G) {
          rc = wlaunch(ctx, G, k_otf_parts<G.value>, 3, parts, "on-the-fly sweep, staples", a, gr, p,
                       r, ctx->F);
        });
        if (rc) break;
        measure_form(ctx, gr.nthr, [&](auto G) {
          rc = wlaunch(ctx, G, k_otf_links<G.value>,
                       wide ? OTF_LINK_SLOTS_WIDE : OTF_LINK_SLOTS, gr.nthr,
                       "on-the-fly sweep, links", a, gr, p, r, (const double2 *)ctx->F, wide);
        });
      }
    return rc;
  }
  const bool planes = otf_by_planes(ctx, gr);
  with_form(ctx, gr.nthr, [&](auto G) {
    for (long p = 0; p < steps && !rc; p++)
      rc = ctx->c1 != 0.0 ? wlaunch(ctx, G, k_sweep_imp_otf<G.value>, IMP_SLOTS, gr.nthr,
                                    "on-the-fly sweep", a, gr, p)
                          : wlaunch(ctx, G, k_sweep_otf<G.value>, LINK_SLOTS + (planes ? 1 : 0), gr.nthr,
                                    "on-the-fly sweep", a, gr, p, planes);
  });
  return rc;
}

// The Jacobi sweep plaquette by plaquette, slab by slab of direction 0: the
// plaquettes of a slab, then its links.  A slab's links also need the
// plaquettes of the plane before it, kept in the other buffer; the first slab
// takes them from the last plane, whose plaquettes are formed ahead for it.
template <bool FF, int G>
static int launch_sweep_plaq(nspt_ctx *ctx, SweepArgs a) {
  const std::integral_constant<int, G> g;
  const int L0 = ctx->L[0], s0 = ctx->geo.s0;
  auto plaq = [&](int x, int n, int buf) {
    a.site0 = x * s0;
    a.nsite = n * s0;
    a.plaq = ctx->plaq[buf];
    return wlaunch(ctx, g, k_plaq<FF, G>, PLAQ_SLOTS, 6L * a.nsite, "sweep, plaquettes", a);
  };
  int cur = 0, rc = NSPT_OK;
  a.prev = ctx->plaq[0];
  a.prev0 = 0;
  if (ctx->slab < L0) {
    rc = plaq(L0 - 1, 1, 1);
    a.prev = ctx->plaq[1];
    a.prev0 = a.site0;
  }
  for (int x = 0; x < L0 && !rc; x += ctx->slab) {
    rc = plaq(x, std::min(ctx->slab, L0 - x), cur);
    if (!rc)
      rc = wlaunch(ctx, g, k_update<FF, G>, UPDATE_SLOTS, 4L * a.nsite, "sweep, links", a);
    a.prev = a.plaq;
    a.prev0 = a.site0;
    cur ^= 1;
  }
  return rc;
}

static int launch_sweep(nspt_ctx *ctx, const SweepArgs &a) {
  const bool ff = (ctx->flags & NSPT_PRECISION_FF) != 0;
  const long nl = 4 * ctx->V;
  int rc = NSPT_OK;
  with_form(ctx, nl, [&](auto G) {
    constexpr int g = G.value;
    if constexpr (g != ORDERED) {
      if (ctx->tr_rows == 6) {
        if (ctx->plaq[0])
          rc = ff ? launch_sweep_plaq<true, g>(ctx, a) : launch_sweep_plaq<false, g>(ctx, a);
        else
          rc = ff ? wlaunch(ctx, G, k_update_alone<true, g>, ALONE_SLOTS, nl, "sweep", a)
                  : wlaunch(ctx, G, k_update_alone<false, g>, ALONE_SLOTS, nl, "sweep", a);
        return;
      }
    }
    if (ctx->c1 != 0.0)
      rc = wlaunch(ctx, G, k_sweep_imp<g>, IMP_SLOTS, nl, "sweep", a);
    else
      rc = ff ? wlaunch(ctx, G, k_sweep_link<true, g>, LINK_SLOTS, nl, "sweep", a)
              : wlaunch(ctx, G, k_sweep_link<false, g>, LINK_SLOTS, nl, "sweep", a);
  });
  return rc;
}

// Whether the sweep goes plaquette by plaquette: unless the order of the links is
// fixed, the action has rectangles, the sums have an order to keep, or a flag
// other than 1 meets a twisted face (where each link's staples see flags of their
// own).
static bool by_plaquettes(const nspt_ctx *ctx) {
  return !(ctx->flags & NSPT_UPDATE_ONTHEFLY) && ctx->c1 == 0.0 && !ordered(ctx) &&
         (ctx->unit_flags || !ctx->geo.twist);
}

// Plaquette records: of the whole lattice where that is two slabs of SLAB_SITES
// sites or fewer, else of two such slabs, and of smaller ones where they would
// leave less than half of the free memory to others.  Taken at the end of a
// context's creation (0.5 to 0.9 ms, as much as a first sweep of a small lattice)
// and, where they are not held, before a call's sweeps.  Without them each link
// forms its own plaquettes (k_update_alone): 8^4 N=24 2.40 ms instead of 1.05, 12^4
// N=8 2.19 and 1.02, in float-float 9.5 and 3.4.
static void take_records(nspt_ctx *ctx) {
  if (ctx->plaq_bytes || !by_plaquettes(ctx)) return;
  const OnDevice current(ctx->dev);
  size_t room = 0, total = 0;
  if (cudaMemGetInfo(&room, &total) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  const int L0 = ctx->L[0];
  const long plane = ctx->V / L0;
  const size_t rec = (size_t)plane * 18 * link_rec(ctx->N) * sizeof(double2);
  int slab = (int)std::min<long>(L0, (SLAB_SITES + plane - 1) / plane);
  if (2 * slab >= L0) slab = L0;
  auto bytes = [&] { return rec * (slab < L0 ? 2 * slab : L0); };
  while (slab > 1 && bytes() > room / 2) slab = std::min((slab + 1) / 2, L0 / 2);
  if (bytes() > room / 2 || cudaMalloc(&ctx->plaq[0], rec * slab) != cudaSuccess ||
      (slab < L0 && cudaMalloc(&ctx->plaq[1], rec * slab) != cudaSuccess)) {
    cudaGetLastError();
    free_records(ctx);
    return;
  }
  ctx->slab = slab;
  ctx->plaq_bytes = bytes();
  ctx->bytes += ctx->plaq_bytes;
  ctx->launch_gen++;
}

static int do_sweep(nspt_ctx *ctx, double dt, bool use_noise) {
  SweepArgs a;
  memset(&a, 0, sizeof(a));
  a.U = ctx->U;
  a.F = ctx->F;
  a.Lg = (ctx->flags & NSPT_ZEROMODE) ? ctx->Lg : nullptr;
  a.obs = ctx->obs;
  a.obs_tr = ctx->obs_tr;
  a.noise = use_noise ? ctx->noise : nullptr;
  a.seed = ctx->seed;
  a.step = ctx->counter;
  a.stepp = ctx->dcounter;
  a.obs_tr2 = ctx->obs_tr2;
  a.c1 = ctx->c1;
  a.c0 = 1. - 8. * ctx->c1;
  a.ff_scale = ctx->ff_e;
  // QuenchedAllocate: stau = sqrt(tau_g); tau_g /= -(2 NC)  (Quenched.cc:584-589)
  a.stau = sqrt(dt);
  double tg = dt;
  tg /= -(2 * 3);
  a.tau_g = tg;
  a.N = ctx->N;
  a.SS = ctx->SS;
  a.g = ctx->geo;
  a.Ut = ctx->U;
  const bool otf = (ctx->flags & NSPT_UPDATE_ONTHEFLY) != 0;
  ctx->tr_rows = by_plaquettes(ctx) ? 6 : 4;
  if (otf) {
    // in place; with twisted boundaries F keeps the step's start field for
    // the reads across a twisted face (the reference's copy sites)
    a.F = ctx->U;
    if (ctx->geo.twist) {
      if (!ctx->snap_valid) {
        const size_t nb = (size_t)4 * ctx->V * link_rec(ctx->N) * sizeof(double2);
        CK(cudaMemcpyAsync(ctx->F, ctx->U, nb, cudaMemcpyDeviceToDevice, ctx->st));
        ctx->snap_valid = true;
      }
      a.Ut = ctx->F;
    }
  }
  if ((ctx->flags & NSPT_PRECISION_FF) && ctx->ff_auto) {
    // per-order scale of the float-float products, fitted to this field
    CK(cudaMemsetAsync(ctx->ff_mx, 0, ctx->N * sizeof(unsigned long long), ctx->st));
    k_order_absmax<<<dim3(2 * ctx->nsm, ctx->N), 256, 0, ctx->st>>>(ctx->U, ctx->N,
                                                                    (size_t)ctx->V, ctx->ff_mx);
    k_ff_fit<<<1, 1, 0, ctx->st>>>(ctx->ff_mx, ctx->N, ctx->ff_e);
    CK(cudaGetLastError());
  }
  const bool timed = ctx->kcount < nspt_ctx::KEV;
  if (timed) CK(cudaEventRecord(ctx->kev[2 * ctx->kcount], ctx->st));
  int rc = otf ? launch_sweep_otf(ctx, a) : launch_sweep(ctx, a);
  if (rc) return rc;
  if (timed) {
    CK(cudaEventRecord(ctx->kev[2 * ctx->kcount + 1], ctx->st));
    ctx->kcount++;
  }
  rc = reduce_sweep_obs(ctx);
  if (rc) return rc;
  k_inc<<<1, 1, 0, ctx->st>>>(ctx->dcounter);
  CK(cudaGetLastError());
  if (!otf) {
    std::swap(ctx->U, ctx->F);
  }
  ctx->counter++;
  ctx->have_obs = true;
  ctx->lg_current = a.Lg != nullptr;  // the sweep stored log U' per link
  return NSPT_OK;
}

static int do_zero_modes(nspt_ctx *ctx) {
  const int N = ctx->N;
  double *mm = ctx->red + red_mm(ctx);
  int rc = NSPT_OK;
  const int width = 4 * (int)link_rec(N);
  if (ordered(ctx)) {
    k_logsum<<<(width + LOGSUM_COLS - 1) / LOGSUM_COLS, 256, 0, ctx->st>>>(ctx->Lg, ctx->V, width,
                                                                           (double2 *)mm);
    CK(cudaGetLastError());
  } else if ((rc = colsum(ctx, (const double *)ctx->Lg, ctx->V, 2 * width, mm))) {
    return rc;
  }
  with_form(ctx, 4 * ctx->V, [&](auto G) {
    rc = wlaunch(ctx, G, k_zero_modes<G.value>, SERIES_SLOTS, 4 * ctx->V, "zero modes", ctx->U,
                 ctx->Lg, (const double2 *)mm, 1.0 / (double)ctx->V, N, ctx->SS, ctx->geo);
  });
  if (rc == NSPT_OK) ctx->lg_current = true;  // Lg = the new field's log
  return rc;
}

static int fft4d(nspt_ctx *ctx, double2 *data, int sign) {
  const int N = ctx->N;
  const size_t V = (size_t)ctx->V;
  const int strides[4] = {ctx->geo.s0, ctx->geo.s1, ctx->geo.s2, 1};
  for (int d = 3; d >= 0; d--) {
    const int n = ctx->L[d];
    const long nlines = (long)9 * N * (long)(V / n);
    const unsigned grid = (unsigned)((nlines + 127) / 128);
    switch (n) {
      case 2: k_fft_pow2<2><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      case 4: k_fft_pow2<4><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      case 8: k_fft_pow2<8><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      case 16: k_fft_pow2<16><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      case 32: k_fft_pow2<32><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      case 64: k_fft_pow2<64><<<grid, 128, 0, ctx->st>>>(data, nlines, strides[d], V, sign); break;
      default:
        k_fft_direct<<<grid, 128, 0, ctx->st>>>(data, nlines, n, strides[d], V, sign);
    }
    CK(cudaGetLastError());
  }
  return NSPT_OK;
}

// Extents with a compile-time FFT plan (fft.cuh); others use fft4d.
#define NSPT_FFT_SIZES(X) X(2) X(3) X(4) X(5) X(6) X(8) X(10) X(12) X(16) X(20) X(24) X(32)

static bool fft_planned(int n) {
#define NSPT_FFT_CASE(n_) if (n == n_) return true;
  NSPT_FFT_SIZES(NSPT_FFT_CASE)
#undef NSPT_FFT_CASE
  return false;
}

template <int n>
static void fft_t_launch(nspt_ctx *ctx, double2 *data, int inv) {
  const long nlines = (long)9 * ctx->N * (ctx->V / n);
  const unsigned grid = (unsigned)((nlines + 127) / 128);
  const size_t smem = (size_t)128 * (n | 1) * sizeof(double2);
  cudaFuncSetAttribute(k_fft_t<n>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  k_fft_t<n><<<grid, 128, smem, ctx->st>>>(data, nlines, ctx->ftw + 3 * 128, inv);
}

template <int n>
static void fft_strided_launch(nspt_ctx *ctx, double2 *data, int d, int inv) {
  const long nlines = (long)9 * ctx->N * (ctx->V / n);
  const int st = d == 0 ? ctx->geo.s0 : d == 1 ? ctx->geo.s1 : ctx->geo.s2;
  k_fft_strided<n><<<(unsigned)((nlines + 127) / 128), 128, 0, ctx->st>>>(
      data, nlines, st, (size_t)ctx->V, ctx->ftw + d * 128, inv);
}

template <int n>
static void fft_x_launch(nspt_ctx *ctx, double2 *data, double alpha) {
  const long nlines = (long)9 * ctx->N * (ctx->V / n);
  k_fft_x_scale<n><<<(unsigned)((nlines + 127) / 128), 128, 0, ctx->st>>>(
      data, nlines, ctx->geo, ctx->ftw, alpha, ctx->p2);
}

// Wg = iFFT(-alpha / p^2 FFT(Wg)) in seven passes (fft.cuh), or
// NSPT_ERR_ARG when an extent has no compile-time plan.
static int fa_fft_fused(nspt_ctx *ctx, double alpha) {
  for (int d = 0; d < 4; d++)
    if (!fft_planned(ctx->L[d])) return NSPT_ERR_ARG;
  double2 *Wg = ctx->Wg;
  auto t_pass = [&](int inv) {
    switch (ctx->L[3]) {
#define NSPT_FFT_CASE(n_) case n_: fft_t_launch<n_>(ctx, Wg, inv); break;
      NSPT_FFT_SIZES(NSPT_FFT_CASE)
#undef NSPT_FFT_CASE
    }
  };
  auto s_pass = [&](int d, int inv) {
    switch (ctx->L[d]) {
#define NSPT_FFT_CASE(n_) case n_: fft_strided_launch<n_>(ctx, Wg, d, inv); break;
      NSPT_FFT_SIZES(NSPT_FFT_CASE)
#undef NSPT_FFT_CASE
    }
  };
  t_pass(0);
  s_pass(2, 0);
  s_pass(1, 0);
  switch (ctx->L[0]) {  // forward x, -alpha / p^2, backward x
#define NSPT_FFT_CASE(n_) case n_: fft_x_launch<n_>(ctx, Wg, alpha); break;
    NSPT_FFT_SIZES(NSPT_FFT_CASE)
#undef NSPT_FFT_CASE
  }
  s_pass(1, 1);
  s_pass(2, 1);
  t_pass(1);
  CK(cudaGetLastError());
  return NSPT_OK;
}

static int do_fa(nspt_ctx *ctx, double alpha) {
  const int N = ctx->N, SS = ctx->SS;
  const long nl = 4 * ctx->V;
  const Geo geo = ctx->geo;
  cudaStream_t st = ctx->st;
  // log U per link (nspt.cc:874-875); after the zero-mode subtraction Lg
  // already holds it (k_zero_modes)
  int rc = NSPT_OK;
  if (!ctx->lg_current) {
    with_form(ctx, nl, [&](auto G) {
      rc = wlaunch(ctx, G, k_log_links<G.value>, SERIES_SLOTS, nl, "FA logs",
                   (const double2 *)ctx->U, ctx->Lg, N, SS, geo);
    });
    if (rc) return rc;
  }
  k_fa_div<<<dim3((unsigned)((ctx->V + 31) / 32), (unsigned)((9 * N + 31) / 32)), 256, 0, st>>>(
      ctx->Lg, ctx->Wg, N, geo);
  CK(cudaGetLastError());
  rc = fa_fft_fused(ctx, alpha);
  if (rc == NSPT_ERR_ARG) {  // an extent without a compile-time FFT plan
    const size_t tot = (size_t)9 * N * ctx->V;
    const unsigned eg = (unsigned)std::min<size_t>((tot + 255) / 256, (size_t)ctx->nsm * 32);
    if ((rc = fft4d(ctx, ctx->Wg, -1))) return rc;
    k_fa_scale<<<eg, 256, 0, st>>>(ctx->Wg, N, geo, alpha, ctx->p2);
    CK(cudaGetLastError());
    if ((rc = fft4d(ctx, ctx->Wg, +1))) return rc;
  } else if (rc) {
    return rc;
  }
  with_form(ctx, ctx->V, [&](auto G) {
    rc = wlaunch(ctx, G, k_fa_gt<G.value>, SERIES_SLOTS, ctx->V, "FA gauge transform",
                 (const double2 *)ctx->Wg, ctx->Gx, N, SS, geo);
  });
  if (rc) return rc;
  with_form(ctx, nl, [&](auto G) {
    rc = wlaunch(ctx, G, k_fa_apply<G.value>, APPLY_SLOTS, nl, "FA apply", (const double2 *)ctx->U,
                 (const double2 *)ctx->Gx, ctx->F, N, SS, geo);
  });
  if (rc) return rc;
  std::swap(ctx->U, ctx->F);
  ctx->lg_current = false;
  return NSPT_OK;
}

// Whether a barrier step of the local gauge fixing has a team (k_local_gf_team)
// and not a group per reference thread.  A team is the shorter chain, a CTA of 8
// warps for it the dearer occupancy: 12^4 N=8 with blocks of 2 (16 steps of 1296
// threads) takes 1.16 ms with teams and 0.63 with groups, 10^3*8 (500 threads)
// 0.505 and 0.53, 8^4 (256) 0.30 and 0.52, 6*8*8*9 N=11 (48 threads, 9 sites
// each) 1.28 and 3.18.  So teams serve up to two waves of the CTAs that fit, and
// the ORDERED form, with one team on an SM, one: 6*8*8*9 N=15 4.7 and 7.5 ms,
// but 8^4 N=16 2.5 and 2.1.  NSPT_LGF_TEAM asks for no more of them: 16^4 N=4 (4096
// threads) takes 2.7 ms with teams and 0.72 with groups.  Teams and groups have the
// same lanes per link and form every sum alike: the links are the same bit for bit.
template <int G>
static bool team_fits(const nspt_ctx *ctx, long nthr, size_t &smem) {
  smem = (LEAD + (size_t)team_slots<G>() * group_stride(1, ctx->SS)) * sizeof(double2);
  if (ctx->gf_form == NSPT_LGF_GROUP || smem > ctx->smem_optin) return false;
  const long fit = std::min<long>(G == ORDERED ? 1 : 2, (long)(228 * 1024 / (smem + 1024)));
  return nthr <= (G == ORDERED ? 1 : 2) * fit * ctx->nsm;
}

template <int G>
static bool local_gf_team(nspt_ctx *ctx, const double2 *Ut, double alpha, const LgfGrid &gr,
                          long steps, int &rc) {
  size_t smem;
  if (!team_fits<G>(ctx, gr.nthr, smem)) return false;
  cudaFuncSetAttribute(k_local_gf_team<G>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)ctx->smem_optin);
  for (long p = 0; p < steps; p++)
    k_local_gf_team<G><<<(unsigned)gr.nthr, 32 * TEAM_WARPS, smem, ctx->st>>>(
        ctx->U, Ut, ctx->N, ctx->SS, ctx->geo, alpha, gr, p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ctx->err = std::string("local gauge fixing: ") + cudaGetErrorString(e);
    rc = NSPT_ERR_CUDA;
  }
  return true;
}

// stochastic_gauge_fixing (nspt.cc:660-862) with the context's thread
// grid: one launch per barrier step, a team or a group per reference thread.
static int do_local_gf(nspt_ctx *ctx, double alpha) {
  long steps;
  const LgfGrid gr = thread_grid(ctx, steps);
  // reads across a twisted face: the step's start field after an on-the-fly
  // sweep (the reference's copy sites before twist_boundary)
  const double2 *Ut = ctx->snap_valid ? ctx->F : ctx->U;
  ctx->lg_current = false;
  int rc = NSPT_OK;
  if (ordered(ctx) ? local_gf_team<ORDERED>(ctx, Ut, alpha, gr, steps, rc)
                   : local_gf_team<32>(ctx, Ut, alpha, gr, steps, rc))
    return rc;
  with_form(ctx, gr.nthr, [&](auto G) {
    for (long p = 0; p < steps && !rc; p++)
      rc = wlaunch(ctx, G, k_local_gf<G.value>, lgf_slots<G.value>(), gr.nthr, "local gauge fixing", ctx->U, Ut,
                   ctx->N, ctx->SS, ctx->geo, alpha, gr, p);
  });
  return rc;
}

// minb: the smallest block along a split direction.  The reference needs 2
// (threads of one barrier step then share no link); an on-the-fly sweep of
// an improved action needs 3, because its rectangles reach two sites: with
// blocks of 2 the reference's own threaded run races and differs from run
// to run.
static bool grid_ok(const int L[4], const int grid[4], int minb = 2) {
  for (int d = 0; d < 4; d++) {
    if (grid[d] < 1 || L[d] % grid[d]) return false;
    if (grid[d] > 1 && L[d] / grid[d] < minb) return false;
  }
  return true;
}

static int grid_min_block(const nspt_ctx *ctx) {
  return (ctx->flags & NSPT_UPDATE_ONTHEFLY) && ctx->c1 != 0.0 ? 3 : 2;
}

// ---------------- context ----------------

static int upload_constants(nspt_ctx *ctx) {
  double2 om[4][9], omd[4][9];
  memset(om, 0, sizeof(om));
  for (int d = 0; d < 4; d++)
    for (int e = 0; e < 9; e += 4) om[d][e] = make_double2(1.0, 0.0);
  // twistmatrices.h:158-240
  om[1][0] = make_double2(cos(-2. * M_PI / 3.), sin(-2. * M_PI / 3.));
  om[1][8] = make_double2(cos(2. * M_PI / 3.), sin(2. * M_PI / 3.));
  for (int e = 0; e < 9; e++) om[2][e] = make_double2(0, 0), om[3][e] = make_double2(0, 0);
  om[2][1] = om[2][5] = om[2][6] = make_double2(1.0, 0.0);
  om[3][1] = make_double2(cos(-2. * M_PI / 3.), sin(-2. * M_PI / 3.));
  om[3][5] = make_double2(1.0, 0.0);
  om[3][6] = make_double2(cos(2. * M_PI / 3.), sin(2. * M_PI / 3.));
  for (int d = 0; d < 4; d++)
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) omd[d][3 * i + j] = make_double2(om[d][3 * j + i].x, -om[d][3 * j + i].y);
  CK(cudaMemcpyToSymbol(c_om, om, sizeof(om)));
  CK(cudaMemcpyToSymbol(c_omd, omd, sizeof(omd)));
  double p2[4][128];
  memset(p2, 0, sizeof(p2));
  for (int d = 0; d < 4; d++)
    for (int i = 0; i < ctx->L[d]; i++) {  // lattice.h:1144-1169
      double p = 2 * M_PI * i / ctx->L[d];
      double h = sin(p * 0.5);
      h *= 4 * h;
      p2[d][i] = h;
    }
  CK(cudaMemcpy(ctx->p2, p2, sizeof(p2), cudaMemcpyHostToDevice));
  double2 tw[64];
  for (int k = 0; k < 64; k++) {
    double ang = -1.0 * 2.0 * M_PI * (double)k / 64.0;
    tw[k] = make_double2(cos(ang), sin(ang));
  }
  CK(cudaMemcpyToSymbol(c_tw64, tw, sizeof(tw)));
  if (ctx->ftw) {
    std::vector<double2> ftw(4 * 128, make_double2(0.0, 0.0));
    for (int d = 0; d < 4; d++)
      for (int t = 0; t < ctx->L[d]; t++) {
        const double ang = -2.0 * M_PI * (double)t / (double)ctx->L[d];
        ftw[d * 128 + t] = make_double2(cos(ang), sin(ang));
      }
    CK(cudaMemcpy(ctx->ftw, ftw.data(), ftw.size() * sizeof(double2), cudaMemcpyHostToDevice));
  }
  return NSPT_OK;
}

static void free_all(nspt_ctx *ctx) {
  void *ptrs[] = {ctx->U, ctx->F, ctx->Lg, ctx->Wg, ctx->Gx, ctx->p2, ctx->ftw, ctx->dcounter,
                  ctx->loop_part, ctx->obs_tr2, ctx->ff_e, ctx->ff_mx, ctx->plaq[0], ctx->plaq[1],
                  ctx->obs, ctx->obs_tr, ctx->red, ctx->red_part, ctx->meas, ctx->noise};
  for (void *p : ptrs)
    if (p) cudaFree(p);
}

static HostStage g_stage;

extern "C" int nspt_create(const int L[4], int N, unsigned flags, double alpha, nspt_ctx **out) {
  nspt_ctx *ctx = nullptr;
  if (!out || !L) return NSPT_ERR_ARG;
  *out = nullptr;
  if (N < 1 || N > NSPT_MAX_ORDER) return NSPT_ERR_ORDER;
  const unsigned actions = NSPT_ACTION_TLSYM | NSPT_ACTION_IWA | NSPT_ACTION_DBW2;
  const unsigned known = NSPT_TWIST_Y | NSPT_TWIST_Z | NSPT_TWIST_T | NSPT_ZEROMODE | NSPT_GF_FA |
                         NSPT_GF_LOCAL | actions | NSPT_PRECISION_FF | NSPT_UPDATE_ONTHEFLY;
  if (flags & ~known) return NSPT_ERR_ARG;
  // the on-the-fly update is built for the FP64 sweeps
  if ((flags & NSPT_UPDATE_ONTHEFLY) && (flags & NSPT_PRECISION_FF)) return NSPT_ERR_ARG;
  // float-float products are built into the Wilson sweep only
  if ((flags & NSPT_PRECISION_FF) && (flags & actions)) return NSPT_ERR_ARG;
  if (__builtin_popcount(flags & actions) > 1) return NSPT_ERR_ARG;
  // the reference has improved actions with periodic boundaries only (choices.h:110)
  if ((flags & actions) && (flags & (NSPT_TWIST_Y | NSPT_TWIST_Z | NSPT_TWIST_T)))
    return NSPT_ERR_ARG;
  if ((flags & NSPT_GF_FA) && (flags & NSPT_GF_LOCAL)) return NSPT_ERR_ARG;
  long V = 1;
  for (int d = 0; d < 4; d++) {
    if (L[d] < 2 || L[d] > 128) return NSPT_ERR_ARG;
    V *= L[d];
  }
  // the reference defines zero modes and FA only with periodic boundaries
  if ((flags & (NSPT_TWIST_Y | NSPT_TWIST_Z | NSPT_TWIST_T)) && (flags & (NSPT_ZEROMODE | NSPT_GF_FA)))
    return NSPT_ERR_ARG;
  if (V * 4 * 9L * N > (1L << 40)) return NSPT_ERR_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return NSPT_ERR_NODEVICE;
  ctx = new nspt_ctx();
  memset(ctx->L, 0, sizeof(ctx->L));
  for (int d = 0; d < 4; d++) ctx->L[d] = L[d];
  ctx->N = N;
  ctx->flags = flags;
  ctx->alpha = alpha;
  ctx->V = V;
  ctx->U = ctx->F = ctx->Lg = ctx->Wg = ctx->Gx = nullptr;
  ctx->plaq[0] = ctx->plaq[1] = ctx->meas = nullptr;
  ctx->plaq_bytes = 0;
  ctx->slab = L[0];
  ctx->unit_flags = true;
  ctx->tr_rows = 4;
  ctx->p2 = nullptr;
  ctx->ftw = nullptr;
  ctx->dcounter = nullptr;
  ctx->sweep_warps = 0;
  ctx->lg_current = false;
  ctx->snap_valid = false;
  ctx->launch_gen = 0;
  ctx->loop_part = nullptr;
  ctx->loop_part_n = 0;
  ctx->timeout_s = 0.0;
  ctx->busy = false;
  ctx->obs_tr2 = nullptr;
  ctx->ff_e = nullptr;
  ctx->ff_mx = nullptr;
  ctx->ff_auto = true;
  // improved action parameters, Quenched.cc:311-322
  ctx->c1 = (flags & NSPT_ACTION_TLSYM) ? -1.0 / 12.0
          : (flags & NSPT_ACTION_IWA)   ? -0.331
          : (flags & NSPT_ACTION_DBW2)  ? -1.4088
                                        : 0.0;
  // the finest thread grid the reference accepts: blocks of 2 sites where L
  // is even, one thread along odd extents (for an improved action on the
  // fly: blocks of the smallest size >= 3 dividing L)
  for (int d = 0; d < 4; d++) {
    if (grid_min_block(ctx) == 2) {
      ctx->gf_grid[d] = (L[d] % 2 == 0) ? L[d] / 2 : 1;
    } else {
      int b = 3;
      while (L[d] % b) b++;
      ctx->gf_grid[d] = L[d] / b;
    }
  }
  ctx->gf_form = NSPT_LGF_AUTO;
  ctx->obs = ctx->obs_tr = ctx->red = ctx->red_part = ctx->noise = nullptr;
  ctx->noise_pending = false;
  ctx->have_obs = false;
  ctx->seed = 0x5eed5eedULL;
  ctx->counter = 0;
  ctx->last_ms = 0.f;
  ctx->bytes = 0;
  auto fail = [&](int code) {
    free_all(ctx);
    delete ctx;
    return code;
  };
  if (cudaGetDevice(&ctx->dev) != cudaSuccess) return fail(NSPT_ERR_CUDA);
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, ctx->dev) != cudaSuccess) return fail(NSPT_ERR_CUDA);
  ctx->nsm = prop.multiProcessorCount;
  ctx->smem_optin = prop.sharedMemPerBlockOptin;
  Geo &g = ctx->geo;
  for (int d = 0; d < 4; d++) g.L[d] = L[d];
  g.V = (int)V;
  g.s2 = L[3];
  g.s1 = L[2] * L[3];
  g.s0 = L[1] * L[2] * L[3];
  g.twist = 0;
  if (flags & NSPT_TWIST_Y) g.twist |= 2u;
  if (flags & NSPT_TWIST_Z) g.twist |= 4u;
  if (flags & NSPT_TWIST_T) g.twist |= 8u;
  ctx->SS = (int)link_rec(N);
  // every kernel's slots of one warp must fit in a CTA
  if (group_shape(32, 1, 4, ctx->SS, ctx->smem_optin).gpc < 1) return fail(NSPT_ERR_ORDER);
  if (cudaStreamCreateWithFlags(&ctx->st, cudaStreamNonBlocking) != cudaSuccess) return fail(NSPT_ERR_CUDA);
  cudaEventCreate(&ctx->ev0);
  cudaEventCreate(&ctx->ev1);
  for (int i = 0; i < 2 * nspt_ctx::KEV; i++) cudaEventCreate(&ctx->kev[i]);
  ctx->kcount = 0;
  ctx->last_kernel_ms = 0.0;
  const size_t links = (size_t)4 * V * link_rec(N) * sizeof(double2);
  const size_t nl = (size_t)4 * V;
  const size_t width = std::max<size_t>({12 * (size_t)N, 8 * (size_t)(N + 1), 8 * link_rec(N)});
  auto alloc = [&](void **p, size_t n) {
    if (dev_alloc(p, n, ctx->dev) != cudaSuccess) return false;
    ctx->bytes += n;
    return true;
  };
  bool ok = alloc((void **)&ctx->U, links) && alloc((void **)&ctx->F, links) &&
            alloc((void **)&ctx->obs, nl * 3 * N * sizeof(double)) &&
            alloc((void **)&ctx->obs_tr, nl * 2 * (N + 1) * sizeof(double)) &&
            alloc((void **)&ctx->red, red_size(ctx) * sizeof(double)) &&
            alloc((void **)&ctx->red_part, COLSUM_CHUNKS * width * sizeof(double)) &&
            alloc((void **)&ctx->meas, (size_t)MEASURE_CTAS * (N + 1) * sizeof(double2)) &&
            alloc((void **)&ctx->p2, 4 * 128 * sizeof(double)) &&
            alloc((void **)&ctx->dcounter, sizeof(unsigned long long));
  if (ok && (flags & (NSPT_ZEROMODE | NSPT_GF_FA))) ok = alloc((void **)&ctx->Lg, links);
  if (ok && ctx->c1 != 0.0)
    ok = alloc((void **)&ctx->obs_tr2, nl * 2 * (N + 1) * sizeof(double));
  if (ok && (flags & NSPT_PRECISION_FF))
    ok = alloc((void **)&ctx->ff_e, sizeof(int)) &&
         alloc((void **)&ctx->ff_mx, N * sizeof(unsigned long long));
  if (ok && (flags & NSPT_GF_FA))
    ok = alloc((void **)&ctx->Wg, (size_t)9 * N * V * sizeof(double2)) &&
         alloc((void **)&ctx->Gx, links / 4) && alloc((void **)&ctx->ftw, 4 * 128 * sizeof(double2));
  if (!ok) {
    cudaGetLastError();
    cudaStreamDestroy(ctx->st);
    return fail(NSPT_ERR_NOMEM);
  }
  if (upload_constants(ctx) != NSPT_OK) return fail(NSPT_ERR_CUDA);
  if (cudaMemsetAsync(ctx->dcounter, 0, sizeof(unsigned long long), ctx->st) != cudaSuccess ||
      (ctx->ff_e && cudaMemsetAsync(ctx->ff_e, 0, sizeof(int), ctx->st) != cudaSuccess)) {
    cudaStreamDestroy(ctx->st);
    return fail(NSPT_ERR_CUDA);
  }
  g_stage.user(1);
  {
    std::lock_guard<std::mutex> lock(g_ctx.mu);
    g_ctx.all.push_back(ctx);
  }
  {
    std::lock_guard<std::recursive_mutex> in_use(ctx->use);
    take_records(ctx);
  }
  *out = ctx;
  return nspt_cold_start(ctx);
}

extern "C" int nspt_destroy(nspt_ctx *ctx) {
  if (!ctx) return NSPT_ERR_ARG;
  {
    std::lock_guard<std::mutex> lock(g_ctx.mu);
    g_ctx.all.erase(std::find(g_ctx.all.begin(), g_ctx.all.end(), ctx));
  }
  cudaStreamSynchronize(ctx->st);
  free_all(ctx);
  cudaEventDestroy(ctx->ev0);
  cudaEventDestroy(ctx->ev1);
  for (int i = 0; i < 2 * nspt_ctx::KEV; i++) cudaEventDestroy(ctx->kev[i]);
  cudaStreamDestroy(ctx->st);
  delete ctx;
  g_stage.user(-1);
  return NSPT_OK;
}

extern "C" size_t nspt_device_bytes(const nspt_ctx *ctx) { return ctx ? ctx->bytes.load() : 0; }

static void set_unit_flags(nspt_ctx *ctx, bool unit) {
  if (ctx->unit_flags != unit) ctx->launch_gen++;  // the sweep's route may change
  ctx->unit_flags = unit;
}

extern "C" int nspt_cold_start(nspt_ctx *ctx) {
  if (!ctx) return NSPT_ERR_ARG;
  ctx->lg_current = false;
  ctx->snap_valid = false;  // a new field: no stale twisted reads
  set_unit_flags(ctx, true);
  k_cold<<<ctx->nsm * 8, 256, 0, ctx->st>>>(ctx->U, (size_t)4 * ctx->V, ctx->N);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(ctx->st));
  return NSPT_OK;
}

static const size_t kChunkBytes = 64u << 20;

static int field_copy(nspt_ctx *ctx, void *host, void *dev, size_t bytes, bool to_host) {
  CK(cudaStreamSynchronize(ctx->st));
  CK(g_stage.copy(ctx->st, ctx->dev, host, dev, bytes, to_host));
  return NSPT_OK;
}

// What an upload leaves to find out: whether every link's flag is 1
static int read_flags(nspt_ctx *ctx) {
  int *other = (int *)ctx->meas, h = 0;
  CK(cudaMemsetAsync(other, 0, sizeof(int), ctx->st));
  k_other_flags<<<ctx->nsm * 8, 256, 0, ctx->st>>>(ctx->U, (size_t)4 * ctx->V, ctx->N, other);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&h, other, sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  set_unit_flags(ctx, h == 0);
  return NSPT_OK;
}

extern "C" int nspt_upload_links(nspt_ctx *ctx, const void *aos, int A) {
  if (!ctx || !aos || A < ctx->N) return NSPT_ERR_ARG;
  ctx->lg_current = false;
  ctx->snap_valid = false;  // a new field: no stale twisted reads
  const size_t per_site = 4 * (1 + 9 * (size_t)A) * sizeof(double2);
  if (A == ctx->N) {  // the device layout
    const int rc = field_copy(ctx, const_cast<void *>(aos), ctx->U, per_site * ctx->V, false);
    return rc ? rc : read_flags(ctx);
  }
  const int cs = (int)std::max<size_t>(1, std::min<size_t>(kChunkBytes / per_site, ctx->V));
  double2 *buf = nullptr;
  CK(dev_alloc((void **)&buf, per_site * cs, ctx->dev));
  int rc = NSPT_OK;
  for (long s0 = 0; s0 < ctx->V; s0 += cs) {
    const int n = (int)std::min<long>(cs, ctx->V - s0);
    cudaError_t e = cudaMemcpyAsync(buf, (const char *)aos + per_site * s0, per_site * n,
                                    cudaMemcpyHostToDevice, ctx->st);
    if (e == cudaSuccess) {
      k_unpack<<<ctx->nsm * 8, 256, 0, ctx->st>>>(buf, A, (int)s0, n, ctx->U, ctx->N);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
      ctx->err = std::string("upload: ") + cudaGetErrorString(e);
      rc = NSPT_ERR_CUDA;
      break;
    }
  }
  cudaStreamSynchronize(ctx->st);
  cudaFree(buf);
  return rc ? rc : read_flags(ctx);
}

extern "C" int nspt_download_links(nspt_ctx *ctx, void *aos, int A) {
  if (!ctx || !aos || A < ctx->N) return NSPT_ERR_ARG;
  const size_t per_site = (size_t)4 * (1 + 9 * A) * sizeof(double2);
  if (A == ctx->N)  // the device layout
    return field_copy(ctx, aos, ctx->U, per_site * ctx->V, true);
  const int cs = (int)std::max<size_t>(1, std::min<size_t>(kChunkBytes / per_site, ctx->V));
  double2 *buf = nullptr;
  CK(dev_alloc((void **)&buf, per_site * cs, ctx->dev));
  int rc = NSPT_OK;
  for (long s0 = 0; s0 < ctx->V; s0 += cs) {
    const int n = (int)std::min<long>(cs, ctx->V - s0);
    k_pack<<<ctx->nsm * 8, 256, 0, ctx->st>>>(buf, A, (int)s0, n, ctx->U, ctx->N);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
      e = cudaMemcpyAsync((char *)aos + per_site * s0, buf, per_site * n, cudaMemcpyDeviceToHost,
                          ctx->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->st);
    if (e != cudaSuccess) {
      ctx->err = std::string("download: ") + cudaGetErrorString(e);
      rc = NSPT_ERR_CUDA;
      break;
    }
  }
  cudaFree(buf);
  return rc;
}

extern "C" int nspt_set_noise(nspt_ctx *ctx, const double *eta) {
  if (!ctx || !eta) return NSPT_ERR_ARG;
  const size_t n = (size_t)ctx->V * 4 * 8 * sizeof(double);
  if (!ctx->noise) {
    if (dev_alloc((void **)&ctx->noise, n, ctx->dev) != cudaSuccess) {
      cudaGetLastError();
      ctx->noise = nullptr;
      return NSPT_ERR_NOMEM;
    }
    ctx->bytes += n;
  }
  CK(cudaMemcpyAsync(ctx->noise, eta, n, cudaMemcpyHostToDevice, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  ctx->noise_pending = true;
  return NSPT_OK;
}

extern "C" int nspt_seed(nspt_ctx *ctx, uint64_t seed, uint64_t counter) {
  if (!ctx) return NSPT_ERR_ARG;
  ctx->seed = seed;
  ctx->counter = counter;
  ctx->launch_gen++;
  const unsigned long long c = counter;
  CK(cudaMemcpyAsync(ctx->dcounter, &c, sizeof(c), cudaMemcpyHostToDevice, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  return NSPT_OK;
}

extern "C" int nspt_get_seed(nspt_ctx *ctx, uint64_t *seed, uint64_t *counter) {
  if (!ctx || !seed || !counter) return NSPT_ERR_ARG;
  *seed = ctx->seed;
  *counter = ctx->counter;
  return NSPT_OK;
}

// Device time of a call: events on the context's stream around its launches.
// Wait for the context's stream, at most timeout_s seconds when a limit is
// set: the device work itself is never interrupted; past the limit the call
// returns NSPT_ERR_TIMEOUT and the next call waits for that work first.
static int wait_stream(nspt_ctx *ctx, cudaEvent_t done) {
  if (ctx->timeout_s <= 0.0) {
    CK(cudaEventSynchronize(done));
    ctx->busy = false;
    return NSPT_OK;
  }
  const auto t0 = std::chrono::steady_clock::now();
  for (;;) {
    const cudaError_t e = cudaEventQuery(done);
    if (e == cudaSuccess) break;
    if (e != cudaErrorNotReady) CK(e);
    const double el = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (el > ctx->timeout_s) {
      ctx->busy = true;
      char msg[96];
      snprintf(msg, sizeof(msg), "device work still running after %.3g s", el);
      ctx->err = msg;
      return NSPT_ERR_TIMEOUT;
    }
  }
  ctx->busy = false;
  return NSPT_OK;
}

static int timed_begin(nspt_ctx *ctx) {
  if (ctx->busy) {  // the work a timed-out call left behind
    CK(cudaEventRecord(ctx->ev1, ctx->st));
    int rc = wait_stream(ctx, ctx->ev1);
    if (rc) return rc;
  }
  ctx->kcount = 0;
  CK(cudaEventRecord(ctx->ev0, ctx->st));
  return NSPT_OK;
}
static int timed_end(nspt_ctx *ctx) {
  CK(cudaEventRecord(ctx->ev1, ctx->st));
  int rc = wait_stream(ctx, ctx->ev1);
  if (rc) return rc;
  cudaEventElapsedTime(&ctx->last_ms, ctx->ev0, ctx->ev1);
  double sum = 0.0;
  for (int i = 0; i < ctx->kcount; i++) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->kev[2 * i], ctx->kev[2 * i + 1]);
    sum += ms;
  }
  ctx->last_kernel_ms = ctx->kcount ? sum / ctx->kcount : 0.0;
  return NSPT_OK;
}

extern "C" int nspt_gauge_wilson(nspt_ctx *ctx, double dt) {
  if (!ctx || !(dt >= 0.0)) return NSPT_ERR_ARG;
  std::lock_guard<std::recursive_mutex> in_use(ctx->use);
  take_records(ctx);
  int rc = timed_begin(ctx);
  if (rc) return rc;
  const bool use = ctx->noise_pending;
  rc = do_sweep(ctx, dt, use);
  ctx->noise_pending = false;
  if (rc) return rc;
  return timed_end(ctx);
}

extern "C" int nspt_zero_modes_subtraction(nspt_ctx *ctx) {
  if (!ctx) return NSPT_ERR_ARG;
  if (!(ctx->flags & NSPT_ZEROMODE) || !ctx->have_obs) return NSPT_ERR_STATE;
  int rc = timed_begin(ctx);
  if (rc || (rc = do_zero_modes(ctx))) return rc;
  return timed_end(ctx);
}

extern "C" int nspt_fa_gauge_fixing(nspt_ctx *ctx, double alpha) {
  if (!ctx) return NSPT_ERR_ARG;
  if (!(ctx->flags & NSPT_GF_FA)) return NSPT_ERR_STATE;
  int rc = timed_begin(ctx);
  if (rc || (rc = do_fa(ctx, alpha))) return rc;
  return timed_end(ctx);
}

// Sums over planes and sites of the 1x2, 2x2, 2x4 and 4x4 loop traces,
// h[q * (N+1) + k], un-normalised (k_loops, then its per-CTA rows summed)
static int loop_sums(nspt_ctx *ctx, std::vector<double2> &h) {
  const int N = ctx->N, row = 4 * (N + 1);
  const long units = 6L * ctx->V;
  const int lanes = form_lanes(ctx, units);
  const Shape sh = group_shape(lanes, 4, LOOP_SLOTS + LOOP_EXTRA, ctx->SS, ctx->smem_optin);
  if (sh.gpc < 1) return NSPT_ERR_ORDER;
  const int grid = (int)std::min<long>((units + sh.gpc - 1) / sh.gpc, 8L * ctx->nsm);
  const size_t need = (size_t)(grid + 1) * row;
  if (need > ctx->loop_part_n) {
    if (ctx->loop_part) cudaFree(ctx->loop_part);
    ctx->loop_part = nullptr;
    ctx->loop_part_n = 0;
    if (dev_alloc((void **)&ctx->loop_part, need * sizeof(double2), ctx->dev) != cudaSuccess) {
      cudaGetLastError();
      return NSPT_ERR_NOMEM;
    }
    ctx->loop_part_n = need;
  }
  double2 *part = ctx->loop_part, *res = ctx->loop_part + (size_t)grid * row;
  int rc = timed_begin(ctx);
  if (rc) return rc;
  measure_form(ctx, units, [&](auto G) {
    // the two-link lines go where the next sweep's field will
    rc = wlaunch(ctx, G, k_lines<G.value>, 2, 4L * ctx->V, "lines", (const double2 *)ctx->U, ctx->F,
                 N, ctx->SS, ctx->geo);
    if (rc) return;
    cudaFuncSetAttribute(k_loops<G.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)ctx->smem_optin);
    k_loops<G.value><<<grid, 32 * sh.warps, sh.smem, ctx->st>>>(ctx->U, ctx->F, N, ctx->SS,
                                                                ctx->geo, part, sh.gpc);
  });
  if (rc) return rc;
  CK(cudaGetLastError());
  k_rows_sum<<<(row + 127) / 128, 128, 0, ctx->st>>>(part, grid, row, res);
  CK(cudaGetLastError());
  h.resize(row);
  CK(cudaMemcpyAsync(h.data(), res, row * sizeof(double2), cudaMemcpyDeviceToHost, ctx->st));
  return timed_end(ctx);
}

extern "C" int nspt_wilson_loops(nspt_ctx *ctx, double *loops) {
  if (!ctx || !loops) return NSPT_ERR_ARG;
  if (ctx->geo.twist) return NSPT_ERR_STATE;  // the reference has them with periodic bc only
  const int N = ctx->N;
  std::vector<double2> h;
  int rc = loop_sums(ctx, h);
  if (rc) return rc;
  // loopNorm = 1/(3*2*3*V), halved for 1x2 and 2x4 (nspt.cc:1280-1306)
  const double norm = 1. / (3 * 2 * 3 * (double)ctx->V);
  const double fac[4] = {.5 * norm, norm, .5 * norm, norm};
  for (int q = 0; q < 4; q++)
    for (int k = 0; k <= N; k++) {
      loops[2 * (q * (N + 1) + k)] = h[q * (N + 1) + k].x * fac[q];
      loops[2 * (q * (N + 1) + k) + 1] = h[q * (N + 1) + k].y * fac[q];
    }
  return NSPT_OK;
}

extern "C" int nspt_wl2x2(nspt_ctx *ctx, double *loop) {
  if (!ctx || !loop) return NSPT_ERR_ARG;
  if (ctx->geo.twist) return NSPT_ERR_STATE;  // __WILLOOP_2x2__ is periodic only (choices.h:75-78)
  const int N = ctx->N;
  std::vector<double2> h;
  int rc = loop_sums(ctx, h);
  if (rc) return rc;
  // WL2x2 walks each plane's 2x2 loop the other way round from ComputeLoops'
  // 2x2 (mu > nu, along mu first): its trace is the complex conjugate.
  // Normalisation rVol * D18 (nspt.cc:1121).
  const double norm = 1. / (18. * (double)ctx->V);
  for (int k = 0; k <= N; k++) {
    loop[2 * k] = h[(N + 1) + k].x * norm;
    loop[2 * k + 1] = -h[(N + 1) + k].y * norm;
  }
  return NSPT_OK;
}

extern "C" int nspt_local_gauge_fixing(nspt_ctx *ctx, double alpha) {
  if (!ctx) return NSPT_ERR_ARG;
  int rc = timed_begin(ctx);
  if (rc || (rc = do_local_gf(ctx, alpha))) return rc;
  return timed_end(ctx);
}

extern "C" int nspt_set_gf_grid(nspt_ctx *ctx, const int grid[4]) {
  if (!ctx || !grid || !grid_ok(ctx->L, grid, grid_min_block(ctx))) return NSPT_ERR_ARG;
  for (int d = 0; d < 4; d++) ctx->gf_grid[d] = grid[d];
  ctx->launch_gen++;
  return NSPT_OK;
}

extern "C" int nspt_set_local_gf_form(nspt_ctx *ctx, int form) {
  if (!ctx) return NSPT_ERR_ARG;
  if (form != NSPT_LGF_AUTO && form != NSPT_LGF_GROUP && form != NSPT_LGF_TEAM) return NSPT_ERR_ARG;
  ctx->gf_form = form;
  ctx->launch_gen++;
  return NSPT_OK;
}

extern "C" int nspt_step(nspt_ctx *ctx, double dt, int nsteps, int gf_every) {
  if (!ctx || nsteps < 0 || !(dt >= 0.0) || gf_every < 0) return NSPT_ERR_ARG;
  std::lock_guard<std::recursive_mutex> in_use(ctx->use);
  take_records(ctx);
  int rc0 = timed_begin(ctx);
  if (rc0) return rc0;
  for (int s = 0; s < nsteps; s++) {
    const bool use = ctx->noise_pending;
    int rc = do_sweep(ctx, dt, use);
    ctx->noise_pending = false;
    if (rc) return rc;
    if (ctx->flags & NSPT_ZEROMODE)
      if ((rc = do_zero_modes(ctx))) return rc;
    if ((ctx->flags & NSPT_GF_FA) && gf_every > 0 && ((ctx->counter % gf_every) == 0))
      if ((rc = do_fa(ctx, ctx->alpha))) return rc;
    if ((ctx->flags & NSPT_GF_LOCAL) && gf_every > 0 && ((ctx->counter % gf_every) == 0))
      if ((rc = do_local_gf(ctx, ctx->alpha))) return rc;
    ctx->snap_valid = false;  // twist_boundary ends the step (nspt.cc:1025-1027)
  }
  return timed_end(ctx);
}

extern "C" int nspt_twist_boundary(nspt_ctx *ctx) {
  if (!ctx) return NSPT_ERR_ARG;
  ctx->snap_valid = false;
  return NSPT_OK;
}

extern "C" double nspt_last_step_ms(const nspt_ctx *ctx) { return ctx ? ctx->last_ms : 0.0; }
extern "C" double nspt_last_kernel_ms(const nspt_ctx *ctx) {
  return ctx ? ctx->last_kernel_ms : 0.0;
}

extern "C" int nspt_observables(nspt_ctx *ctx, double *plaq, double *norm, double *trU) {
  if (!ctx) return NSPT_ERR_ARG;
  if (!ctx->have_obs) return NSPT_ERR_STATE;
  const int N = ctx->N;
  std::vector<double> r(red_mm(ctx));
  CK(cudaMemcpyAsync(r.data(), ctx->red, r.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  if (plaq) {  // nspt.cc:570-597
    const double *t = r.data() + red_tr(ctx);
    for (int k = 0; k <= N; k++) {
      double re = 0.0, im = 0.0;
      for (int q = 0; q < ctx->tr_rows; q++) {
        re += ctx->tr_rows == 6 ? 4. * t[q * (N + 1) + k] : t[2 * (q * (N + 1) + k)];
        im += ctx->tr_rows == 6 ? 0.0 : t[2 * (q * (N + 1) + k) + 1];
      }
      plaq[2 * k] = re / (double)(72 * ctx->V);
      plaq[2 * k + 1] = im / (double)(72 * ctx->V);
    }
  }
  for (int k = 0; k < N; k++) {
    double nrm = 0.0;
    for (int mu = 0; mu < 4; mu++) {
      const double *o = r.data() + 3 * (size_t)N * mu;
      nrm += o[k];
      if (trU) {
        trU[2 * (mu * N + k)] = o[N + 2 * k] / (double)(3 * ctx->V);
        trU[2 * (mu * N + k) + 1] = o[N + 2 * k + 1] / (double)(3 * ctx->V);
      }
    }
    if (norm) norm[k] = nrm / (double)(12 * ctx->V);
  }
  return NSPT_OK;
}

extern "C" int nspt_set_timeout(nspt_ctx *ctx, double seconds) {
  if (!ctx || !(seconds >= 0.0)) return NSPT_ERR_ARG;
  ctx->timeout_s = seconds;
  return NSPT_OK;
}

extern "C" int nspt_set_ff_scale(nspt_ctx *ctx, int automatic, int e) {
  if (!ctx) return NSPT_ERR_ARG;
  if (!(ctx->flags & NSPT_PRECISION_FF)) {
    ctx->err = "float-float scale: context created without NSPT_PRECISION_FF";
    return NSPT_ERR_STATE;
  }
  ctx->launch_gen++;
  if (automatic) {
    ctx->ff_auto = true;
    return NSPT_OK;
  }
  if ((long)std::abs(e) * ctx->N > 1000) {
    ctx->err = "float-float scale: |e| N above 1000";
    return NSPT_ERR_ARG;
  }
  ctx->ff_auto = false;
  CK(cudaMemcpyAsync(ctx->ff_e, &e, sizeof(int), cudaMemcpyHostToDevice, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  return NSPT_OK;
}

extern "C" int nspt_get_ff_scale(nspt_ctx *ctx, int *e) {
  if (!ctx || !e) return NSPT_ERR_ARG;
  if (!(ctx->flags & NSPT_PRECISION_FF)) {
    ctx->err = "float-float scale: context created without NSPT_PRECISION_FF";
    return NSPT_ERR_STATE;
  }
  CK(cudaMemcpyAsync(e, ctx->ff_e, sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  return NSPT_OK;
}

extern "C" int nspt_rect_observables(nspt_ctx *ctx, double *w2) {
  if (!ctx || !w2) return NSPT_ERR_ARG;
  if (ctx->c1 == 0.0 || !ctx->have_obs) return NSPT_ERR_STATE;
  const int N = ctx->N;
  std::vector<double> r(8 * (N + 1));
  CK(cudaMemcpyAsync(r.data(), ctx->red + red_tr2(ctx), r.size() * sizeof(double),
                     cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  for (int k = 0; k <= N; k++) {  // nspt.cc:586-597
    double re = 0.0, im = 0.0;
    for (int mu = 0; mu < 4; mu++) {
      re += r[2 * (mu * (N + 1) + k)];
      im += r[2 * (mu * (N + 1) + k) + 1];
    }
    w2[2 * k] = re / (double)(72 * ctx->V);
    w2[2 * k + 1] = im / (double)(72 * ctx->V);
  }
  return NSPT_OK;
}

extern "C" int nspt_plaquette_measure(nspt_ctx *ctx, double *plaq) {
  if (!ctx || !plaq) return NSPT_ERR_ARG;
  const int N = ctx->N;
  const long units = 6L * ctx->V;
  const Shape sh = group_shape(form_lanes(ctx, units), 4, MEASURE_SLOTS, ctx->SS, ctx->smem_optin);
  if (sh.gpc < 1) return NSPT_ERR_ORDER;
  const int grid = (int)std::min<long>((units + sh.gpc - 1) / sh.gpc, MEASURE_CTAS);
  measure_form(ctx, units, [&](auto G) {
    cudaFuncSetAttribute(k_plaq_trace<G.value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)ctx->smem_optin);
    k_plaq_trace<G.value><<<grid, 32 * sh.warps, sh.smem, ctx->st>>>(
        ctx->U, link_rec(N), N, ctx->SS, ctx->geo, ctx->meas, N + 1, sh.gpc);
  });
  CK(cudaGetLastError());
  double *tmp = ctx->red + red_mm(ctx);  // free outside zero modes
  int rc = colsum(ctx, (const double *)ctx->meas, grid, 2 * (N + 1), tmp);
  if (rc) return rc;
  std::vector<double2> r(N + 1);
  CK(cudaMemcpyAsync(r.data(), tmp, r.size() * sizeof(double2), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  ctx->have_obs = false;  // the last sweep's observables are to be read before a measurement
  for (int k = 0; k <= N; k++) {  // nspt.cc:1398-1404
    plaq[2 * k] = r[k].x / (double)(ctx->V * 72);
    plaq[2 * k + 1] = r[k].y / (double)(ctx->V * 72);
  }
  return NSPT_OK;
}

extern "C" int nspt_save_config(nspt_ctx *ctx, const char *path, int A) {
  if (!ctx || !path || A < ctx->N) return NSPT_ERR_ARG;
  std::vector<double> host((size_t)ctx->V * 4 * (1 + 9 * A) * 2);
  int rc = nspt_download_links(ctx, host.data(), A);
  if (rc) return rc;
  std::vector<double> plaq(2 * (ctx->N + 1));
  rc = nspt_plaquette_measure(ctx, plaq.data());
  if (rc) return rc;
  std::vector<double> trailer(2 * (A + 1), 0.0);
  std::copy(plaq.begin(), plaq.end(), trailer.begin());
  FILE *f = fopen(path, "wb");
  if (!f) return NSPT_ERR_IO;
  bool ok = fwrite(host.data(), sizeof(double), host.size(), f) == host.size() &&
            fwrite(trailer.data(), sizeof(double), trailer.size(), f) == trailer.size();
  ok = (fclose(f) == 0) && ok;
  return ok ? NSPT_OK : NSPT_ERR_IO;
}

extern "C" int nspt_load_config(nspt_ctx *ctx, const char *path, int A, double *plaq_trailer) {
  if (!ctx || !path || A < ctx->N) return NSPT_ERR_ARG;
  FILE *f = fopen(path, "rb");
  if (!f) return NSPT_ERR_IO;
  std::vector<double> host((size_t)ctx->V * 4 * (1 + 9 * A) * 2);
  std::vector<double> trailer(2 * (A + 1));
  // io::load checks the byte count (QCDenvNODEpt_test.h:370-374)
  fseek(f, 0, SEEK_END);
  const long sz = ftell(f);
  fseek(f, 0, SEEK_SET);
  const long want = (long)((host.size() + trailer.size()) * sizeof(double));
  bool ok = sz == want && fread(host.data(), sizeof(double), host.size(), f) == host.size() &&
            fread(trailer.data(), sizeof(double), trailer.size(), f) == trailer.size();
  fclose(f);
  if (!ok) return NSPT_ERR_IO;
  if (plaq_trailer) std::copy(trailer.begin(), trailer.end(), plaq_trailer);
  return nspt_upload_links(ctx, host.data(), A);
}

extern "C" int nspt_load_lower_order(nspt_ctx *ctx, const char *path, int loworder,
                                     double *plaq_trailer) {
  if (!ctx || !path) return NSPT_ERR_ARG;
  // QCDenvNODEpt_test.h:377-380: no more orders than the field holds
  if (loworder < 1 || loworder > ctx->N) return NSPT_ERR_ORDER;
  const int lo = loworder, N = ctx->N;
  FILE *f = fopen(path, "rb");
  if (!f) return NSPT_ERR_IO;
  const size_t ser_lo = 2 * (1 + 9 * (size_t)lo), ser_n = 2 * (1 + 9 * (size_t)N);
  std::vector<double> file((size_t)ctx->V * 4 * ser_lo);
  std::vector<double> trailer(2 * (lo + 1));
  // the exact byte count of a loworder file (QCDenvNODEpt_test.h:387-390)
  fseek(f, 0, SEEK_END);
  const long sz = ftell(f);
  fseek(f, 0, SEEK_SET);
  const long want = (long)((file.size() + trailer.size()) * sizeof(double));
  bool ok = sz == want && fread(file.data(), sizeof(double), file.size(), f) == file.size() &&
            fread(trailer.data(), sizeof(double), trailer.size(), f) == trailer.size();
  fclose(f);
  if (!ok) return NSPT_ERR_IO;
  // orders 1..lo from the file, every order above zero (QCDenvNODEpt_test.h:396-411)
  std::vector<double> host((size_t)ctx->V * 4 * ser_n, 0.0);
  for (size_t l = 0; l < (size_t)ctx->V * 4; l++)
    std::copy(file.begin() + l * ser_lo, file.begin() + (l + 1) * ser_lo, host.begin() + l * ser_n);
  std::vector<double>().swap(file);
  int rc = nspt_upload_links(ctx, host.data(), N);
  if (rc) return rc;
  // U = exp(reH(log U)) per link (QCDenvNODEpt_test.h:414-417)
  with_form(ctx, 4 * ctx->V, [&](auto G) {
    rc = wlaunch(ctx, G, k_unitarise<G.value>, SERIES_SLOTS, 4 * ctx->V, "unitarise", ctx->U, N,
                 ctx->SS, ctx->geo);
  });
  if (rc) return rc;
  set_unit_flags(ctx, true);
  CK(cudaStreamSynchronize(ctx->st));
  ctx->have_obs = false;
  if (plaq_trailer) std::copy(trailer.begin(), trailer.end(), plaq_trailer);
  return NSPT_OK;
}

extern "C" int nspt_measure_fp64_peak(double *tflops) {
  nspt_ctx *ctx = nullptr;
  if (!tflops) return NSPT_ERR_ARG;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  cudaDeviceProp prop;
  CK(cudaGetDeviceProperties(&prop, dev));
  double *out = nullptr;
  CK(cudaMalloc(&out, sizeof(double)));
  const int blocks = prop.multiProcessorCount * 8, threads = 256, iters = 4096;
  k_fp64_peak<<<blocks, threads>>>(out, 64, 1.0);  // warm-up
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0);
  k_fp64_peak<<<blocks, threads>>>(out, iters, 1.0);
  cudaEventRecord(e1);
  cudaError_t e = cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return NSPT_ERR_CUDA;
  const double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return NSPT_OK;
}

// allocation-free plaquette of a caller-owned device field
#include "noalloc.cuh"

// batches of replicas in one CUDA graph
#include "batch.cuh"
