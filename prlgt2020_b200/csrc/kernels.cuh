// kernels.cuh -- the NSPT Langevin kernels for sm_100a (FP64).
//
// Device layout of a link field: one record of 1 + 9 N double2 per link,
//   U[(4*site + mu) * (1 + 9*N)]                          flag (order 0)
//   U[(4*site + mu) * (1 + 9*N) + 1 + 9*(k-1) + 3*r + c]  order k = 1..N
// the reference's own order of a field (ptGluon_fld, site then mu, row major
// colour), site = lexicographic index with t fastest (GETINDEX, lattice.h:37).
// A kernel takes a link whole, so a link is contiguous: staging one reads 3.4
// KB in a row at 24 orders, where planes of one component each gave 216 pieces
// of 16 bytes, half a 32-byte sector used.  The logarithms (Lg) and the gauge
// transformation (Gx, one record per site) are records too; only the FFT's
// work field is planes, Wg[e * V + site], e = 9*(k-1) + 3*r + c.
//
// Every link update is done by a group of 9 lanes, three to a warp, or by a warp, with a few
// shared-memory series slots (wseries.cuh); a group's work is independent of all
// others.  Only the teams of the local gauge fixing, the transpose of the FFT's
// input and the sums have block barriers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wseries.cuh"

namespace nspt {

struct Geo {
  int L[4];
  int V;
  int s0, s1, s2;  // site strides of directions 0, 1, 2 (direction 3: 1)
  unsigned twist;  // bit d: direction d twisted
};

// exp(-2 pi i k / 64), k < 64, radix-2 FFT twiddles.
__constant__ double2 c_tw64[64];

__device__ __forceinline__ void coords(const Geo &g, int site, int *x) {
  x[0] = site / g.s0;
  int r = site - x[0] * g.s0;
  x[1] = r / g.s1;
  r -= x[1] * g.s1;
  x[2] = r / g.s2;
  x[3] = r - x[2] * g.s2;
}

struct Nb {
  int site;
  unsigned fwd, bwd;  // directions wrapped forward / backward
};

// Site of x + s1*e_d1 + s2*e_d2 (s = -1, 0, +1) with periodic wrap.
__device__ __forceinline__ Nb neighbour(const Geo &g, const int *x, int d1, int s1, int d2 = 0,
                                        int s2 = 0) {
  int y[4];  // selects, not y[d1]: an array indexed at run time lives in memory
#pragma unroll
  for (int d = 0; d < 4; d++) y[d] = x[d] + (d == d1 ? s1 : 0) + (d == d2 ? s2 : 0);
  Nb n;
  n.fwd = 0;
  n.bwd = 0;
#pragma unroll
  for (int d = 0; d < 4; d++) {
    if (y[d] < 0) {
      y[d] += g.L[d];
      n.bwd |= 1u << d;
    } else if (y[d] >= g.L[d]) {
      y[d] -= g.L[d];
      n.fwd |= 1u << d;
    }
  }
  n.site = y[0] * g.s0 + y[1] * g.s1 + y[2] * g.s2 + y[3];
  return n;
}

// double2 in the record of one link
__host__ __device__ __forceinline__ size_t link_rec(int N) { return 1 + 9 * (size_t)N; }
// record of link (mu, site)
__device__ __forceinline__ size_t link_at(int mu, int site, int N) {
  return ((size_t)site * 4 + mu) * link_rec(N);
}

// This lane's group: its index in the grid and the offset of its slots.  A CTA
// holds gpc groups, as many as shared memory has room for (at most 32 / G per
// warp), dealt to its warps as evenly as possible; lanes without a group, and
// groups past the last unit, have none of the work (ok false).
__host__ __device__ __forceinline__ int group_stride(int slots, int SS) {
  const int n = slots * SS;
  return n + (4 - n % 8 + 8) % 8;
}
template <int G>
struct Grp {
  int lane, slot;
  long id;
  bool ok;
  __device__ __forceinline__ Grp(int slots, int SS, int gpc, long units) {
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5, g = (threadIdx.x & 31) / glanes<G>();
    const int base = gpc / nw, extra = gpc - base * nw;
    const int gi = w * base + min(w, extra) + g;
    lane = glane<G>();
    slot = LEAD + gi * group_stride(slots, SS);
    id = (long)blockIdx.x * gpc + gi;
    ok = g < base + (w < extra ? 1 : 0) && id < units;
  }
};

// Link (mu, n.site) into a slot, twisted where its read crossed a twisted
// face.  Two or three links are begun together and waited for once.
template <int G>
__device__ __forceinline__ void stage_link(int slot, const double2 *U, int mu, const Nb &n, int N) {
  wstage<G>(slot, U + link_at(mu, n.site, N), (int)link_rec(N));
}
template <int G>
__device__ __forceinline__ void twist_link(int slot, const Nb &n, const Geo &g, int N) {
  const unsigned tb = n.bwd & g.twist, tf = n.fwd & g.twist;
  if (tb | tf) wtwist<G>(slot, tb, tf, N);
}
__device__ __forceinline__ Nb nb_self(int site) {
  Nb n;
  n.site = site;
  n.fwd = n.bwd = 0;
  return n;
}

// ---------------- Philox-4x32-10 (Salmon et al., SC'11) ----------------
__device__ __forceinline__ uint4 philox(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    if (r) {
      k.x += 0x9E3779B9u;
      k.y += 0xBB67AE85u;
    }
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
  }
  return c;
}
// uniform in (0, 1] with 53 random bits
__device__ __forceinline__ double u53(uint32_t hi, uint32_t lo) {
  const uint64_t b = ((((uint64_t)hi) << 32) | lo) >> 11;
  return ((double)b + 1.0) * (1.0 / 9007199254740992.0);
}
// 8 Gaussians of variance 1/2 (the reference's convention, MyRand.cc:119-127):
// pair q (0..3), which lane q of the link's warp draws
__device__ __forceinline__ double2 philox_gauss_pair(uint64_t seed, uint64_t step, uint32_t link,
                                                     int q) {
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const uint4 r = philox(make_uint4(link, (uint32_t)q, (uint32_t)step, (uint32_t)(step >> 32)), key);
  const double u1 = u53(r.x, r.y), u2 = u53(r.z, r.w);
  const double rad = sqrt(-log(u1));
  double sn, cs;
  sincospi(2.0 * u2, &sn, &cs);
  return make_double2(rad * cs, rad * sn);
}

// SU3rand mapping of 8 Gaussians to a row-major 3x3, MyMath.cc:256-292.
__device__ __forceinline__ void su3rand(const double *g, double2 *P) {
  const double sD3 = 0.57735026918962573;  // sqrt(1/3), MyMath.h:49
#pragma unroll
  for (int e = 0; e < 9; e++) P[e] = cz();
  P[1] = make_double2(g[1], g[0]);
  P[3] = make_double2(-g[1], g[0]);
  P[2] = make_double2(g[3], g[2]);
  P[6] = make_double2(-g[3], g[2]);
  P[5] = make_double2(g[5], g[4]);
  P[7] = make_double2(-g[5], g[4]);
  const double gg = g[7] * sD3;
  P[0] = make_double2(0.0, gg + g[6]);
  P[4] = make_double2(0.0, gg - g[6]);
  P[8] = make_double2(0.0, -2. * gg);
}

struct SweepArgs {
  const double2 *U;
  double2 *F;
  double2 *Lg;         // log(U') per link (zero modes) or null
  double *obs;         // per link: norm[N], then Tr U_k[N] (re, im)
  double *obs_tr;      // traces of U * staples: plaquette path, per (site, plane) Re Tr P of
                       // orders 0..N; link path, per link Tr (re, im) of orders 0..N
  double *obs_tr2;     // link path: per link Tr(U * rectangle staples), improved actions
  const double *noise; // [V][4][8] injected, or null (Philox)
  uint64_t seed, step;
  const unsigned long long *stepp;  // device step counter (Philox), or null: use step
  double c0, c1;       // improved action weights (Quenched.cc:311-322)
  const int *ff_scale;  // float-float products: per-order scale exponent (device)
  double tau_g, stau;  // -dt/6, sqrt(dt)  (Quenched.cc:584-589)
  int N, SS;
  // on-the-fly update: what a read across a twisted face sees, the field of
  // the step's start (the reference's copy sites, refreshed by
  // twist_boundary only); the Jacobi sweep reads U there too
  const double2 *Ut;
  Geo g;
  // plaquette path: slab of sites [site0, site0 + nsite), its plaquette records
  // (plaq), and those of the sites from prev0 on (prev), which hold the plane
  // before the slab
  double2 *plaq;
  const double2 *prev;
  int site0, nsite, prev0;
};

// ---------------- shared parts of the sweeps ----------------

// Observables of a link in slot Y (nspt.cc:393-402): Re Tr(U_k U_k^dag), Tr U_k
template <int G>
__device__ __forceinline__ void link_obs(const SweepArgs &a, int Y, size_t link) {
  const double2 *sm = wsm();
  const int N = a.N;
  double *o = a.obs + link * 3 * N;
  for (int k = 1 + glane<G>(); k <= N; k += glanes<G>()) {
    const double2 *u = sm + Y + 9 * k - 8;
    double nrm = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      double d = 0.0;
#pragma unroll
      for (int l = 0; l < 3; l++) d += u[3 * i + l].x * u[3 * i + l].x + u[3 * i + l].y * u[3 * i + l].y;
      nrm += d;
    }
    o[k - 1] = nrm;
    const double2 t = cadd(cadd(u[0], u[4]), u[8]);
    o[N + 2 * (k - 1)] = t.x;
    o[N + 2 * (k - 1) + 1] = t.y;
  }
}

// Traces of orders 0..N of a slot (ptSU3::Tr, QCDpt.cc:115-122)
template <int G>
__device__ __forceinline__ void link_trace(double *o, int P, int N) {
  const double2 *sm = wsm();
  for (int k = glane<G>(); k <= N; k += glanes<G>()) {
    const double2 *p = sm + P + 9 * k - 8;
    const double2 f = sm[P];
    const double2 t = k ? cadd(cadd(p[0], p[4]), p[8]) : make_double2(3. * f.x, 3. * f.y);
    o[2 * k] = t.x;
    o[2 * k + 1] = t.y;
  }
}

// The rest of a link update once the force (nspt.cc:392-416) is in slot W:
// W = reH(W) tau_g - stau eta (nspt.cc:416-423), F = exp(W) U (nspt.cc:429)
// and the link's log for the zero modes (nspt.cc:432-439).  All slots are
// overwritten; link = mu V + site numbers the noise.
template <int G, bool DAG>
__device__ __forceinline__ void update_link(const SweepArgs &a, int T, int Y, int W, int mu,
                                            int site) {
  double2 *sm = wsm();
  const int N = a.N, lane = glane<G>();
  double gz[8];
  {
    double2 p = cz();
    if (lane < 4) {
      if (a.noise) {
        const double *e = a.noise + ((size_t)site * 4 + mu) * 8 + 2 * lane;
        p = make_double2(__ldg(e), __ldg(e + 1));
      } else {
        p = philox_gauss_pair(a.seed, a.stepp ? *a.stepp : a.step,
                              (uint32_t)((long)mu * a.g.V + site), lane);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int src = gfirst<G>() + q;
      gz[2 * q] = __shfl_sync(gmask<G>(), p.x, src);
      gz[2 * q + 1] = __shfl_sync(gmask<G>(), p.y, src);
    }
  }
  for (int k = 1 + lane; k <= N; k += glanes<G>()) {
    double2 *p = sm + W + 9 * k - 8;
    double2 m[9];
#pragma unroll
    for (int e = 0; e < 9; e++) m[e] = p[e];
    reh3(m);
#pragma unroll
    for (int e = 0; e < 9; e++) m[e] = cscale(m[e], a.tau_g);
    if (k == 1) {
      double2 eta[9];
      su3rand(gz, eta);
#pragma unroll
      for (int e = 0; e < 9; e++) m[e] = csub(m[e], cscale(eta[e], a.stau));
    }
#pragma unroll
    for (int e = 0; e < 9; e++) p[e] = m[e];
  }
  if (lane == 0) sm[W] = cz();
  gsync<G>();
  const int E = ser_exp_to<G, DAG>(W, T, Y, N);
  const size_t at = link_at(mu, site, N);
  wstage<G>(T, a.U + at, (int)link_rec(N));
  wstage_wait<G>();
  ser_mul<G>(T, E, T, N, DAG ? MUL_DAG : 0);
  wstore<G>(a.F + at, T, (int)link_rec(N));
  if (a.Lg) {
    gsync<G>();
    ser_log<G, DAG>(T, W, Y, N);
    wstore<G>(a.Lg + at, Y, (int)link_rec(N));
  }
}

// ---------------- Jacobi sweep, plaquette by plaquette ----------------
//
// gauge_wilson, nspt.cc:362-439.  The six staples of a link take 12 products
// and U times their sum one more.  A plaquette x, mu < nu has four of them in
// common with its other links: with
//   A = U_mu(x) U_nu(x+mu),  B = U_nu(x) U_mu(x+nu),  P = A B^dag,
// the upper staples (QCDenvNODEpt_test.h:555) give
//   U_mu(x) [U_nu(x+mu) B^dag] = P  and  U_nu(x) [U_mu(x+nu) A^dag] = P^dag,
// and the lower ones (QCDenvNODEpt_test.h:556) are A^dag U_nu(x) for the link
// (mu, x+nu) and B^dag U_mu(x) for the link (nu, x+mu).  Five products per
// plaquette, 7.5 per link, and one more for U times the sum of the three lower
// staples: 8.5 products per link instead of 13.  All four traces of the
// plaquette are Tr P or its conjugate.
//
// The three results of a plaquette (P and the two lower staples) go through
// global memory as records, slab by slab of direction 0 (SweepArgs): 62 KB per
// site at 24 orders, written and read once, 0.02 us per site at the HBM's rate
// where the sweep takes 0.3.
constexpr int PLAQ_SLOTS = 3;

__device__ __forceinline__ void plane_dirs(int pl, int &mu, int &nu) {
  mu = pl < 3 ? 0 : (pl < 5 ? 1 : 2);
  nu = pl < 3 ? pl + 1 : (pl < 5 ? pl - 1 : 3);
}
__device__ __forceinline__ int plane_of(int mu, int nu) {  // mu < nu
  return mu == 0 ? nu - 1 : mu + nu;
}
// record q (0: P, 1: lower staple of (mu, x+nu), 2: of (nu, x+mu)) of plane pl
// of the s-th site of a slab
__device__ __forceinline__ size_t plaq_at(long s, int pl, int q, int N) {
  return ((size_t)(s * 6 + pl) * 3 + q) * link_rec(N);
}

template <bool FF, int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_plaq(SweepArgs a, int gpc) {
  const Grp<G> w(PLAQ_SLOTS, a.SS, gpc, 6L * a.nsite);
  if (!w.ok) return;
  const int N = a.N, S0 = w.slot, S1 = S0 + a.SS, S2 = S1 + a.SS;
  const int ffe = FF ? *a.ff_scale : 0;
  const int s = (int)(w.id / 6), pl = (int)(w.id - 6 * (long)s), site = a.site0 + s;
  int mu, nu, x[4];
  plane_dirs(pl, mu, nu);
  coords(a.g, site, x);
  const Nb self = nb_self(site), um = neighbour(a.g, x, mu, 1), un = neighbour(a.g, x, nu, 1);
  stage_link<G>(S0, a.U, mu, self, N);
  stage_link<G>(S1, a.U, nu, um, N);
  stage_link<G>(S2, a.U, nu, self, N);
  wstage_wait<G>();
  twist_link<G>(S1, um, a.g, N);
  ser_mul_x<FF, G>(S1, S0, S1, N, ffe, MUL_DAG);                                  // A
  stage_link<G>(S0, a.U, mu, un, N);
  cp_commit();
  ser_mul_x<FF, G>(0, S1, S2, N, ffe, MUL_DA, a.plaq + plaq_at(s, pl, 1, N));     // A^dag U_nu
  wstage_wait<G>();
  twist_link<G>(S0, un, a.g, N);
  ser_mul_x<FF, G>(S2, S2, S0, N, ffe, MUL_DAG);                                  // B
  stage_link<G>(S0, a.U, mu, self, N);
  cp_commit();
  ser_mul_x<FF, G>(S1, S1, S2, N, ffe, MUL_DB);                                   // P
  wstore<G>(a.plaq + plaq_at(s, pl, 0, N), S1, (int)link_rec(N));
  const double2 *sm = wsm();
  double *o = a.obs_tr + ((size_t)site * 6 + pl) * (N + 1);
  for (int k = w.lane; k <= N; k += glanes<G>()) {
    const double2 *p = sm + S1 + 9 * k - 8;
    o[k] = k ? p[0].x + p[4].x + p[8].x : 3. * sm[S1].x;
  }
  wstage_wait<G>();
  ser_mul_x<FF, G>(0, S2, S0, N, ffe, MUL_DA, a.plaq + plaq_at(s, pl, 2, N));     // B^dag U_mu
}

constexpr int UPDATE_SLOTS = 3;

// Second half of the Jacobi sweep, per link (mu, x): the force from the
// plaquette records, then the update.
template <bool FF, int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_update(SweepArgs a, int gpc) {
  const Grp<G> w(UPDATE_SLOTS, a.SS, gpc, 4L * a.nsite);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int N = a.N, T = w.slot, Y = T + a.SS, W = Y + a.SS, n = (int)link_rec(N);
  const int site = a.site0 + (int)(w.id >> 2), mu = (int)(w.id & 3);
  int x[4];
  coords(a.g, site, x);
  stage_link<G>(Y, a.U, mu, nb_self(site), N);
  cp_commit();
  // W = the three lower staples: of the plaquette at x - nu, twisted as a
  // whole where x - nu is across a twisted face (the product of twisted links
  // is the twisted product)
  const double2 *low[3];
  unsigned crossed = 0;
#pragma unroll
  for (int h = 0; h < 3; h++) {
    const int nu = h + (h >= mu ? 1 : 0), pl = mu < nu ? plane_of(mu, nu) : plane_of(nu, mu);
    const Nb d = neighbour(a.g, x, nu, -1);
    const int ls = d.site - a.site0;
    const bool here = ls >= 0 && ls < a.nsite;
    low[h] = (here ? a.plaq : a.prev) +
             plaq_at(here ? ls : d.site - a.prev0, pl, mu < nu ? 1 : 2, N);
    if (d.bwd & a.g.twist) crossed |= 1u << h;
  }
  if (!crossed) {
    for (int e = w.lane; e < n; e += glanes<G>())
      sm[W + e] = cadd(cadd(__ldg(low[0] + e), __ldg(low[1] + e)), __ldg(low[2] + e));
  } else {
#pragma unroll
    for (int h = 0; h < 3; h++) {
      wstage<G>(T, low[h], n);
      wstage_wait<G>();
      if (crossed >> h & 1) wtwist<G>(T, 1u << (h + (h >= mu ? 1 : 0)), 0u, N);
      for (int e = w.lane; e < n; e += glanes<G>())
        sm[W + e] = h ? cadd(sm[W + e], sm[T + e]) : sm[T + e];
      gsync<G>();
    }
  }
  cp_wait0();
  gsync<G>();
  link_obs<G>(a, Y, (size_t)site * 4 + mu);
  ser_mul_x<FF, G>(W, Y, W, N, FF ? *a.ff_scale : 0, 0);
  // the upper staples: U_mu(x) times their sum is P of the planes where mu is
  // the first direction and P^dag where it is the second (nu < mu: h < mu)
  const double2 *up[3];
#pragma unroll
  for (int h = 0; h < 3; h++) {
    const int nu = h + (h >= mu ? 1 : 0);
    up[h] = a.plaq + plaq_at(w.id >> 2, mu < nu ? plane_of(mu, nu) : plane_of(nu, mu), 0, N);
  }
  for (int e = 1 + w.lane; e < n; e += glanes<G>()) {
    const int k9 = (e - 1) / 9 * 9, m = e - 1 - k9, et = 1 + k9 + 3 * (m % 3) + m / 3;
    double2 v = sm[W + e];
#pragma unroll
    for (int h = 0; h < 3; h++)
      v = cadd(v, h < mu ? cconj(__ldg(up[h] + et)) : __ldg(up[h] + e));
    sm[W + e] = v;
  }
  gsync<G>();
  update_link<G, false>(a, T, Y, W, mu, site);
}

// The same sweep without the records, for contexts that found no memory for
// them: a link forms its six plaquettes itself, with the products of k_plaq and
// the sums of k_update in their order, so that the field has the same bits
// whichever way a sweep went.  16 products per link instead of 8.5.
constexpr int ALONE_SLOTS = 4;

// Record q of plaquette (x, mu < nu) in S1 (q = 0, 1) or S2 (q = 2): see plaq_at
template <bool FF, int G>
__device__ __forceinline__ int plaq_part(const SweepArgs &a, int S0, int S1, int S2, int q, int mu,
                                         int nu, int site, int ffe) {
  const int N = a.N;
  int x[4];
  coords(a.g, site, x);
  const Nb self = nb_self(site), um = neighbour(a.g, x, mu, 1), un = neighbour(a.g, x, nu, 1);
  stage_link<G>(S2, a.U, nu, self, N);
  if (q != 2) {
    stage_link<G>(S0, a.U, mu, self, N);
    stage_link<G>(S1, a.U, nu, um, N);
    wstage_wait<G>();
    twist_link<G>(S1, um, a.g, N);
    ser_mul_x<FF, G>(S1, S0, S1, N, ffe, MUL_DAG);  // A
  }
  if (q == 1) {
    ser_mul_x<FF, G>(S1, S1, S2, N, ffe, MUL_DA);
    return S1;
  }
  stage_link<G>(S0, a.U, mu, un, N);
  wstage_wait<G>();
  twist_link<G>(S0, un, a.g, N);
  ser_mul_x<FF, G>(S2, S2, S0, N, ffe, MUL_DAG);  // B
  if (q == 0) {
    ser_mul_x<FF, G>(S1, S1, S2, N, ffe, MUL_DB);
    return S1;
  }
  stage_link<G>(S0, a.U, mu, self, N);
  wstage_wait<G>();
  ser_mul_x<FF, G>(S2, S2, S0, N, ffe, MUL_DA);
  return S2;
}

template <bool FF, int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_update_alone(SweepArgs a, int gpc) {
  const Grp<G> w(ALONE_SLOTS, a.SS, gpc, 4L * a.g.V);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int N = a.N, n = (int)link_rec(N), ffe = FF ? *a.ff_scale : 0;
  const int S0 = w.slot, S1 = S0 + a.SS, S2 = S1 + a.SS, W = S2 + a.SS;
  const int site = (int)(w.id >> 2), mu = (int)(w.id & 3);
  int x[4];
  coords(a.g, site, x);
  // t < 3: the lower staples into W; t >= 3: U_mu(x) W, then the plaquettes at x
#pragma unroll 1
  for (int t = 0; t < 6; t++) {
    const int h = t % 3, nu = h + (h >= mu ? 1 : 0);
    if (t == 3) {
      stage_link<G>(S0, a.U, mu, nb_self(site), N);
      wstage_wait<G>();
      link_obs<G>(a, S0, (size_t)site * 4 + mu);
      ser_mul_x<FF, G>(W, S0, W, N, ffe, 0);
    }
    const bool first = mu < nu;
    const Nb d = neighbour(a.g, x, nu, -1);
    const int S = plaq_part<FF, G>(a, S0, S1, S2, t >= 3 ? 0 : first ? 1 : 2, first ? mu : nu,
                                   first ? nu : mu, t >= 3 ? site : d.site, ffe);
    if (t < 3) {
      if (d.bwd & a.g.twist) wtwist<G>(S, 1u << nu, 0u, N);
      for (int e = w.lane; e < n; e += glanes<G>()) sm[W + e] = h ? cadd(sm[W + e], sm[S + e]) : sm[S + e];
    } else {
      for (int e = 1 + w.lane; e < n; e += glanes<G>()) {
        const int k9 = (e - 1) / 9 * 9, m = e - 1 - k9, et = 1 + k9 + 3 * (m % 3) + m / 3;
        sm[W + e] = cadd(sm[W + e], first ? sm[S + e] : cconj(sm[S + et]));
      }
      if (first) {
        double *o = a.obs_tr + ((size_t)site * 6 + plane_of(mu, nu)) * (N + 1);
        for (int k = w.lane; k <= N; k += glanes<G>()) {
          const double2 *p = sm + S + 9 * k - 8;
          o[k] = k ? p[0].x + p[4].x + p[8].x : 3. * sm[S].x;
        }
      }
    }
    gsync<G>();
  }
  update_link<G, false>(a, S0, S1, W, mu, site);
}

// ---------------- sweeps link by link ----------------

// Thread grid of the reference's OpenMP build (choices.h:124-128): n[d]
// threads along direction d (ntt, ntx, nty, ntz), blocks of bs[d] sites
// (Quenched.cc:518-531).  Threads take a barrier after every iteration of
// the deepest split direction dmax (nspt.cc:796-815); between two barriers a
// thread walks a segment of seg sites.
struct LgfGrid {
  int n[4], bs[4];
  int dmax;   // -1 when no direction is split
  int nthr;
  long seg;
};

// The sites one reference thread visits in one barrier step of
// stochastic_gauge_fixing (nspt.cc:731-828): thread tid owns block b of the
// grid; the barrier step fixes the offset rel inside the split directions;
// the directions that are not split are walked whole, the last fastest.
struct LgfWalk {
  int b[4], rel[4];
  __device__ __forceinline__ LgfWalk(const LgfGrid &gr, long tid, long step) {
    b[0] = (int)(tid / ((long)gr.n[1] * gr.n[2] * gr.n[3]));
    b[1] = (int)((tid / ((long)gr.n[2] * gr.n[3])) % gr.n[1]);
    b[2] = (int)((tid / gr.n[3]) % gr.n[2]);
    b[3] = (int)(tid % gr.n[3]);
    long q = step;
#pragma unroll
    for (int d = 3; d >= 0; d--) {
      rel[d] = 0;
      if (d <= gr.dmax) {
        rel[d] = (int)(q % gr.bs[d]);
        q /= gr.bs[d];
      }
    }
  }
  // coordinates of the r-th site of the walk
  __device__ __forceinline__ void site(const LgfGrid &gr, const Geo &geo, long r, int *x) const {
    long t = r;
#pragma unroll
    for (int d = 3; d >= 0; d--) {
      if (d <= gr.dmax) {
        x[d] = gr.bs[d] * b[d] + rel[d];
      } else {
        x[d] = (int)(t % geo.L[d]);
        t /= geo.L[d];
      }
    }
  }
};

// A link of a chain into a slot (not waited for).  Otf (on-the-fly update):
// a read across a twisted face comes from the step's start field.
template <int G>
__device__ __forceinline__ void chain_stage(const SweepArgs &a, int slot, int d, const Nb &n) {
  const bool cross = ((n.fwd | n.bwd) & a.g.twist) != 0;
  stage_link<G>(slot, cross ? a.Ut : a.U, d, n, a.N);
}

// Wilson update of link (mu, site) by its six staples: each as its chain of
// links, multiplied left to right in T with the third link in Y, daggers taken
// by the product:
//   upper U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag          (QCDenvNODEpt_test.h:555)
//   lower U_nu(x+mu-nu)^dag U_mu(x-nu)^dag U_nu(x-nu)    (QCDenvNODEpt_test.h:556)
// For the on-the-fly update, whose links must be visited in order, and for
// fields with flags other than 1 across twisted faces.
//
// The six are added up one by one in W; with a slot Z (ORDERED, see
// otf_by_planes) a plane's two first, then the planes: (p0 + p1) + p2.
template <bool FF, int G>
__device__ __forceinline__ void link_one(const SweepArgs &a, int T, int Y, int W, int mu,
                                         int site, int Z = -1) {
  const int N = a.N, ffe = FF ? *a.ff_scale : 0;
  const bool planes = G == ORDERED && Z >= 0;
  int x[4];
  coords(a.g, site, x);
  const Nb self = nb_self(site);
#pragma unroll 1
  for (int h = 0; h < 6; h++) {
    const int q = h >> 1, nu = q + (q >= mu ? 1 : 0);
    const bool up = !(h & 1);
    const Nb l0 = up ? neighbour(a.g, x, mu, 1) : neighbour(a.g, x, nu, -1, mu, 1);
    const Nb l1 = neighbour(a.g, x, nu, up ? 1 : -1);
    chain_stage<G>(a, T, nu, l0);
    chain_stage<G>(a, Y, mu, l1);
    wstage_wait<G>();
    twist_link<G>(T, l0, a.g, N);
    twist_link<G>(Y, l1, a.g, N);
    ser_mul_x<FF, G>(T, T, Y, N, ffe, up ? MUL_DB : MUL_DA | MUL_DB);
    const Nb l2 = up ? self : l1;
    chain_stage<G>(a, Y, nu, l2);
    wstage_wait<G>();
    twist_link<G>(Y, l2, a.g, N);
    ser_mul_x<FF, G>(planes && q ? Z : W, T, Y, N, ffe,
                     (up ? MUL_DB : MUL_DAG) | ((planes ? !up : h > 0) ? MUL_ACC : 0));
    if (planes && q && !up) {
      double2 *sm = wsm();
      for (int e = glane<G>(); e < (int)link_rec(N); e += glanes<G>())
        sm[W + e] = cadd(sm[W + e], sm[Z + e]);
      gsync<G>();
    }
  }
  chain_stage<G>(a, Y, mu, self);
  wstage_wait<G>();
  const size_t link = (size_t)site * 4 + mu;
  link_obs<G>(a, Y, link);
  ser_mul_x<FF, G>(W, Y, W, N, ffe, MUL_DAG);
  link_trace<G>(a.obs_tr + link * 2 * (N + 1), W, N);
  gsync<G>();
  update_link<G, true>(a, T, Y, W, mu, site);
}

constexpr int LINK_SLOTS = 3;

template <bool FF, int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_sweep_link(SweepArgs a, int gpc) {
  const Grp<G> w(LINK_SLOTS, a.SS, gpc, 4L * a.g.V);
  if (!w.ok) return;
  link_one<FF, G>(a, w.slot, w.slot + a.SS, w.slot + 2 * a.SS, (int)(w.id & 3), (int)(w.id >> 2));
}

// gauge_wilson with UPDATE_ONTHEFLY, the reference's default (choices.h:61,
// nspt.cc:355-460): one barrier step of its OpenMP thread grid.  One group per
// reference thread walks that thread's sites (LgfWalk) and updates their links
// in place, mu = 0..3, each seeing the links updated before it; the threads of
// one barrier step touch disjoint links.
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_sweep_otf(SweepArgs a, LgfGrid gr, long step, bool planes, int gpc) {
  const Grp<G> w(LINK_SLOTS + (planes ? 1 : 0), a.SS, gpc, gr.nthr);
  if (!w.ok) return;
  const LgfWalk walk(gr, w.id, step);
#pragma unroll 1
  for (long r = 0; r < 4 * gr.seg; r++) {
    int x[4];
    walk.site(gr, a.g, r >> 2, x);
    const int site = x[0] * a.g.s0 + x[1] * a.g.s1 + x[2] * a.g.s2 + x[3];
    link_one<false, G>(a, w.slot, w.slot + a.SS, w.slot + 2 * a.SS, (int)(r & 3), site,
                       planes ? w.slot + 3 * a.SS : -1);
    // the next link's copies read what this one wrote
    __threadfence();
    gsync<G>();
  }
}

// The on-the-fly update of a periodic field in two launches per site of the walk.
// What a site's four links need of other sites' links does not change while they
// are updated one after the other: the 12 lower staples (two products each) and
// the 6 corners U_mu(x+nu)^dag after U_nu(x+mu), each of which serves the upper
// staples of both its links.  k_otf_parts forms them, all independent (unit
// t * nthr + thread: the groups of a warp mostly do the same part), and
// k_otf_links is left with 5 products and an exponential per link in a row
// instead of 13.  12^4 N=8 (16 steps of 1296 threads): a step took 190 us in one
// launch and takes 45 and 90; bound by the latency of the links' chains, 9 warps
// on an SM (otf_in_parts has the other sizes).
constexpr int OTF_PARTS = 18, OTF_LINK_SLOTS = 3, OTF_LINK_SLOTS_WIDE = 8;

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_otf_parts(SweepArgs a, LgfGrid gr, long step, long r, double2 *parts, int gpc) {
  const Grp<G> w(3, a.SS, gpc, (long)OTF_PARTS * gr.nthr);
  if (!w.ok) return;
  const int T = w.slot, Y = T + a.SS, Z = Y + a.SS, N = a.N;
  const int t = (int)(w.id / gr.nthr), thr = (int)(w.id - (long)t * gr.nthr);
  int x[4], mu, nu;
  LgfWalk(gr, thr, step).site(gr, a.g, r, x);
  const bool corner = t >= 12;
  if (corner) {
    plane_dirs(t - 12, mu, nu);
  } else {
    mu = t / 3;
    nu = t - 3 * mu;
    nu += nu >= mu ? 1 : 0;
  }
  const Nb l0 = corner ? neighbour(a.g, x, mu, 1) : neighbour(a.g, x, nu, -1, mu, 1);
  const Nb l1 = neighbour(a.g, x, nu, corner ? 1 : -1);
  stage_link<G>(T, a.U, nu, l0, N);
  stage_link<G>(Y, a.U, mu, l1, N);
  if (!corner) stage_link<G>(Z, a.U, nu, l1, N);
  wstage_wait<G>();
  ser_mul<G>(T, T, Y, N, corner ? MUL_DB : MUL_DA | MUL_DB);
  if (!corner) ser_mul<G>(T, T, Z, N, MUL_DAG);
  wstore<G>(parts + (size_t)w.id * link_rec(N), T, (int)link_rec(N));
}

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_otf_links(SweepArgs a, LgfGrid gr, long step, long r, const double2 *parts, bool wide, int gpc) {
  const Grp<G> w(wide ? OTF_LINK_SLOTS_WIDE : OTF_LINK_SLOTS, a.SS, gpc, gr.nthr);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int N = a.N, n = (int)link_rec(N), lane = glane<G>();
  // sum, corners, the site's links: wide, a slot for each of the three and of the four
  const int step_slot = wide ? a.SS : 0;
  const int W = w.slot, T = W + a.SS, S = T + a.SS + 2 * step_slot;
  const size_t part = (size_t)gr.nthr * n;
  parts += (size_t)w.id * n;
  int x[4];
  LgfWalk(gr, w.id, step).site(gr, a.g, r, x);
  const int site = x[0] * a.g.s0 + x[1] * a.g.s1 + x[2] * a.g.s2 + x[3];
#pragma unroll 1
  for (int mu = 0; mu < 4; mu++) {
    auto stage = [&](int q) {
      const int nu = q + (q >= mu ? 1 : 0);
      wstage<G>(T + q * step_slot, parts + (12 + plane_of(min(mu, nu), max(mu, nu))) * part, n);
      wstage<G>(S + nu * step_slot, a.U + link_at(nu, site, N), n);
    };
    const int Y = S + mu * step_slot;
    if (wide) {
      for (int q = 0; q < 3; q++) stage(q);
      wstage<G>(Y, a.U + link_at(mu, site, N), n);
    } else {
      stage(0);
    }
    const double2 *low = parts + 3 * mu * part;
    for (int e = lane; e < n; e += glanes<G>())
      sm[W + e] = cadd(cadd(low[e], low[part + e]), low[2 * part + e]);
    wstage_wait<G>();
#pragma unroll 1
    for (int q = 0; q < 3; q++) {
      const int nu = q + (q >= mu ? 1 : 0);
      ser_mul<G>(W, T + q * step_slot, S + nu * step_slot, N,
                 (mu < nu ? MUL_DB : MUL_DA | MUL_DB) | MUL_ACC);
      if (!wide) {
        if (q < 2)
          stage(q + 1);
        else
          wstage<G>(Y, a.U + link_at(mu, site, N), n);
        wstage_wait<G>();
      }
    }
    link_obs<G>(a, Y, (size_t)site * 4 + mu);
    ser_mul<G>(W, Y, W, N, MUL_DAG);
    link_trace<G>(a.obs_tr + ((size_t)site * 4 + mu) * 2 * (N + 1), W, N);
    gsync<G>();
    update_link<G, true>(a, T, Y, W, mu, site);
    // the next link's copies read what this one wrote
    __threadfence();
    gsync<G>();
  }
}

// ---------------- improved gauge actions ----------------

// Sweep with an improved gauge action (TLSYM, IWA, DBW2; periodic boundaries):
// gauge_wilson, nspt.cc:272-308.  Besides the Wilson staples W, the six 2x1
// rectangles of staple2x1 (QCDenvNODEpt_test.h:579-611) per plane go to W2; the
// force is c0 U W + c1 U W2, and Tr(U W2) is the w2 observable.  Every staple
// is a chain of links (daggered where the reference takes a dagger of a path:
// dag(A B C) = C^dag B^dag A^dag), multiplied left to right in T.
//
// The chains of a plane as a table: link (direction m: mu, n: nu; offsets
// along mu and nu; dagger) and what follows its product: nothing, the sum W,
// or the sum W2.  Two rectangles begin with a Wilson staple's first two links,
// whose product serves both:
//   upper U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag, and
//   U_nu(x+mu) U_mu(x+nu)^dag U_mu(x-mu+nu)^dag U_nu(x-mu)^dag U_mu(x-mu);
//   lower U_nu(x+mu-nu)^dag U_mu(x-nu)^dag U_nu(x-nu), and
//   U_nu(x+mu-nu)^dag U_mu(x-nu)^dag U_mu(x-mu-nu)^dag U_nu(x-mu-nu) U_mu(x-mu).
constexpr int IMP_SLOTS = 4;
struct ImpStep {
  signed char start, is_nu, i, j, dag, sum;  // sum: 0 T *= link, 1 W += T link, 2 W2 += T link
};
constexpr int IMP_STEPS = 32;
__constant__ ImpStep c_imp[IMP_STEPS] = {
    {1, 1, 1, 0, 0, 0},   {0, 0, 0, 1, 1, 0},   {0, 1, 0, 0, 1, 1},  // upper Wilson
    {0, 0, -1, 1, 1, 0},  {0, 1, -1, 0, 1, 0},  {0, 0, -1, 0, 0, 2},
    {1, 1, 1, -1, 1, 0},  {0, 0, 0, -1, 1, 0},  {0, 1, 0, -1, 0, 1},  // lower Wilson
    {0, 0, -1, -1, 1, 0}, {0, 1, -1, -1, 0, 0}, {0, 0, -1, 0, 0, 2},
    {1, 1, 1, 0, 0, 0},   {0, 1, 1, 1, 0, 0},   {0, 0, 0, 2, 1, 0},
    {0, 1, 0, 1, 1, 0},   {0, 1, 0, 0, 1, 2},
    {1, 0, 1, 0, 0, 0},   {0, 1, 2, 0, 0, 0},   {0, 0, 1, 1, 1, 0},
    {0, 0, 0, 1, 1, 0},   {0, 1, 0, 0, 1, 2},
    {1, 1, 1, -1, 1, 0},  {0, 1, 1, -2, 1, 0},  {0, 0, 0, -2, 1, 0},
    {0, 1, 0, -2, 0, 0},  {0, 1, 0, -1, 0, 2},
    {1, 0, 1, 0, 0, 0},   {0, 1, 2, -1, 1, 0},  {0, 0, 1, -1, 1, 0},
    {0, 0, 0, -1, 1, 0},  {0, 1, 0, -1, 0, 2}};

template <int G>
__device__ __forceinline__ void imp_one(const SweepArgs &a, int T, int Y, int W, int W2, int mu,
                                        int site) {
  double2 *sm = wsm();
  const int N = a.N, lane = glane<G>(), n = (int)link_rec(N);
  int x[4];
  coords(a.g, site, x);
  bool dag0 = false;  // T still holds the chain's first link as stored, daggered or not
#pragma unroll 1
  for (int h = 0; h < 3 * IMP_STEPS; h++) {
    const int p = h / IMP_STEPS, nu = p + (p >= mu ? 1 : 0);
    const ImpStep st = c_imp[h - p * IMP_STEPS];
    int y[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
    for (int d = 0; d < 4; d++) {
      y[d] += (d == mu ? st.i : 0) + (d == nu ? st.j : 0);
      y[d] = ((y[d] % a.g.L[d]) + a.g.L[d]) % a.g.L[d];
    }
    const int at = y[0] * a.g.s0 + y[1] * a.g.s1 + y[2] * a.g.s2 + y[3];
    const int slot = st.start ? T : Y;
    wstage<G>(slot, a.U + link_at(st.is_nu ? nu : mu, at, N), n);
    if (st.start) {  // waited for with the second link
      dag0 = st.dag != 0;
      continue;
    }
    wstage_wait<G>();
    const unsigned mode = MUL_DAG | (dag0 ? MUL_DA : 0) | (st.dag ? MUL_DB : 0);
    if (st.sum == 0) {
      ser_mul<G>(T, T, Y, N, mode);
      dag0 = false;
    } else {
      // a plane's first term of each sum is the third and the sixth step
      const bool first = p == 0 && (h == 2 || h == 5);
      ser_mul<G>(st.sum == 1 ? W : W2, T, Y, N, mode | (first ? 0 : MUL_ACC));
    }
  }
  // U W and U W2 (nspt.cc:286-303), traces, force c0 U W + c1 U W2
  wstage<G>(Y, a.U + link_at(mu, site, N), n);
  wstage_wait<G>();
  const size_t link = (size_t)site * 4 + mu;
  link_obs<G>(a, Y, link);
  ser_mul<G>(W, Y, W, N, MUL_DAG);
  ser_mul<G>(W2, Y, W2, N, MUL_DAG);
  link_trace<G>(a.obs_tr + link * 2 * (N + 1), W, N);
  link_trace<G>(a.obs_tr2 + link * 2 * (N + 1), W2, N);
  gsync<G>();
  for (int e = lane; e < n; e += glanes<G>()) sm[W + e] = cadd(cscale(sm[W + e], a.c0), cscale(sm[W2 + e], a.c1));
  gsync<G>();
  update_link<G, true>(a, T, Y, W, mu, site);
}

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_sweep_imp(SweepArgs a, int gpc) {
  const Grp<G> w(IMP_SLOTS, a.SS, gpc, 4L * a.g.V);
  if (!w.ok) return;
  imp_one<G>(a, w.slot, w.slot + a.SS, w.slot + 2 * a.SS, w.slot + 3 * a.SS, (int)(w.id & 3),
             (int)(w.id >> 2));
}

// The improved-action sweep on the fly: as k_sweep_otf
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>()) k_sweep_imp_otf(SweepArgs a, LgfGrid gr, long step, int gpc) {
  const Grp<G> w(IMP_SLOTS, a.SS, gpc, gr.nthr);
  if (!w.ok) return;
  const LgfWalk walk(gr, w.id, step);
#pragma unroll 1
  for (long r = 0; r < 4 * gr.seg; r++) {
    int x[4];
    walk.site(gr, a.g, r >> 2, x);
    const int site = x[0] * a.g.s0 + x[1] * a.g.s1 + x[2] * a.g.s2 + x[3];
    imp_one<G>(a, w.slot, w.slot + a.SS, w.slot + 2 * a.SS, w.slot + 3 * a.SS, (int)(r & 3), site);
    __threadfence();
    gsync<G>();
  }
}

// ---------------- plaquette measurement ----------------

// Re Tr of the product of two slots' series, op(A) B^dag, orders 0..N, a lane
// per order: Tr(X Y^dag)_k = sum over entries of X_ij conj(Y_ij)
__device__ __forceinline__ double2 trace_dag(int X, int Y, int k) {
  const double2 *sm = wsm();
  const double2 x0 = sm[X], y0 = sm[Y];
  if (k == 0) return cscale(cmul(x0, cconj(y0)), 3.0);
  const double2 *xk = sm + X + 9 * k - 8, *yk = sm + Y + 9 * k - 8;
  double2 s = cadd(cmul(x0, cconj(cadd(cadd(yk[0], yk[4]), yk[8]))),
                   cmul(cadd(cadd(xk[0], xk[4]), xk[8]), cconj(y0)));
  for (int i = 1; i < k; i++) {
    const double2 *p = sm + X + 9 * i - 8, *q = sm + Y + 9 * (k - i) - 8;
#pragma unroll
    for (int e = 0; e < 9; e++) cfma(s, p[e], cconj(q[e]));
  }
  return s;
}

constexpr int MEASURE_SLOTS = 4;


// plaquette_measure (nspt.cc:1362-1383): the sum over links of Tr(U * staples)
// meets every plaquette four times, as Tr P or its conjugate, so a plaquette
// takes two products and a trace.  Field: records of `ser` double2 per link.
// A twisted link has flag 1 in the view of the link whose staple crosses the
// face (nspt.cc:115-121); where stored flags are not 1 the four views differ and
// are summed one by one.  Warps walk the plaquettes grid-stride, a lane per
// order; a CTA adds its warps' sums in order into partial[blockIdx].
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_plaq_trace(const double2 *U, size_t ser, int N, int SS, Geo g, double2 *partial, int row, int gpc) {
  const long units = 6L * g.V;
  const Grp<G> w(MEASURE_SLOTS, SS, gpc, units);
  double2 *sm = wsm();
  const int S0 = w.slot, S1 = S0 + SS, S2 = S1 + SS, S3 = S2 + SS, n = (int)link_rec(N);
  constexpr int PL = G == 32 ? 2 : 6;  // orders per lane, of 49 at most
  double2 acc[PL];
#pragma unroll
  for (int h = 0; h < PL; h++) acc[h] = cz();
#pragma unroll 1
  for (long u = w.ok ? w.id : units; u < units; u += (long)gridDim.x * gpc) {
    const int site = (int)(u / 6), pl = (int)(u - 6L * site);
    int mu, nu, x[4];
    plane_dirs(pl, mu, nu);
    coords(g, site, x);
    const Nb um = neighbour(g, x, mu, 1), un = neighbour(g, x, nu, 1);
    const bool cm = um.fwd & g.twist, cn = un.fwd & g.twist;
    bool odd = false;
#pragma unroll 1
    for (int view = 0; view < (odd ? 3 : 1); view++) {
      gsync<G>();
      wstage<G>(S0, U + ((size_t)site * 4 + mu) * ser, n);
      wstage<G>(S1, U + ((size_t)um.site * 4 + nu) * ser, n);
      wstage<G>(S2, U + ((size_t)site * 4 + nu) * ser, n);
      wstage<G>(S3, U + ((size_t)un.site * 4 + mu) * ser, n);
      wstage_wait<G>();
      const double2 f1 = sm[S1], f3 = sm[S3];
      if (cm || cn) {
        auto not1 = [&](double2 f) { return f.x != 1.0 || f.y != 0.0; };
        odd = not1(sm[S0]) || not1(f1) || not1(sm[S2]) || not1(f3);
        gsync<G>();
      }
      twist_link<G>(S1, um, g, N);
      twist_link<G>(S3, un, g, N);
      if (view && w.lane == 0) {
        // view 1: of the link (mu, x+nu), view 2: of (nu, x+mu)
        if (view == 1 && cn) sm[S0] = sm[S1] = sm[S2] = make_double2(1.0, 0.0), sm[S3] = f3;
        if (view == 2 && cm) sm[S0] = sm[S2] = sm[S3] = make_double2(1.0, 0.0), sm[S1] = f1;
      }
      gsync<G>();
      ser_mul<G>(S1, S0, S1, N);
      ser_mul<G>(S3, S2, S3, N);
#pragma unroll
      for (int h = 0; h < PL; h++) {
        const int k = w.lane + glanes<G>() * h;
        if (k > N) continue;
        const double2 t = trace_dag(S1, S3, k);
        if (view == 0) acc[h].x += (odd ? 2. : 4.) * t.x;
        if (view == 1) acc[h] = cadd(acc[h], cconj(t));
        if (view == 2) acc[h] = cadd(acc[h], t);
      }
    }
  }
  __syncthreads();
  if (w.ok) {
    const int gi = (int)(w.id - (long)blockIdx.x * gpc);
#pragma unroll
    for (int h = 0; h < PL; h++)
      if (w.lane + glanes<G>() * h <= N) sm[gi * (N + 1) + w.lane + glanes<G>() * h] = acc[h];
  }
  __syncthreads();
  const long left = units - (long)blockIdx.x * gpc;
  for (int k = threadIdx.x; k <= N; k += blockDim.x) {
    double2 t = cz();
    for (int q = 0; q < gpc && q < left; q++) t = cadd(t, sm[q * (N + 1) + k]);
    partial[(size_t)blockIdx.x * row + k] = t;
  }
}

// Sums over the lattice of the logs' records, one per mu and entry, in the order
// that ORDERED runs keep: 256 partial sums over the sites s = t (mod 256), added
// as a tree.  A block takes LOGSUM_COLS neighbouring entries.
constexpr int LOGSUM_COLS = 8;
__global__ void __launch_bounds__(256)
    k_logsum(const double2 *__restrict__ Lg, long V, int width, double2 *out) {
  __shared__ double2 sh[256];
  const int t = threadIdx.x, c0 = blockIdx.x * LOGSUM_COLS;
  double2 acc[LOGSUM_COLS];
#pragma unroll
  for (int c = 0; c < LOGSUM_COLS; c++) acc[c] = cz();
  for (long s = t; s < V; s += 256) {
    const double2 *p = Lg + (size_t)s * width + c0;
#pragma unroll
    for (int c = 0; c < LOGSUM_COLS; c++)
      if (c0 + c < width) acc[c] = cadd(acc[c], p[c]);
  }
#pragma unroll
  for (int c = 0; c < LOGSUM_COLS; c++) {
    sh[t] = acc[c];
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
      if (t < w) sh[t] = cadd(sh[t], sh[t + w]);
      __syncthreads();
    }
    if (t == 0 && c0 + c < width) out[c0 + c] = sh[0];
    __syncthreads();
  }
}

// Advance a device step counter by one (a kernel, so that it replays
// inside a captured CUDA graph).
__global__ void k_inc(unsigned long long *c) { *c += 1ull; }

// U = exp(reH(log U - MM[mu]/V)) per link: zero_modes_subtraction,
// nspt.cc:605-654 (log U is the per-link log stored by the sweep; MM: its
// sums over the lattice, one record per mu).  The exponent Y = reH(log U -
// MM/V) goes back into Lg: log(exp(Y)) = Y holds exactly for truncated series
// (one variable, so the log and exp series invert each other order by order),
// so Lg then holds log U of the new field, which FA gauge fixing would
// otherwise recompute (nspt.cc:874-875).
constexpr int SERIES_SLOTS = 3;

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_zero_modes(double2 *U, double2 *Lg, const double2 *MM, double rvol, int N, int SS, Geo geo,
                 int gpc) {
  const Grp<G> w(SERIES_SLOTS, SS, gpc, 4L * geo.V);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int P = w.slot, Y = P + SS, R = Y + SS, n = (int)link_rec(N);
  double2 *lg = Lg + (size_t)w.id * n;
  const double2 *mm = MM + (size_t)(w.id & 3) * n;
  for (int e = w.lane; e < n; e += glanes<G>()) {
    const double2 m = __ldg(mm + e);  // MM / V rounded before it is subtracted
    sm[P + e] = make_double2(lg[e].x - __dmul_rn(m.x, rvol), lg[e].y - __dmul_rn(m.y, rvol));
  }
  gsync<G>();
  ser_reH<G>(P, N);
  wstore<G>(lg, P, n);
  wstore<G>(U + (size_t)w.id * n, ser_exp_to<G, false>(P, Y, R, N), n);
}

// U = exp(reH(log U)) per link: the unitarisation the reference applies to
// a configuration loaded with fewer orders than it evolves
// (ptGluon_fld::loadlowerorder, QCDenvNODEpt_test.h:414-417).  Flag 1.
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_unitarise(double2 *U, int N, int SS, Geo geo, int gpc) {
  const Grp<G> w(SERIES_SLOTS, SS, gpc, 4L * geo.V);
  if (!w.ok) return;
  const int X = w.slot, Y = X + SS, R = Y + SS, n = (int)link_rec(N);
  wstage<G>(X, U + (size_t)w.id * n, n);
  wstage_wait<G>();
  ser_log<G, false>(X, Y, R, N);
  ser_reH<G>(R, N);
  wstore<G>(U + (size_t)w.id * n, ser_exp_to<G, false>(R, Y, X, N), n);
}

// Lg = log(U) per link (the logs FAstochastic_gauge_fixing needs, nspt.cc:874-875).
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_log_links(const double2 *U, double2 *Lg, int N, int SS, Geo geo, int gpc) {
  const Grp<G> w(SERIES_SLOTS, SS, gpc, 4L * geo.V);
  if (!w.ok) return;
  const int X = w.slot, Y = X + SS, R = Y + SS, n = (int)link_rec(N);
  wstage<G>(X, U + (size_t)w.id * n, n);
  wstage_wait<G>();
  ser_log<G, false>(X, Y, R, N);
  wstore<G>(Lg + (size_t)w.id * n, R, n);
}

// G(x) = exp(reH(Wg(x) / V))  (nspt.cc:902-906), a record per site.
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_fa_gt(const double2 *Wg, double2 *Gx, int N, int SS, Geo geo, int gpc) {
  const Grp<G> w(SERIES_SLOTS, SS, gpc, geo.V);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int P = w.slot, Y = P + SS, R = Y + SS, n = (int)link_rec(N);
  const double dv = (double)geo.V;
  for (int e = w.lane; e < 9 * N; e += glanes<G>()) {
    const double2 v = __ldg(Wg + (size_t)e * geo.V + w.id);
    sm[P + 1 + e] = make_double2(v.x / dv, v.y / dv);
  }
  gsync<G>();
  ser_reH<G>(P, N);
  wstore<G>(Gx + (size_t)w.id * n, ser_exp_to<G, false>(P, Y, R, N), n);
}

// U_mu(x) <- G(x) U_mu(x) G(x+mu)^dag  (nspt.cc:912-916), written to F.
constexpr int APPLY_SLOTS = 3;

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_fa_apply(const double2 *U, const double2 *Gx, double2 *F, int N, int SS, Geo geo,
               int gpc) {
  const Grp<G> w(APPLY_SLOTS, SS, gpc, 4L * geo.V);
  if (!w.ok) return;
  const int T = w.slot, Y = T + SS, H = Y + SS, n = (int)link_rec(N);
  const int site = (int)(w.id >> 2), mu = (int)(w.id & 3);
  int x[4];
  coords(geo, site, x);
  wstage<G>(T, Gx + (size_t)site * n, n);
  wstage<G>(Y, U + (size_t)w.id * n, n);
  wstage<G>(H, Gx + (size_t)neighbour(geo, x, mu, 1).site * n, n);
  wstage_wait<G>();
  ser_mul<G>(Y, T, Y, N, MUL_DAG);
  ser_mul<G>(Y, Y, H, N, MUL_DB);
  wstore<G>(F + (size_t)w.id * n, Y, n);
}

// ---------------- local stochastic gauge fixing ----------------

// One barrier step of stochastic_gauge_fixing (nspt.cc:660-862), in place:
// one group per reference thread, walking its segment site by site.  Sites
// of different threads are >= 2 apart and share no link, so the result is
// the reference's with the same thread grid.  Per site: W = sum_mu U_mu(x) -
// U_mu(x-mu) (twisted read across a twisted face), W -= W^dag, Trless,
// U_mu(x) <- exp(alpha W) U_mu(x), U_mu(x-mu) <- U_mu(x-mu) exp(-alpha W)
// (twist_mu(exp(-alpha W)) = Omega W2 Omega^dag when x-mu wraps a twisted
// face, nspt.cc:690-719).  alpha W is antihermitian, so exp(-alpha W) is the
// dagger of exp(alpha W): one exponential and daggered products.
constexpr int TEAM_WARPS = 8;

template <int G>
__host__ __device__ constexpr int lgf_slots() {
  return G == ORDERED ? 4 : 3;
}

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_local_gf(double2 *U, const double2 *Ut, int N, int SS, Geo geo, double alpha, LgfGrid gr,
               long step, int gpc) {
  const Grp<G> w(lgf_slots<G>(), SS, gpc, gr.nthr);
  if (!w.ok) return;
  double2 *sm = wsm();
  const int X = w.slot, Y = X + SS, E = Y + SS, n = (int)link_rec(N);
  const double D3 = 1.0 / 3.0;
  const LgfWalk walk(gr, w.id, step);
#pragma unroll 1
  for (long r = 0; r < gr.seg; r++) {
    int x[4];
    walk.site(gr, geo, r, x);
    const int site = x[0] * geo.s0 + x[1] * geo.s1 + x[2] * geo.s2 + x[3];
    // W = sum_mu U_mu(x) - U_mu(x-mu)  (nspt.cc:672-675)
#pragma unroll 1
    for (int mu = 0; mu < 4; mu++) {
      const Nb bn = neighbour(geo, x, mu, -1);
      const bool cross = (bn.bwd & geo.twist) != 0;
      wstage<G>(Y, U + link_at(mu, site, N), n);
      wstage<G>(E, (cross ? Ut : U) + link_at(mu, bn.site, N), n);
      wstage_wait<G>();
      twist_link<G>(E, bn, geo, N);
      for (int e = w.lane; e < n; e += glanes<G>())
        sm[X + e] = cadd(mu == 0 ? cz() : sm[X + e], csub(sm[Y + e], sm[E + e]));
      gsync<G>();
    }
    // X = alpha Trless(W - W^dag) (nspt.cc:679-682, QCDpt.cc:124-136, 185-194)
    for (int k = 1 + w.lane; k <= N; k += glanes<G>()) {
      double2 *p = sm + X + 9 * k - 8;
      double2 a[9], b[9];
#pragma unroll
      for (int e = 0; e < 9; e++) a[e] = p[e];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int q = 0; q < 3; q++) b[3 * i + q] = csub(a[3 * i + q], cconj(a[3 * q + i]));
      const double2 tr = cadd(cadd(b[0], b[4]), b[8]);
      const double2 z = make_double2(D3 * tr.x, D3 * tr.y);
      b[0] = csub(b[0], z);
      b[4] = csub(b[4], z);
      b[8] = csub(b[8], z);
#pragma unroll
      for (int e = 0; e < 9; e++) p[e] = cscale(b[e], alpha);
    }
    if (w.lane == 0) sm[X] = cz();
    gsync<G>();
    // P = exp(X), and M = exp(-X): P's dagger, or with ORDERED summed by itself
    int P = X, M = X;
    if constexpr (G == ORDERED) {
      P = E;
      M = E + SS;
      ser_exp_horner<G, true>(X, Y, P, N);
      ser_exp_horner<G, true>(X, Y, M, N, -1.0);
    } else {
      ser_exp<G, true>(X, Y, E, N);
    }
#pragma unroll 1
    for (int t = 0; t < 8; t++) {
      // even: U_mu(x) <- P U_mu(x); odd: U_mu(x-mu) <- U_mu(x-mu) M, twisted
      // across a twisted face
      const int mu = t >> 1;
      const bool fwd = !(t & 1);
      const int S = G == ORDERED ? X : E;  // a slot free now
      const Nb back = neighbour(geo, x, mu, -1);
      double2 *rec = U + link_at(mu, fwd ? site : back.site, N);
      wstage<G>(Y, rec, n);
      int R = M;
      if (!fwd && ((back.bwd & geo.twist) >> mu & 1u)) {
        for (int e = w.lane; e < n; e += glanes<G>()) sm[S + e] = sm[M + e];
        gsync<G>();
        wtwist<G>(S, 0u, 1u << mu, N);
        R = S;
      }
      wstage_wait<G>();
      ser_mul<G>(Y, fwd ? P : Y, fwd ? Y : R, N, fwd || G == ORDERED ? MUL_DAG : MUL_DB);
      wstore<G>(rec, Y, n);
      gsync<G>();
    }
    // the next site's copies read links written here
    __threadfence();
    gsync<G>();
  }
}

// The same by a team: a CTA per reference thread, for barrier steps with few
// threads, where the time is that of one site's chain.  The site's eight links
// are staged at once, by all groups of the CTA (task t < 4: U_t(x), t >= 4:
// U_{t-4}(x-mu)), the exponential is one group's (ORDERED: exp(alpha W) and
// exp(-alpha W) two groups'), and the eight products are dealt to the groups from
// the staged copies (no other thread writes those links between the barriers).
// Slots: the eight links, four twisted copies, X and the exponential's.
template <int G>
__host__ __device__ constexpr int team_slots() {
  return G == ORDERED ? 17 : 15;
}

template <int G>
__global__ void __launch_bounds__(32 * TEAM_WARPS, G == ORDERED ? 1 : 2)
    k_local_gf_team(double2 *U, const double2 *Ut, int N, int SS, Geo geo, double alpha,
                    LgfGrid gr, long step) {
  double2 *sm = wsm();
  const int g = (threadIdx.x & 31) / glanes<G>(), per = 32 / glanes<G>();
  const int workers = (blockDim.x >> 5) * per;
  const int me = g < per ? (threadIdx.x >> 5) * per + g : workers;  // workers: a lane without
  const int lane = glane<G>(), n = (int)link_rec(N), GS = group_stride(1, SS);
  const int S = LEAD, Tw = S + 8 * GS, X = Tw + 4 * GS, Y = X + GS, E = Y + GS;
  const double D3 = 1.0 / 3.0;
  const LgfWalk walk(gr, blockIdx.x, step);
#pragma unroll 1
  for (long r = 0; r < gr.seg; r++) {
    int x[4];
    walk.site(gr, geo, r, x);
    const int site = x[0] * geo.s0 + x[1] * geo.s1 + x[2] * geo.s2 + x[3];
    for (int t = me; t < 8; t += workers) {
      const int mu = t & 3;
      const Nb bn = neighbour(geo, x, mu, -1);
      wstage<G>(S + t * GS, U + link_at(mu, t < 4 ? site : bn.site, N), n);
      // a back link read across a twisted face, as the step's start field has it
      if (t >= 4 && Ut != U && (bn.bwd & geo.twist))
        wstage<G>(Tw + mu * GS, Ut + link_at(mu, bn.site, N), n);
    }
    cp_commit();
    cp_wait0();
    __syncthreads();
    // alpha Trless(W - W^dag), W = sum_mu U_mu(x) - U_mu(x-mu), a thread per order
    for (int k = 1 + threadIdx.x; k <= N; k += blockDim.x) {
      double2 w[9], b[9];
#pragma unroll
      for (int mu = 0; mu < 4; mu++) {
        const unsigned tb = neighbour(geo, x, mu, -1).bwd & geo.twist;
        const double2 *f = sm + S + mu * GS + 9 * k - 8;
        const double2 *q = sm + (tb && Ut != U ? Tw + mu * GS : S + (4 + mu) * GS) + 9 * k - 8;
        double2 m[9];
#pragma unroll
        for (int e = 0; e < 9; e++) m[e] = q[e];
        if (tb) twist3(m, tb, 0u);
#pragma unroll
        for (int e = 0; e < 9; e++) w[e] = cadd(mu == 0 ? cz() : w[e], csub(f[e], m[e]));
      }
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int q = 0; q < 3; q++) b[3 * i + q] = csub(w[3 * i + q], cconj(w[3 * q + i]));
      const double2 tr = cadd(cadd(b[0], b[4]), b[8]);
      const double2 z = make_double2(D3 * tr.x, D3 * tr.y);
      b[0] = csub(b[0], z);
      b[4] = csub(b[4], z);
      b[8] = csub(b[8], z);
      double2 *o = sm + X + 9 * k - 8;
#pragma unroll
      for (int e = 0; e < 9; e++) o[e] = cscale(b[e], alpha);
    }
    if (threadIdx.x == 0) sm[X] = cz();
    __syncthreads();
    int P = X, M = X;
    if constexpr (G == ORDERED) {
      P = E;
      M = E + 2 * GS;
      if (me == 0) ser_exp_horner<G, true>(X, Y, P, N);
      if (me == 1) ser_exp_horner<G, true>(X, E + GS, M, N, -1.0);
    } else {
      if (me == 0) ser_exp<G, true>(X, Y, E, N);
    }
    __syncthreads();
    for (int t = me; t < 8; t += workers) {
      const int mu = t & 3, A = S + t * GS;
      const bool fwd = t < 4;
      const Nb back = neighbour(geo, x, mu, -1);
      int R = M;
      if (!fwd && ((back.bwd & geo.twist) >> mu & 1u)) {
        R = Tw + mu * GS;
        for (int e = lane; e < n; e += glanes<G>()) sm[R + e] = sm[M + e];
        gsync<G>();
        wtwist<G>(R, 0u, 1u << mu, N);
      }
      ser_mul<G>(A, fwd ? P : A, fwd ? A : R, N, fwd || G == ORDERED ? MUL_DAG : MUL_DB);
      wstore<G>(U + link_at(mu, fwd ? site : back.site, N), A, n);
    }
    // the next site's copies read links written here
    __threadfence();
    __syncthreads();
  }
}

// ---------------- Fourier-accelerated gauge fixing ----------------

// Wg(x) = sum_mu [log U_mu(x) - log U_mu(x-mu)]  (nspt.cc:871-877), from
// records to planes: a CTA takes 32 sites and 32 entries at a time, reads each
// record's run of entries and writes each plane's run of sites through a
// shared tile.
__global__ void __launch_bounds__(256) k_fa_div(const double2 *__restrict__ Lg,
                                                double2 *__restrict__ Wg, int N, Geo geo) {
  __shared__ double2 tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int n9 = 9 * N;
  const size_t rec = link_rec(N), V = (size_t)geo.V;
  const int e = blockIdx.y * 32 + tx, s0 = blockIdx.x * 32;
  for (int q = ty; q < 32; q += 8) {
    const int site = s0 + q;
    double2 v = cz();
    if (site < geo.V && e < n9) {
      int x[4];
      coords(geo, site, x);
#pragma unroll
      for (int mu = 0; mu < 4; mu++) {
        const int b = neighbour(geo, x, mu, -1).site;
        v = cadd(v, csub(__ldg(Lg + ((size_t)site * 4 + mu) * rec + 1 + e),
                         __ldg(Lg + ((size_t)b * 4 + mu) * rec + 1 + e)));
      }
    }
    tile[q][tx] = v;
  }
  __syncthreads();
  for (int q = ty; q < 32; q += 8) {
    const int ee = blockIdx.y * 32 + q, site = s0 + tx;
    if (site < geo.V && ee < n9) Wg[(size_t)ee * V + site] = tile[tx][q];
  }
}

// Wg(p) *= -alpha / p2hat(p), Wg(0) = 0  (nspt.cc:881-894)
// p2: the context's lattice momenta p2hat[d][n] = 4 sin^2(pi n / L_d)
// (lattice.h:1144-1169), 128 entries per direction.
__global__ void k_fa_scale(double2 *Wg, int N, Geo geo, double alpha, const double *__restrict__ p2) {
  const size_t V = (size_t)geo.V;
  const size_t tot = (size_t)9 * N * V;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t e = i / V;
    const int site = (int)(i - e * V);
    double f = 0.0;
    if (site != 0) {
      int x[4];
      coords(geo, site, x);
      f = -(alpha / (p2[x[0]] + p2[128 + x[1]] + p2[256 + x[2]] + p2[384 + x[3]]));
    }
    Wg[i] = cscale(Wg[i], f);
  }
}

// One pass of a 4-D FFT: all lines along one direction (length n, site stride
// st) of every plane, one thread per line; unnormalised, sign -1 forward
// (FFTW_FORWARD) / +1 backward.  Power-of-two n: radix-2 in registers.
template <int n>
__global__ void k_fft_pow2(double2 *data, long nlines, int st, size_t V, int sign) {
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= nlines) return;
  const long per_plane = (long)V / n;
  const long p = id / per_plane, rem = id - p * per_plane;
  const long outer = rem / st, inner = rem - outer * st;
  double2 *b = data + (size_t)p * V + (size_t)outer * n * st + inner;
  double2 v[n];
#pragma unroll
  for (int i = 0; i < n; i++) {
    int r = 0;
#pragma unroll
    for (int q = 1, t = i; q < n; q <<= 1, t >>= 1) r = (r << 1) | (t & 1);
    v[r] = b[(size_t)i * st];
  }
#pragma unroll
  for (int len = 2; len <= n; len <<= 1) {
    const int half = len >> 1;
#pragma unroll
    for (int k = 0; k < half; k++) {
      double2 w = c_tw64[k * (64 / len)];
      if (sign > 0) w.y = -w.y;
#pragma unroll
      for (int s0 = 0; s0 < n; s0 += len) {
        const double2 bb = cmul(v[s0 + k + half], w);
        v[s0 + k + half] = csub(v[s0 + k], bb);
        v[s0 + k] = cadd(v[s0 + k], bb);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < n; i++) b[(size_t)i * st] = v[i];
}

// Direct DFT for other lengths (n <= 128), one thread per line.
__global__ void k_fft_direct(double2 *data, long nlines, int n, int st, size_t V, int sign) {
  const long id = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (id >= nlines) return;
  const long per_plane = (long)V / n;
  const long p = id / per_plane, rem = id - p * per_plane;
  const long outer = rem / st, inner = rem - outer * st;
  double2 *b = data + (size_t)p * V + (size_t)outer * n * st + inner;
  double2 in[128];
  for (int i = 0; i < n; i++) in[i] = b[(size_t)i * st];
  for (int k = 0; k < n; k++) {
    double2 acc = cz();
    for (int i = 0; i < n; i++) {
      const int m = (int)(((long)k * i) % n);
      double sn, cs;
      sincospi((double)sign * 2.0 * (double)m / (double)n, &sn, &cs);
      acc = cadd(acc, cmul(in[i], make_double2(cs, sn)));
    }
    b[(size_t)k * st] = acc;
  }
}

// Column sums of a matrix of `rows` rows of `width` doubles, rows in a fixed
// order: block (i, j) sums the j-th chunk of rows of columns 32 i .. 32 i + 31
// into out[j][width].  Launched twice, the second time over the chunks.
__global__ void __launch_bounds__(256)
    k_colsum(const double *__restrict__ in, long rows, int width, long chunk, double *out) {
  __shared__ double sh[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  const long r0 = blockIdx.y * chunk, r1 = r0 + chunk < rows ? r0 + chunk : rows;
  double s = 0.0;
  if (c < width)
    for (long r = r0 + ty; r < r1; r += 8) s += in[(size_t)r * width + c];
  sh[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < width) {
    for (int q = 1; q < 8; q++) s += sh[q][tx];
    out[(size_t)blockIdx.y * width + c] = s;
  }
}

// ---------------- float-float scale exponent ----------------

// mx[k-1] = max over the field's order-k entries of max(|re|, |im|), as the
// bit pattern of a non-negative double (ordered like the value); one row of
// blocks per order (blockIdx.y), mx zeroed by the caller
__global__ void k_order_absmax(const double2 *__restrict__ U, int N, size_t V,
                               unsigned long long *mx) {
  const int k = blockIdx.y + 1;
  const size_t per = 36 * V;  // entries of one order
  double m = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < per;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t l = i / 9;
    const double2 v = __ldg(U + l * link_rec(N) + 1 + 9 * (size_t)(k - 1) + (i - 9 * l));
    m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0 && m > 0.0)
    atomicMax(mx + (k - 1), (unsigned long long)__double_as_longlong(m));
}

// Per-order scale exponent: order k is multiplied by 2^(e k) before its
// float-float split.  e = -(slope of log2 max|U_k| over k), a least-squares
// fit over the orders that are non-zero, so that the scaled orders keep one
// common size whatever their geometric growth or decay; |e| N <= 1000.
__global__ void k_ff_fit(const unsigned long long *mx, int N, int *e_out) {
  double sk = 0, sl = 0, skk = 0, skl = 0;
  int n = 0;
  for (int k = 1; k <= N; k++) {
    const double m = __longlong_as_double((long long)mx[k - 1]);
    if (m > 0.0) {
      const double l = (double)ilogb(m);
      sk += k;
      sl += l;
      skk += (double)k * k;
      skl += k * l;
      n++;
    }
  }
  int e = 0;
  if (n >= 2) {
    const double slope = (n * skl - sk * sl) / (n * skk - sk * sk);
    e = (int)rint(-slope);
  }
  const int lim = 1000 / (N > 0 ? N : 1);
  *e_out = max(-lim, min(lim, e));
}

// Host field chunk (sites [s0, s0+cs), the reference's layout with A >= N
// orders per link) <-> device records; with A = N the two are one copy.
__global__ void k_unpack(const double2 *__restrict__ aos, int A, int s0, int cs, double2 *U,
                         int N) {
  const size_t rec = link_rec(N), ser = 1 + 9 * (size_t)A, tot = (size_t)cs * 4 * rec;
  double2 *dst = U + (size_t)s0 * 4 * rec;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t l = i / rec;
    dst[i] = aos[l * ser + (i - l * rec)];
  }
}
__global__ void k_pack(double2 *__restrict__ aos, int A, int s0, int cs, const double2 *U, int N) {
  const size_t rec = link_rec(N), ser = 1 + 9 * (size_t)A, tot = (size_t)cs * 4 * ser;
  const double2 *src = U + (size_t)s0 * 4 * rec;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t l = i / ser, e = i - l * ser;
    aos[i] = e < rec ? src[l * rec + e] : cz();
  }
}

// *other = 1 where a link's flag is not 1
__global__ void k_other_flags(const double2 *__restrict__ U, size_t nlinks, int N, int *other) {
  bool any = false;
  for (size_t l = blockIdx.x * (size_t)blockDim.x + threadIdx.x; l < nlinks;
       l += (size_t)gridDim.x * blockDim.x) {
    const double2 f = U[l * link_rec(N)];
    any |= !(f.x == 1.0 && f.y == 0.0);
  }
  if (any) *other = 1;
}

__global__ void k_cold(double2 *U, size_t nlinks, int N) {
  const size_t rec = link_rec(N), tot = nlinks * rec;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot;
       i += (size_t)gridDim.x * blockDim.x)
    U[i] = i % rec ? cz() : make_double2(1.0, 0.0);
}

// FP64 FMA throughput probe: 8 independent chains per thread.
__global__ void k_fp64_peak(double *out, int iters, double seed) {
  double a[8];
#pragma unroll
  for (int q = 0; q < 8; q++) a[q] = seed + q + threadIdx.x * 1e-9;
  const double m = 0.999999999, ad = 1e-12;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int u = 0; u < 16; u++)
#pragma unroll
      for (int q = 0; q < 8; q++) a[q] = fma(a[q], m, ad);
  }
  double s = 0;
#pragma unroll
  for (int q = 0; q < 8; q++) s += a[q];
  if (s == 12345.678) out[0] = s;  // keeps the chains live
}

}  // namespace nspt
