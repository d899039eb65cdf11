// Wilson loops of ComputeLoops (nspt.cc:1148-1312): 1x2 (both
// orientations), 2x2, 2x4 (both) and 4x4 loops in every plane mu < nu,
// summed over the lattice and traced, per order.  Periodic boundaries, as
// the reference computes them only there (__MANY_LOOP__ under PERIODIC_BC).
//
// One group per (plane, site).  The reference closes each loop with a
// product by a daggered path, W += P Q^dag; only Tr W is printed, so the last
// product is replaced by Tr(P Q^dag) = sum over cells of P_ij conj(Q_ij),
// order by order.  Three slots per group (two paths and a staging slot) and
// the group's four trace accumulators; CTAs sum their groups, and a last
// kernel their rows, in a fixed order.
#pragma once

namespace nspt {

constexpr int LOOP_SLOTS = 3, LOOP_EXTRA = 1;  // 1 + 9 N >= 4 (N + 1) for the accumulators (N = 1: 10)

// acc[k] += Tr(X Y^dag)_k, k = 0..N, a lane per order
template <int G>
__device__ __forceinline__ void trace_dag_acc(int X, int Y, int N, int acc) {
  double2 *sm = wsm();
  for (int k = glane<G>(); k <= N; k += glanes<G>()) sm[acc + k] = cadd(sm[acc + k], trace_dag(X, Y, k));
  gsync<G>();
}

// A path of the loops: a chain of n forward links, link m in direction
// (dirs >> m) & 1 (0: mu, 1: nu) at the site reached by the links before it.
struct LoopPath {
  int n;
  unsigned dirs;
};

struct LoopCtx {
  const double2 *U;
  int N, mu, nu;
  int X[4];
  Geo geo;
};

// site X + i mu + j nu (periodic)
__device__ __forceinline__ int loop_site(const LoopCtx &q, int i, int j) {
  int y[4];
#pragma unroll
  for (int d = 0; d < 4; d++)
    y[d] = (q.X[d] + (d == q.mu ? i : 0) + (d == q.nu ? j : 0)) % q.geo.L[d];
  return y[0] * q.geo.s0 + y[1] * q.geo.s1 + y[2] * q.geo.s2 + y[3];
}

// A <- path[from..n) applied to A (from = 0: A is formed from the first
// link); (i, j) is the site where link `from` starts, updated to the end
template <int G>
__device__ __forceinline__ void loop_chain(const LoopCtx &q, int A, int S, const LoopPath &p,
                                           int from, int &i, int &j) {
#pragma unroll 1
  for (int m = from; m < p.n; m++) {
    wstage<G>(m == 0 ? A : S, q.U + link_at((p.dirs >> m & 1) ? q.nu : q.mu, loop_site(q, i, j), q.N),
           (int)link_rec(q.N));
    if (m > 0) {  // the first link is waited for with the second
      wstage_wait<G>();
      ser_mul<G>(A, A, S, q.N);
    }
    if (p.dirs >> m & 1) j++; else i++;
  }
}

// Per (plane, site), the loops of ComputeLoops as pairs of paths P, Q from
// x, traced as Tr(P Q^dag) (bl = mu mu from x, ld = nu nu from x, cd the
// two nu links after bl, and so on, as named in nspt.cc:1160-1270):
//   2x2        P = bl cd           Q = ld ml
//   2x4 up     P = bl cd cu        Q = ld lu tl
//   4x4        P = bl br rd ru     Q = ld lu tl tr
//   2x4 right  P = bl br rd        Q = ld ml mr
//   1x2        P = bl U_nu         Q = U_nu U_mu U_mu
//   1x2        P = U_mu U_nu U_nu  Q = ld U_mu
// Three slots per group: P and Q (paths, each extended in place link by
// link) and S (the staged link).  A path is extended when the next loop's
// path starts with it (bl cd -> bl cd cu, ld lu tl -> ld lu tl tr) and
// formed afresh otherwise: 40 products and 6 traces per (plane, site).
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_loops(const double2 *U, int N, int SS, Geo geo, double2 *partial, int gpc) {
  double2 *sm = wsm();
  const int row = 4 * (N + 1);
  const long units = 6L * geo.V;
  // the accumulators follow the three slots, in a stretch of LOOP_EXTRA slots
  const Grp<G> w(LOOP_SLOTS + LOOP_EXTRA, SS, gpc, units);
  const int P = w.slot, Q = P + SS, S = Q + SS, acc = S + SS;
  if (w.ok) {
    for (int e = w.lane; e < row; e += glanes<G>()) sm[acc + e] = cz();
    gsync<G>();
    const int a21 = acc, a22 = acc + (N + 1), a42 = acc + 2 * (N + 1), a44 = acc + 3 * (N + 1);
    LoopCtx q;
    q.U = U;
    q.N = N;
    q.geo = geo;
    const LoopPath p22{4, 0xcu}, q22{4, 0x3u};
    const LoopPath p42u{6, 0x3cu}, q42u{6, 0xfu};
    const LoopPath p44{8, 0xf0u}, q44{8, 0xfu};
    const LoopPath p42r{6, 0x30u}, q42r{6, 0x3u};
    const LoopPath p21a{3, 0x4u}, q21a{3, 0x1u};
    const LoopPath p21b{3, 0x6u}, q21b{3, 0x3u};
    const long stride = (long)gridDim.x * gpc;
#pragma unroll 1
    for (long u = w.id; u < units; u += stride) {
      const int pl = (int)(u / geo.V);
      const int x = (int)(u - (long)pl * geo.V);
      q.mu = pl < 3 ? 0 : (pl < 5 ? 1 : 2);
      q.nu = pl < 3 ? pl + 1 : (pl < 5 ? pl - 1 : 3);
      coords(geo, x, q.X);
      int pi = 0, pj = 0, qi = 0, qj = 0;
      // 2x2
      loop_chain<G>(q, P, S, p22, 0, pi, pj);
      loop_chain<G>(q, Q, S, q22, 0, qi, qj);
      trace_dag_acc<G>(P, Q, N, a22);
      // 2x4 up: P = bl cd extended by cu
      loop_chain<G>(q, P, S, p42u, 4, pi, pj);
      qi = qj = 0;
      loop_chain<G>(q, Q, S, q42u, 0, qi, qj);
      trace_dag_acc<G>(P, Q, N, a42);
      // 4x4: Q = ld lu tl extended by tr
      loop_chain<G>(q, Q, S, q44, 6, qi, qj);
      pi = pj = 0;
      loop_chain<G>(q, P, S, p44, 0, pi, pj);
      trace_dag_acc<G>(P, Q, N, a44);
      // 2x4 right
      pi = pj = qi = qj = 0;
      loop_chain<G>(q, P, S, p42r, 0, pi, pj);
      loop_chain<G>(q, Q, S, q42r, 0, qi, qj);
      trace_dag_acc<G>(P, Q, N, a42);
      // 1x2, both orientations
      pi = pj = qi = qj = 0;
      loop_chain<G>(q, P, S, p21a, 0, pi, pj);
      loop_chain<G>(q, Q, S, q21a, 0, qi, qj);
      trace_dag_acc<G>(P, Q, N, a21);
      pi = pj = qi = qj = 0;
      loop_chain<G>(q, P, S, p21b, 0, pi, pj);
      loop_chain<G>(q, Q, S, q21b, 0, qi, qj);
      trace_dag_acc<G>(P, Q, N, a21);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < row; e += blockDim.x) {
    double2 sum = cz();
    const int gs = group_stride(LOOP_SLOTS + LOOP_EXTRA, SS);
    for (int g = 0; g < gpc && (long)blockIdx.x * gpc + g < units; g++)
      sum = cadd(sum, sm[LEAD + g * gs + LOOP_SLOTS * SS + e]);
    partial[(size_t)blockIdx.x * row + e] = sum;
  }
}

// out[e] = sum over rows of partial[row][e], rows in order
__global__ void k_rows_sum(const double2 *partial, int nrows, int width, double2 *out) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < width; e += gridDim.x * blockDim.x) {
    double2 s = cz();
    for (int r = 0; r < nrows; r++) s = cadd(s, partial[(size_t)r * width + e]);
    out[e] = s;
  }
}

}  // namespace nspt
