// Wilson loops of ComputeLoops (nspt.cc:1148-1312): 1x2 (both
// orientations), 2x2, 2x4 (both) and 4x4 loops in every plane mu < nu,
// summed over the lattice and traced, per order.  Periodic boundaries, as
// the reference computes them only there (__MANY_LOOP__ under PERIODIC_BC).
//
// One group per (plane, site).  The reference closes each loop with a
// product by a daggered path, W += P Q^dag; only Tr W is printed, so the last
// product is replaced by Tr(P Q^dag) = sum over cells of P_ij conj(Q_ij),
// order by order.  Four slots per group (three paths and a staging slot) and
// the group's four trace accumulators; CTAs sum their groups, and a last
// kernel their rows, in a fixed order.
#pragma once

namespace nspt {

constexpr int LOOP_SLOTS = 4, LOOP_EXTRA = 1;  // 1 + 9 N >= 4 (N + 1) for the accumulators (N = 1: 10)

// acc[k] += Tr(X Y^dag)_k, k = 0..N, a lane per order
template <int G>
__device__ __forceinline__ void trace_dag_acc(int X, int Y, int N, int acc) {
  double2 *sm = wsm();
  for (int k = glane<G>(); k <= N; k += glanes<G>()) sm[acc + k] = cadd(sm[acc + k], trace_dag(X, Y, k));
  gsync<G>();
}

struct LoopCtx {
  const double2 *U, *D;  // links, and two-link lines D_mu(x) = U_mu(x) U_mu(x+mu)
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

// Begin the copy of a link (len 1) or two-link line (len 2) along mu (dir 0) or
// nu (1) from x + i mu + j nu
template <int G>
__device__ __forceinline__ void loop_stage(const LoopCtx &q, int slot, int len, int dir, int i,
                                           int j) {
  wstage<G>(slot, (len == 2 ? q.D : q.U) + link_at(dir ? q.nu : q.mu, loop_site(q, i, j), q.N),
            (int)link_rec(q.N));
}

// The two-link lines of every link, which the loops are made of
template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_lines(const double2 *U, double2 *D, int N, int SS, Geo geo, int gpc) {
  const Grp<G> w(2, SS, gpc, 4L * geo.V);
  if (!w.ok) return;
  const int A = w.slot, S = A + SS, n = (int)link_rec(N);
  const int site = (int)(w.id >> 2), mu = (int)(w.id & 3);
  int x[4];
  coords(geo, site, x);
  wstage<G>(A, U + (size_t)w.id * n, n);
  wstage<G>(S, U + link_at(mu, neighbour(geo, x, mu, 1).site, N), n);
  wstage_wait<G>();
  ser_mul<G>(A, A, S, N);
  wstore<G>(D + (size_t)w.id * n, A, n);
}

// Per (plane, site), the loops of ComputeLoops (nspt.cc:1160-1270) as pairs of
// paths P, Q from x to the opposite corner, traced as Tr(P Q^dag).  m, n: two-link
// lines along mu, nu; u: single links.
//   2x2        P = m n        Q = n m
//   2x4 up     P = m n n      R = n n m
//   2x4 right  P = m m n      Q = n m m
//   4x4        P = m m n n    R = n n m m
//   1x2        P = m u        Q = u m
//   1x2        P = u n        Q = n u
// A path that begins with another's is extended in place: 14 products and 6
// traces per (plane, site), and a line per link before (0.7 per plane and site),
// where chains of single links took 40.
constexpr int LOOP_STEPS = 28;
struct LoopStep {
  // slot: 0 P, 1 Q, 2 R; op: 0 begin the slot with the piece, 1 multiply it by the
  // piece, 2 trace of P and the slot into row len
  signed char slot, op, len, dir, i, j;
};
__constant__ LoopStep c_loop[LOOP_STEPS] = {
    {0, 0, 2, 0, 0, 0}, {0, 1, 2, 1, 2, 0}, {1, 0, 2, 1, 0, 0}, {1, 1, 2, 0, 0, 2}, {1, 2, 1},
    {0, 1, 2, 1, 2, 2}, {2, 0, 2, 1, 0, 0}, {2, 1, 2, 1, 0, 2}, {2, 1, 2, 0, 0, 4}, {2, 2, 2},
    {2, 1, 2, 0, 2, 4}, {1, 1, 2, 0, 2, 2}, {0, 0, 2, 0, 0, 0}, {0, 1, 2, 0, 2, 0},
    {0, 1, 2, 1, 4, 0}, {1, 2, 2},          {0, 1, 2, 1, 4, 2}, {2, 2, 3},
    {0, 0, 2, 0, 0, 0}, {0, 1, 1, 1, 2, 0}, {1, 0, 1, 1, 0, 0}, {1, 1, 2, 0, 0, 1}, {1, 2, 0},
    {0, 0, 1, 0, 0, 0}, {0, 1, 2, 1, 1, 0}, {1, 0, 2, 1, 0, 0}, {1, 1, 1, 0, 0, 2}, {1, 2, 0}};

template <int G>
__global__ void __launch_bounds__(32 * CTA_WARPS, sm_ctas<G>())
    k_loops(const double2 *U, const double2 *D, int N, int SS, Geo geo, double2 *partial, int gpc) {
  double2 *sm = wsm();
  const int row = 4 * (N + 1);
  const long units = 6L * geo.V;
  // the accumulators follow the slots, in a stretch of LOOP_EXTRA slots
  const Grp<G> w(LOOP_SLOTS + LOOP_EXTRA, SS, gpc, units);
  const int S = w.slot + 3 * SS, acc = S + SS;
  if (w.ok) {
    for (int e = w.lane; e < row; e += glanes<G>()) sm[acc + e] = cz();
    gsync<G>();
    LoopCtx q;
    q.U = U;
    q.D = D;
    q.N = N;
    q.geo = geo;
#pragma unroll 1
    for (long u = w.id; u < units; u += (long)gridDim.x * gpc) {
      const int pl = (int)(u / geo.V);
      plane_dirs(pl, q.mu, q.nu);
      coords(geo, (int)(u - (long)pl * geo.V), q.X);
#pragma unroll 1
      for (int h = 0; h < LOOP_STEPS; h++) {
        const LoopStep t = c_loop[h];
        const int A = w.slot + t.slot * SS;
        if (t.op == 2) {
          trace_dag_acc<G>(w.slot, A, N, acc + t.len * (N + 1));
        } else {
          loop_stage<G>(q, t.op ? S : A, t.len, t.dir, t.i, t.j);
          if (t.op) {  // the path's first piece is waited for with the second
            wstage_wait<G>();
            ser_mul<G>(A, A, S, N);
          }
        }
      }
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
