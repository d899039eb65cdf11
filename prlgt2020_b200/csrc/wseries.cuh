// wseries.cuh -- truncated power series of 3x3 complex matrices (the
// reference's ptSU3, QCDpt.h:42-226) by groups of lanes, FP64.
//
// A series in shared memory ("slot") has the layout of a link record: the flag
// (order-0 coefficient times the identity), then order k = 1..N, 9 complex
// numbers, row major.  Slots are named by their offset in double2 from the
// start of dynamic shared memory, so that every access is a shared-memory
// instruction also in the functions kept out of line.
//
// The Cauchy product C_k = sum_i A_i B_{k-i} is nine entries of three scalar
// convolutions A[r,l] * B[l,c] each.  A lane makes BLK orders of a convolution at
// a time, with BLK accumulators and a window of BLK right coefficients in
// registers: a step of i loads one left and one right coefficient and feeds BLK
// complex multiply-adds, and no branch depends on the lane.  (The form before, a
// lane per column and order class, had a branch per 3x3 block: 11.5 TFLOP/s
// useful alone at 24 orders of 36.5.)  Two forms:
//   G = 9:  three links per warp; lane 3r + c of a group does the three
//           convolutions of its entry one after another.  Nothing is left to add
//           up between lanes and three links share every instruction.
//   G = 32: one link per warp; 27 lanes (r, c, l) do one convolution each and add
//           up in threes.  430 of 2400 instructions of a product (24 orders) go
//           into that, but a link has three times the warps: the form where few
//           links are at hand, because shared memory holds no more of them (high
//           orders) or the launch has no more.
//
//   G = ORDERED: as G = 9, but all three convolutions of an entry advance together,
//           term by term in the order i, l (three windows, 200 to 255 registers).  The
//           sums are then bit for bit those of a plain loop over i of 3x3
//           products, which every field of a run with logarithms at high order
//           has been made with: there rounding is amplified by some 3 per order
//           (order 20 of a field of size 1: 1e-16 becomes 3e-7), so that a
//           different order of summation is another field.
//
// Groups are 4 (mod 8) 16-byte words apart: a quarter-warp, the unit a 128-bit
// shared load is served in, then finds its words on distinct banks whether an
// operand is read along rows or along columns.
//
// Each convolution is summed in ascending i.  Blocks of orders run from high to low and
// a block is read before it is written: a product may overwrite either operand.
#pragma once
#include <type_traits>

#include "series.cuh"

namespace nspt {

constexpr int CTA_WARPS = 4;   // one per scheduler
constexpr int BLK = 8;         // orders a product accumulates at a time
constexpr int LEAD = 9;        // the products read (and do not use) the words of order 0 before
                               // a slot, so the first slot starts here

__device__ __forceinline__ double2 *wsm() {
  extern __shared__ double2 sm[];
  return sm;
}

// the forms G of a group (see above) and its lanes
constexpr int ORDERED = 10;
template <int G>
__host__ __device__ constexpr int glanes() {
  return G == 32 ? 32 : 9;
}
// CTAs on an SM: 128 registers a thread, 256 for three windows
template <int G>
__host__ __device__ constexpr int sm_ctas() {
  return G == ORDERED ? 2 : 4;
}

// lane of the group, the group's first lane in the warp, its lanes, and a barrier
// of the group
template <int G>
__device__ __forceinline__ int glane() {
  return G == 32 ? threadIdx.x & 31 : (threadIdx.x & 31) % 9;
}
template <int G>
__device__ __forceinline__ int gfirst() {
  return G == 32 ? 0 : (threadIdx.x & 31) / 9 * 9;
}
template <int G>
__device__ __forceinline__ unsigned gmask() {
  return G == 32 ? 0xffffffffu : 511u << gfirst<G>();
}
template <int G>
__device__ __forceinline__ void gsync() {
  __syncwarp(gmask<G>());
}

// The lane's entry (r, c) and, G = 32, term l: lanes 8 r + m, m < 8, are (r, c, l) with m = 3 c + l; the ninth, m = 8, of
// row r is lane 24 + r.  A quarter-warp (the unit a 128-bit load is served in)
// then reads 3 or 8 consecutive 16-byte words: no two share a bank.
template <int G>
struct WLane {
  int lane, r, c;
  static constexpr int l = 0;
  __device__ __forceinline__ WLane() {
    lane = glane<G>();
    r = lane / 3;
    c = lane - 3 * r;
  }
};
template <>
struct WLane<32> {
  int lane, r, c, l;
  __device__ __forceinline__ WLane() {
    lane = threadIdx.x & 31;
    const int m = lane < 24 ? (lane & 7) : 8;
    r = lane < 24 ? (lane >> 3) : min(lane - 24, 2);
    c = m / 3;
    l = m - 3 * c;
  }
  // lane of (r, c, q)
  __device__ __forceinline__ int mate(int q) const {
    const int m = 3 * c + q;
    return m < 8 ? 8 * r + m : 24 + r;
  }
};

__device__ __forceinline__ double2 wshfl(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ double2 wsel3(int l, double2 a, double2 b, double2 c) {
  return make_double2(l == 0 ? a.x : l == 1 ? b.x : c.x, l == 0 ? a.y : l == 1 ? b.y : c.y);
}

// v, or its conjugate when sg = 0x80000000
__device__ __forceinline__ double2 wconj(double2 v, int sg) {
  return make_double2(v.x, __hiloint2double(__double2hiint(v.y) ^ sg, __double2loint(v.y)));
}

// FP64 arithmetic of the product
struct Acc64 {
  typedef double2 T;
  static __device__ __forceinline__ T zero() { return cz(); }
  static __device__ __forceinline__ T in(double2 v, int, int) { return v; }
  static __device__ __forceinline__ void mac(T &c, const T &a, const T &b) { cfma(c, a, b); }
  static __device__ __forceinline__ double2 out(const T &c, int, int) { return c; }
};
// compensated float-float arithmetic (series.cuh): order k scaled by 2^(e k)
struct AccFF {
  typedef ffc T;
  static __device__ __forceinline__ T zero() { return {0.f, 0.f, 0.f, 0.f}; }
  static __device__ __forceinline__ T in(double2 v, int e, int k) {
    return ff_split(v, pow2i(e * k));
  }
  static __device__ __forceinline__ void mac(T &c, const T &a, const T &b) { ff_cmac(c, a, b); }
  static __device__ __forceinline__ double2 out(const T &c, int e, int k) {
    const double s = pow2i(-e * k);
    return make_double2(((double)c.rh + (double)c.rl) * s, ((double)c.ih + (double)c.il) * s);
  }
};

// Modes of ser_mul
constexpr unsigned MUL_DA = 1;   // dagger of A
constexpr unsigned MUL_DB = 2;   // dagger of B
constexpr unsigned MUL_ACC = 4;  // out += A B instead of out = A B
constexpr unsigned MUL_A0 = 8;   // A's flag taken as 0
constexpr unsigned MUL_B0 = 16;  // B's flag taken as 0
constexpr unsigned MUL_MIX = 64;  // sum of two scalar series times matrix series: out = a_0 B + a_1
                                  // B2, a_l the entry l of A's records, B2 = B + aux, flags 0
constexpr unsigned MUL_DAG = 32;  // no dagger, but the copy of the code that takes them: for
                                  // kernels that hold it anyway (instruction cache)

// G = ORDERED: one block's sums of ser_mul_any, the terms in the order i, l.
// left / right: the lane's operands at order 0, entries la / lb apart.
template <class Acc>
__device__ __forceinline__ void ordered_block(typename Acc::T (&acc)[BLK], const double2 *left,
                                              int la, const double2 *right, int lb, int lend,
                                              int sa, int sb, int kb, int N, int aux) {
  typedef typename Acc::T T;
  T w[3][BLK];
  const int j0 = kb > 0 ? kb : 0;
#pragma unroll
  for (int l = 0; l < 3; l++)
#pragma unroll
    for (int q = 0; q < BLK; q++) {
      w[l][q] = Acc::zero();
      if (l < lend && j0 + q >= 1 && j0 + q < N)
        w[l][q] = Acc::in(wconj(right[9 * (j0 + q) + lb * l], sb), aux, j0 + q);
    }
  int i = 1;
  auto steps = [&](auto UU) {
    constexpr int U = decltype(UU)::value;
    T v[3][U + 1];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int l = 0; l < 3; l++) {
        const T a = Acc::in(wconj(left[9 * (i + u) + la * l], sa), aux, i + u);
        v[l][u + 1] = Acc::in(wconj(right[9 * (kb - i - u) + lb * l], sb), aux, kb - i - u);
#pragma unroll
        for (int q = 0; q < BLK; q++)
          Acc::mac(acc[q], a, q >= u ? w[l][q >= u ? q - u : 0] : v[l][q >= u ? 1 : u - q]);
      }
#pragma unroll
    for (int l = 0; l < 3; l++)
#pragma unroll
      for (int q = BLK - 1; q >= 0; q--)
        w[l][q] = q >= U ? w[l][q >= U ? q - U : 0] : v[l][q >= U ? 1 : U - q];
    i += U;
  };
  if (kb > 0 && kb % 2) steps(std::integral_constant<int, 1>());
#pragma unroll 1
  while (i <= kb) steps(std::integral_constant<int, 2>());
#pragma unroll
  for (int t = 0; t < BLK - 1; t++)
#pragma unroll
    for (int l = 0; l < 3; l++) {
      if (kb + t < 0) continue;
      const T a = Acc::in(wconj(left[9 * (kb + 1 + t) + la * l], sa), aux, kb + 1 + t);
#pragma unroll
      for (int q = t + 1; q < BLK; q++) Acc::mac(acc[q], a, w[l][q - t]);
    }
}

// out (a slot, or gout in global memory) <- op(A) op(B) + cx X (X: a slot, or
// -1 for no such term; out's flag is the caller's then unless X is out).  out
// may be any of the operands.  Out of line, a copy without daggers and one that
// takes either (a sign flip per operand loaded); a kernel uses one of them, since
// the SM's instruction cache holds no more (with three copies the GPC's was 73 %
// busy refilling it and a product took half as long again).  aux: MUL_MIX, or AccFF's scale.
template <class Acc, int G, bool DAG>
__device__ __noinline__ void ser_mul_any(int out, int A, int Bs, int N, unsigned mode, int aux,
                                         int X, double cx, double2 *gout) {
  typedef typename Acc::T T;
  constexpr int R = G == 32 ? (BLK + 2) / 3 : BLK;  // orders a lane finishes per block
  double2 *sm = wsm();
  const WLane<G> L;
  const bool da = DAG && (mode & MUL_DA), db = DAG && (mode & MUL_DB);
  const int sa = da ? (int)0x80000000 : 0, sb = db ? (int)0x80000000 : 0;
  const double2 a0 = mode & MUL_A0 ? cz() : wconj(sm[A], sa);
  const double2 b0 = mode & MUL_B0 ? cz() : wconj(sm[Bs], sb);
  const bool one = a0.x == 1.0 && a0.y == 0.0 && b0.x == 1.0 && b0.y == 0.0;
  const bool none = cis0(a0) && cis0(b0);
  // order k, entry l of this lane's operands at pa + 9 k + la l, pb + 9 k + lb l
  const bool mix = mode & MUL_MIX;
  const int pa = A - 8 + (mix ? 0 : da ? L.r : 3 * L.r), la = da ? 3 : 1;
  const int pb = Bs - 8 + (mix ? 3 * L.r + L.c : db ? 3 * L.c : L.c), lb = mix ? aux : db ? 1 : 3;
  const int lend = min(G == 32 ? L.l + 1 : 3, mix ? 2 : 3);
#pragma unroll 1
  for (int kb = N - BLK; kb > -BLK; kb -= BLK) {
    // outputs kb + 1 + q, q < BLK; w[q] = B_{kb + 1 + q - i} at step i
    T acc[BLK];
#pragma unroll
    for (int q = 0; q < BLK; q++) acc[q] = Acc::zero();
    if constexpr (G == ORDERED) {
      ordered_block<Acc>(acc, sm + pa, la, sm + pb, lb, lend, sa, sb, kb, N, aux);
    } else {
#pragma unroll 1
      for (int l = L.l; l < lend; l++) {
        T w[BLK];
        const double2 *pl = sm + pa + la * l, *pr = sm + pb + lb * l;  // at order 0
        if (kb > 0) {
          const double2 *p = pr + 9 * kb;
#pragma unroll
          for (int q = 0; q < BLK; q++) w[q] = Acc::in(wconj(p[9 * q], sb), aux, kb + q);
          int n = kb, i = 1;
          const double2 *pi = pl + 9;
          auto steps = [&](auto UU) {
            constexpr int U = decltype(UU)::value;
            T v[U + 1];
#pragma unroll
            for (int u = 0; u < U; u++) {
              const T a = Acc::in(wconj(pi[9 * u], sa), aux, i + u);
              // needed from the next step on; after the last step of all this is
              // order 0, in bounds (the words before the slot) and not used
              v[u + 1] = Acc::in(wconj(p[-9 * (u + 1)], sb), aux, kb - i - u);
#pragma unroll
              for (int q = 0; q < BLK; q++)
                Acc::mac(acc[q], a, q >= u ? w[q >= u ? q - u : 0] : v[q >= u ? 1 : u - q]);
            }
#pragma unroll
            for (int q = BLK - 1; q >= 0; q--)
              w[q] = q >= U ? w[q >= U ? q - U : 0] : v[q >= U ? 1 : U - q];
            pi += 9 * U;
            p -= 9 * U;
            n -= U;
            i += U;
          };
          // by twos: a longer body has fewer moves of the window, but the SM's
          // instruction cache pays for it.  12^4 N=12 sweep 2.09 ms by twos, 2.25 by
          // fours, 2.09 by ones; 16*16*16*8 N=24 8.39, 8.45 and 8.69
          if (n & 1) steps(std::integral_constant<int, 1>());
#pragma unroll 1
          while (n) steps(std::integral_constant<int, 2>());
        } else {  // the last block has the triangle only, which starts at w[1] = B_1
          w[0] = Acc::zero();
#pragma unroll
          for (int q = 1; q < BLK; q++) {
            w[q] = Acc::zero();
            if (q < N) w[q] = Acc::in(wconj(pr[9 * q], sb), aux, q);
          }
        }
        // the triangle: step i = kb + 1 + t reaches the outputs q > t; a left
        // order below 1 (a last block that sticks out) has no row
        auto triangle = [&](auto whole) {
#pragma unroll
          for (int t = 0; t < BLK - 1; t++) {
            if (!decltype(whole)::value && kb + t < 0) continue;
            const T a = Acc::in(wconj(pl[9 * (kb + 1 + t)], sa), aux, kb + 1 + t);
#pragma unroll
            for (int q = t + 1; q < BLK; q++) Acc::mac(acc[q], a, w[q - t]);
          }
        };
        if (kb >= 0)
          triangle(std::true_type());
        else
          triangle(std::false_type());
      }
    }
    // the orders this lane finishes, k0 .. k0 + m - 1: G = 9 all of the block,
    // G = 32 lane l of an entry a third of it, with its mates' sums
    double2 res[R];
    int k0 = kb + 1, m = BLK;
    if constexpr (G == 32) {
      const int from_next = L.mate(L.l == 2 ? 0 : L.l + 1);
      const int from_prev = L.mate(L.l == 0 ? 2 : L.l - 1);
#pragma unroll
      for (int h = 0; h < R; h++) {
        double2 x[3];
#pragma unroll
        for (int u = 0; u < 3; u++)
          x[u] = h + R * u < BLK
                     ? Acc::out(acc[h + R * u < BLK ? h + R * u : 0], aux, kb + 1 + h + R * u)
                     : cz();
        const double2 v = cadd(wsel3(L.l, x[0], x[1], x[2]),
                               wshfl(wsel3(L.l, x[1], x[2], x[0]), from_prev));
        res[h] = cadd(v, wshfl(wsel3(L.l, x[2], x[0], x[1]), from_next));
      }
      k0 += R * L.l;
      m = L.l == 2 ? BLK - 2 * R : R;
    } else {
#pragma unroll
      for (int h = 0; h < R; h++) res[h] = Acc::out(acc[h], aux, kb + 1 + h);
    }
    const int at = 9 * k0 - 8, rc = 3 * L.r + L.c, cr = 3 * L.c + L.r;
    auto mine = [&](int h) { return (G != 32 || h < m) && k0 + h >= 1; };
    const double2 *xa = sm + A + at + (da ? cr : rc), *xb = sm + Bs + at + (db ? cr : rc);
    // the flags' terms b0 A_k + a0 B_k; a zero flag contributes an exact zero, so
    // its term is skipped (the operand may be unset there)
    if (one) {
#pragma unroll
      for (int h = 0; h < R; h++)
        if (mine(h)) res[h] = cadd(res[h], cadd(wconj(xa[9 * h], sa), wconj(xb[9 * h], sb)));
    } else if (!none) {
#pragma unroll
      for (int h = 0; h < R; h++)
        if (mine(h)) {
          double2 v = cz();
          if (!cis0(b0)) v = cmul(b0, wconj(xa[9 * h], sa));
          if (!cis0(a0)) v = cadd(v, cmul(a0, wconj(xb[9 * h], sb)));
          res[h] = cadd(res[h], v);
        }
    }
    if (X >= 0) {
#pragma unroll
      for (int h = 0; h < R; h++)
        if (mine(h)) res[h] = cadd(res[h], cscale(sm[X + at + 9 * h + rc], cx));
    }
    gsync<G>();
    if (G != 32 || L.lane < 27) {
      if (gout) {
#pragma unroll
        for (int h = 0; h < R; h++)
          if (mine(h)) gout[at + 9 * h + rc] = res[h];
      } else {
#pragma unroll
        for (int h = 0; h < R; h++)
          if (mine(h)) sm[out + at + 9 * h + rc] = res[h];
      }
    }
    gsync<G>();
  }
  if (L.lane == 0 && (X < 0 || X == out)) {
    const double2 f = flag_mul(a0, b0);
    (gout ? gout : sm + out)[0] = X == out ? cadd(sm[out], f) : f;
  }
  gsync<G>();
}

// out (a slot, or gout) <- op(A) op(B), or += with MUL_ACC; flag included.  FP64
// or float-float.
template <bool FF, int G>
__device__ __forceinline__ void ser_mul_x(int out, int A, int Bs, int N, int ffe, unsigned mode,
                                          double2 *gout = nullptr) {
  const int X = mode & MUL_ACC ? out : -1;
  typedef typename std::conditional<FF, AccFF, Acc64>::type Acc;
  if (mode & (MUL_DA | MUL_DB | MUL_DAG))
    ser_mul_any<Acc, G, true>(out, A, Bs, N, mode, ffe, X, 1.0, gout);
  else
    ser_mul_any<Acc, G, false>(out, A, Bs, N, mode, ffe, X, 1.0, gout);
}
template <int G>
__device__ __forceinline__ void ser_mul(int out, int A, int Bs, int N, unsigned mode = 0) {
  ser_mul_x<false, G>(out, A, Bs, N, 0, mode);
}

// R <- p(X) = sum_{n<=N} coef(n) X^n for a series X whose flag counts as 0, by
// Paterson-Stockmeyer with block 2: Y = X^2 once, then Horner in Y,
// S_j = Y S_{j+1} + coef(2j) + coef(2j+1) X, S_j to order N - 2j (Y^j starts at
// order 2j): 1 + N/2 products of sizes 2, 4, ..., N.  X, Y (scratch) and R are
// slots; R's flag becomes coef(0).  DAG: the copy of the product to use.
template <int G, bool DAG, class Coef>
__device__ __forceinline__ void ser_poly(int X, int Y, int R, int N, Coef coef) {
  double2 *sm = wsm();
  const int lane = glane<G>();
  ser_mul<G>(Y, X, X, N, MUL_A0 | MUL_B0 | (DAG ? MUL_DAG : 0));
  const int J = N / 2;
  {
    const double cx = coef(2 * J + 1);
    for (int e = 1 + lane; e <= 9 * N; e += glanes<G>())
      sm[R + e] = e <= 9 * (N - 2 * J) ? cscale(sm[X + e], cx) : cz();
    if (lane == 0) sm[R] = make_double2(coef(2 * J), 0.0);
    gsync<G>();
  }
#pragma unroll 1
  for (int j = J - 1; j >= 0; --j) {
    ser_mul_any<Acc64, G, DAG>(R, Y, R, N - 2 * j, MUL_A0, 0, X, coef(2 * j + 1), nullptr);
    if (lane == 0) sm[R] = make_double2(coef(2 * j), 0.0);
    gsync<G>();
  }
}

// 1 / n!
__constant__ double c_invfact[52] = {
    1.0, 1.0, 0.5, 0.16666666666666666,
    0.041666666666666664, 0.008333333333333333, 0.001388888888888889, 0.0001984126984126984,
    2.48015873015873e-05, 2.7557319223985893e-06, 2.755731922398589e-07, 2.505210838544172e-08,
    2.08767569878681e-09, 1.6059043836821613e-10, 1.1470745597729725e-11, 7.647163731819816e-13,
    4.779477332387385e-14, 2.8114572543455206e-15, 1.5619206968586225e-16, 8.22063524662433e-18,
    4.110317623312165e-19, 1.9572941063391263e-20, 8.896791392450574e-22, 3.868170170630684e-23,
    1.6117375710961184e-24, 6.446950284384474e-26, 2.4795962632247976e-27, 9.183689863795546e-29,
    3.279889237069838e-30, 1.1309962886447716e-31, 3.7699876288159054e-33, 1.216125041553518e-34,
    3.8003907548547434e-36, 1.151633562077195e-37, 3.387157535521162e-39, 9.67759295863189e-41,
    2.6882202662866363e-42, 7.265460179153071e-44, 1.911963205040282e-45, 4.902469756513544e-47,
    1.2256174391283858e-48, 2.9893108271424046e-50, 7.117406731291439e-52, 1.6552108677421951e-53,
    3.7618428812322616e-55, 8.359650847182804e-57, 1.817315401561479e-58, 3.866628513960594e-60,
    8.055476070751236e-62, 1.643974708316579e-63, 3.287949416633158e-65, 6.446959640457172e-67};

// X <- exp(X) for X antihermitian and traceless with flag 0 (exp(const ptSU3&),
// QCDpt.h:200-220: sum_{n<=N} X^n / n!), flag 1.  X2, Z: scratch slots.
//
// Over the commutative ring of truncated series X satisfies its characteristic
// equation (Cayley-Hamilton): with H = -i X hermitian,
//   H^3 = tau H + delta,  tau = tr(H^2) / 2,  delta = tr(H^3) / 3, real series,
// so H^n = P_n + Q_n H + R_n H^2 with real series
//   R_{n+1} = tau R_{n-1} + delta R_{n-2},  Q_n = R_{n+1},  P_n = delta R_{n-1},
// and exp(X) = f0 + f1 X + f2 X^2 with three scalar series.  Two matrix
// products (X^2, and f1 X + f2 X^2 as one), the trace of X^2 X from its diagonal
// and upper triangle (X^2 is hermitian) and N^2/4 steps of scalar work instead of the 1 + N/2 products of Horner in X^2, whose small sizes
// cost a product's fixed part each.  The error against exact arithmetic is that
// of the Horner form (both 1e-16 to 6e-16 per order, up to 40 orders).
// Lanes own orders: up to EXP_LANE each, so G = 9 serves N < 18 (it is used to 14).
constexpr int EXP_LANE = 2;
template <int G, bool DAG>
__device__ __noinline__ void ser_exp(int X, int X2, int Z, int N) {
  double2 *sm = wsm();
  double *smd = reinterpret_cast<double *>(sm);
  const int lane = glane<G>();
  const unsigned copy = MUL_A0 | MUL_B0 | (DAG ? MUL_DAG : 0);
  ser_mul<G>(X2, X, X, N, copy);
  // scratch in Z: (tau, delta) of order k at td + k, then R_{n-2}, R_{n-1}, R_n
  const int td = Z, len = N + 1;
  int r0 = 2 * (Z + len), r1 = r0 + len, r2 = r1 + len;
  double2 own[EXP_LANE];
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++) {
    const int k = lane + glanes<G>() * h;
    own[h] = cz();
    if (k >= 1 && k <= N) {
      const double2 *p = sm + X2 + 9 * k - 8;
      // Im tr(X^2 X)_k, each entry above the diagonal for both of its pair
      double d = 0.0, o = 0.0;
#pragma unroll 2
      for (int i = 2; i < k; i++) {
        const double2 *y = sm + X2 + 9 * i - 8, *x = sm + X + 9 * (k - i) - 8;
        d = fma(y[0].x, x[0].y, d);
        o = fma(y[1].x, x[1].y, o);
        d = fma(y[4].x, x[4].y, d);
        o = fma(-y[1].y, x[1].x, o);
        d = fma(y[8].x, x[8].y, d);
        o = fma(y[2].x, x[2].y, o);
        o = fma(-y[2].y, x[2].x, o);
        o = fma(y[5].x, x[5].y, o);
        o = fma(-y[5].y, x[5].x, o);
      }
      own[h] = make_double2(-0.5 * (p[0].x + p[4].x + p[8].x), fma(2.0, o, d) * (-1.0 / 3.0));
    }
  }
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++) {
    const int k = lane + glanes<G>() * h;
    if (k <= N) {
      sm[td + k] = own[h];
      smd[r0 + k] = smd[r1 + k] = 0.0;
      smd[r2 + k] = k == 0 ? 1.0 : 0.0;
    }
  }
  gsync<G>();
  // s2 = sum c_n i^n R_n, s1 = sum c_n i^n Q_n, s0 = sum c_n i^n R_{n-1}, c_n = 1/n!
  double2 s0[EXP_LANE], s1[EXP_LANE], s2[EXP_LANE];
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++) s0[h] = s1[h] = s2[h] = cz();
  double sg = -1.0;  // i^n for even n
#pragma unroll 1
  for (int n = 2; n <= N + 1; n += 2, sg = -sg) {
    double v1[EXP_LANE], v2[EXP_LANE];  // R_{n+1}, R_{n+2}
    const double cm = sg * c_invfact[n - 1], c0 = sg * c_invfact[n], c1 = sg * c_invfact[n + 1],
                 c2 = sg * c_invfact[n + 2];
#pragma unroll
    for (int h = 0; h < EXP_LANE; h++) {
      const int k = lane + glanes<G>() * h;
      v1[h] = v2[h] = 0.0;
      if (k >= N) continue;  // R is needed to order N - 1
      // R_m starts at order m - 2
#pragma unroll 2
      for (int i = 2; i <= k - (n > 4 ? n - 4 : 0); i++) {
        const double2 t = sm[td + i];
        const double a = smd[r0 + k - i], b = smd[r1 + k - i], c = smd[r2 + k - i];
        v1[h] = fma(t.x, b, v1[h]);
        v2[h] = fma(t.x, c, v2[h]);
        v1[h] = fma(t.y, a, v1[h]);
        v2[h] = fma(t.y, b, v2[h]);
      }
      const double r = smd[r2 + k];
      s2[h].x = fma(c0, r, s2[h].x);
      s2[h].y = fma(c1, v1[h], s2[h].y);
      s1[h].y = fma(-cm, r, s1[h].y);
      s1[h].x = fma(c0, v1[h], s1[h].x);
      s0[h].y = fma(c1, r, s0[h].y);
      s0[h].x = fma(-c2, v1[h], s0[h].x);
    }
    gsync<G>();
#pragma unroll
    for (int h = 0; h < EXP_LANE; h++) {
      const int k = lane + glanes<G>() * h;
      if (k < N) smd[r0 + k] = v1[h], smd[r1 + k] = v2[h];
    }
    const int t = r0;
    r0 = r2;
    r2 = r1;
    r1 = t;
    gsync<G>();
  }
  // f0 = 1 + delta s0, f1 = -i s1, f2 = -s2 (H^2 = -X^2); orders 1..N into Z as
  // the entries 3, 0 and 1 of its records
  const int sp = Z + len;
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++)
    if (lane + glanes<G>() * h <= N) sm[sp + lane + glanes<G>() * h] = s0[h];
  gsync<G>();
  double2 f0[EXP_LANE];
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++) {
    const int k = lane + glanes<G>() * h;
    f0[h] = cz();
    if (k <= N)
      for (int i = 3; i <= k; i++) {
        const double d = sm[td + i].y;
        const double2 v = sm[sp + k - i];
        f0[h].x = fma(d, v.x, f0[h].x);
        f0[h].y = fma(d, v.y, f0[h].y);
      }
  }
  gsync<G>();
#pragma unroll
  for (int h = 0; h < EXP_LANE; h++) {
    const int k = lane + glanes<G>() * h;
    if (k >= 1 && k <= N) {
      double2 *z = sm + Z + 9 * k - 8;
      z[0] = make_double2(s1[h].y, -s1[h].x);
      z[1] = make_double2(-s2[h].x, -s2[h].y);
      z[3] = f0[h];
    }
  }
  gsync<G>();
  // orders >= 1 of f1 and f2 by the product, their order 0 (1 and 1/2) and f0 after
  ser_mul_any<Acc64, G, DAG>(X, Z, X, N, MUL_A0 | MUL_B0 | MUL_MIX, X2 - X, X, 1.0, nullptr);
  for (int e = 1 + lane; e <= 9 * N; e += glanes<G>()) {
    double2 v = cadd(sm[X + e], cscale(sm[X2 + e], 0.5));
    const int m = (e - 1) % 9;
    if (m == 0 || m == 4 || m == 8) v = cadd(v, sm[Z + e - m + 3]);
    sm[X + e] = v;
  }
  if (lane == 0) sm[X] = make_double2(1.0, 0.0);
  gsync<G>();
}

// The same by Horner in X^2, into R (a slot); odd = -1: exp(-X)
template <int G, bool DAG>
__device__ __forceinline__ void ser_exp_horner(int X, int Y, int R, int N, double odd = 1.0) {
  ser_poly<G, DAG>(X, Y, R, N,
                   [odd](int n) { return (n & 1) ? odd * inv_factorial(n) : inv_factorial(n); });
}
// exp of slot X by the form's algorithm; returns the slot it is in (X or R)
template <int G, bool DAG>
__device__ __forceinline__ int ser_exp_to(int X, int Y, int R, int N) {
  if constexpr (G == ORDERED) {
    ser_exp_horner<G, DAG>(X, Y, R, N);
    return R;
  } else {
    ser_exp<G, DAG>(X, Y, R, N);
    return X;
  }
}

// R <- log(U) for U with flag 1 (QCDpt.h:176-198), flag 0; Y scratch
template <int G, bool DAG>
__device__ __forceinline__ void ser_log(int U, int Y, int R, int N) {
  ser_poly<G, DAG>(U, Y, R, N,
                   [](int n) { return n == 0 ? 0.0 : ((n & 1) ? 1.0 : -1.0) / (double)n; });
}

// (M - M^dag)/2 minus a third of the trace times 1 (ptSU3::reH,
// QCDpt.cc:197-209) of one order in registers, row major
__device__ __forceinline__ void reh3(double2 *m) {
  const double D3 = 1.0 / 3.0;
  double2 b[9];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const double2 d = csub(m[3 * r + q], cconj(m[3 * q + r]));
      b[3 * r + q] = make_double2(.5 * d.x, .5 * d.y);
    }
  double2 tr = cadd(cadd(b[0], b[4]), b[8]);
  tr = make_double2(tr.x * D3, D3 * tr.y);
  b[0] = csub(b[0], tr);
  b[4] = csub(b[4], tr);
  b[8] = csub(b[8], tr);
#pragma unroll
  for (int e = 0; e < 9; e++) m[e] = b[e];
}

// reH on a slot, flag 0; lanes split the orders
template <int G>
__device__ __forceinline__ void ser_reH(int P, int N) {
  double2 *sm = wsm();
  const int lane = glane<G>();
  for (int k = 1 + lane; k <= N; k += glanes<G>()) {
    double2 *p = sm + P + 9 * k - 8;
    double2 m[9];
#pragma unroll
    for (int e = 0; e < 9; e++) m[e] = p[e];
    reh3(m);
#pragma unroll
    for (int e = 0; e < 9; e++) p[e] = m[e];
  }
  if (lane == 0) sm[P] = cz();
  gsync<G>();
}

// ---------------- staging ----------------

// Copy n double2 from global memory into a slot, asynchronously and through L2
// (coherent with writes of this kernel); wstage_wait() ends all copies begun.
template <int G>
__device__ __forceinline__ void wstage(int slot, const double2 *src, int n) {
  double2 *sm = wsm();
  for (int e = glane<G>(); e < n; e += glanes<G>()) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(sm + slot + e);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + e) : "memory");
  }
}
template <int G>
__device__ __forceinline__ void wstage_wait() {
  cp_commit();
  cp_wait0();
  gsync<G>();
}

// Twist a staged series for the faces its read crossed: Omega U Omega^dag,
// flag 1 (twist_* returns a default flag, nspt.cc:115-121).
template <int G>
__device__ __noinline__ void wtwist(int slot, unsigned tb, unsigned tf, int N) {
  double2 *sm = wsm();
  const int lane = glane<G>();
  for (int k = 1 + lane; k <= N; k += glanes<G>()) {
    double2 *p = sm + slot + 9 * k - 8;
    double2 m[9];
#pragma unroll
    for (int e = 0; e < 9; e++) m[e] = p[e];
    twist3(m, tb, tf);
#pragma unroll
    for (int e = 0; e < 9; e++) p[e] = m[e];
  }
  if (lane == 0) sm[slot] = make_double2(1.0, 0.0);
  gsync<G>();
}

// The slot to a record in global memory
template <int G>
__device__ __forceinline__ void wstore(double2 *dst, int slot, int n) {
  const double2 *sm = wsm();
  for (int e = glane<G>(); e < n; e += glanes<G>()) dst[e] = sm[slot + e];
}

}  // namespace nspt
