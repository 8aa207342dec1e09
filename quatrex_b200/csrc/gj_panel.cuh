// Register-resident factorization of one Gauss-Jordan panel (n rows x NB
// columns), shared by the one-CTA (zinv.cu) and the cluster
// (zinv_cluster.cu) batched inverses.
//
// LPR lanes (one or two) hold a row of the panel for all of its columns, lane h
// of them columns h, h + LPR, ..., so a column step touches shared memory only for the pivot search partials and the
// broadcast pivot row. Rows are not interchanged: each thread tracks the
// position its row would have after LAPACK's interchanges. Per column k:
//   pivot  p = argmax_{pos >= k} |Re| + |Im| of column k (lowest position on
//          ties, the izamax measure of LAPACK that numpy.linalg.inv uses);
//   the pivot row's thread publishes the row q and takes position k, the
//   row at position k takes position p;
//   with m = x_rk / x_pk every other row is eliminated, x_rc -= m q_c
//   (c != k), x_rk <- -m, and the pivot row becomes q / x_pk.
// Afterwards the rows, stored at their positions, hold the transform T of the
// panel (T = [A_KK^-1 ; -A_RK A_KK^-1] in block form).
//
// A column step is a chain of latencies and of instructions that every warp
// issues: the search compares the measures as integers (one redux of the high
// words and a ballot, a slow path only if they tie) instead of five shuffle
// rounds; the candidate's value travels with the search, so that every thread
// forms 1 / x_pk itself while the pivot row is published; and the loop over the
// columns is rolled. Cycles per column in the inverse at n = 64 / 128 / 256: with
// one lane 1570 / 2020 / 2240, with two 1350 / 1660 / 2450 (half the row to
// publish and to update, twice the warps to search), so two up to n = 128. (Two
// lanes, five shuffle rounds and an unrolled loop took about 3000 at n = 256.)
// These are with four-instruction eliminations; with the six of gj_eliminate they
// are about 50, 30 and 290 more.
// Measured beside it, alone, at n = 64 / 256: one lane 1120 / 1455, every warp
// publishing its candidate row ahead of a single barrier 1130 / 2340, whole
// columns in a warp with the multipliers published 1100 / 2440.
#pragma once

#include "common.cuh"

namespace qtx {

// 1 / z for a complex z. z is scaled by the power of two 2^-e that brings its
// larger part into [0.5, 1) (exact), so that m = |z'|^2 lies in [0.25, 2);
// 1 / m comes from the hardware reciprocal estimate (PTX rcp.approx.ftz.f64)
// refined by three Newton-Raphson steps y <- y + y (1 - m y), each of which
// doubles the number of correct bits; then 1 / z = conj(z') (1 / m) 2^-e.
// A few ulps from the correctly rounded quotient, like Smith's algorithm,
// with one short dependency chain instead of three divisions.
// gj_recip_scaled: the same with frexp / ldexp (any exponent, zero, subnormals).
__device__ __forceinline__ z64 gj_recip_scaled(z64 z) {
  const double mx = fmax(fabs(z.x), fabs(z.y));
  if (mx == 0.0) return make_double2(0.0, 0.0);
  int e;
  frexp(mx, &e);
  const double xs = ldexp(z.x, -e), ys = ldexp(z.y, -e);
  const double m = fma(xs, xs, __dmul_rn(ys, ys));
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
#pragma unroll
  for (int it = 0; it < 3; ++it) y = fma(y, fma(-m, y, 1.0), y);
  return make_double2(ldexp(xs * y, -e), ldexp(-ys * y, -e));
}

// gj_recip: for exponents away from the ends of the range the scale 2^-e is
// built from the exponent field and applied by multiplication (exact, and
// the final product rounds like ldexp), which keeps frexp / ldexp off the
// pivot row's critical path; bit-identical to gj_recip_scaled.
__device__ __forceinline__ z64 gj_recip(z64 z) {
  const double mx = fmax(fabs(z.x), fabs(z.y));
  const int eb = (int)((__double_as_longlong(mx) >> 52) & 0x7FF);  // biased exponent field
  if (eb < 24 || eb > 2000) return gj_recip_scaled(z);             // zero, subnormal or extreme
  const int e = eb - 1022;                                         // frexp's exponent of mx
  const double s = __longlong_as_double((long long)(1023 - e) << 52);  // 2^-e
  const double xs = z.x * s, ys = z.y * s;
  const double m = fma(xs, xs, __dmul_rn(ys, ys));
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
#pragma unroll
  for (int it = 0; it < 3; ++it) y = fma(y, fma(-m, y, 1.0), y);
  return make_double2((xs * y) * s, (-ys * y) * s);
}

__device__ __forceinline__ double gj_abs1(z64 z) { return fabs(z.x) + fabs(z.y); }

// a b and v - m q with the roundings spelled out: every instantiation of the
// factorization gives the same bits, so one block's inverse does not depend on
// the path that the batch size selects. The product is formed before it is
// subtracted: adding its two real products to v one after another (four fma
// instead of six instructions) rounds at the size of v twice and made the error
// of the inverse 1.05 to 1.19 times as large at n = 16, its residual 1.02 to 1.2
// times up to n = 256. It costs 1 to 7 % of the inverse's time (64 x 32 61 -> 62.5
// us, 128 x 32 150.9 both, 256 x 148 1.33 -> 1.37 ms, 256 x 18 0.536 -> 0.573 ms).
__device__ __forceinline__ z64 gj_mul(z64 a, z64 b) {
  return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ z64 gj_eliminate(z64 v, z64 m, z64 q) {
  const z64 t = gj_mul(m, q);
  return make_double2(__dsub_rn(v.x, t.x), __dsub_rn(v.y, t.y));
}

// Shared memory of gj_factor_panel.
template <int NB>
struct GjPanelSmem {
  z64 q[2][NB];                // pivot row, double-buffered by column parity
  z64 val[16];                 // per-warp candidate: value,
  unsigned long long key[16];  // measure + 1 (0: none),
  int pos[16];                 // position
};

// The lane holding the largest key (lowest position on ties) of the warp.
// Every lane takes part in every step of the search.
__device__ __forceinline__ int gj_best_lane(unsigned long long key, int pos) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned m1 = __reduce_max_sync(0xffffffffu, hi);
  unsigned cand = __ballot_sync(0xffffffffu, hi == m1);
  if ((cand & (cand - 1)) != 0) {
    const unsigned lo = hi == m1 ? (unsigned)key : 0u;
    const unsigned m2 = __reduce_max_sync(0xffffffffu, lo);
    const bool c2 = hi == m1 && (unsigned)key == m2;
    const int m3 = __reduce_min_sync(0xffffffffu, c2 ? pos : 0x7fffffff);
    cand = __ballot_sync(0xffffffffu, c2 && pos == m3);
  }
  return __ffs(cand) - 1;
}

// Factors an n x nbp panel (nbp <= NB, n LPR <= 512); the first
// ceil(n LPR / 32) warps of the CTA take part and the others return at once (named barrier 1).
// load(r, c) / store(r, c, v): panel element access (r < n, c < nbp), the same
// memory or not (a barrier separates loads and stores); moved(r, pos), once per
// row after that barrier: row r ends at position pos. sing: shared int, set to
// k + 1 at the first zero pivot if still 0.
template <int NB, int LPR, class Load, class Store, class Moved>
__device__ __forceinline__ void gj_factor_panel(int n, int k0, int nbp, Load load, Store store, Moved moved,
                                                int* sing) {
  __shared__ GjPanelSmem<NB> sm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int C = NB / LPR;
  const int W = (n * LPR + 31) >> 5;
  if (warp >= W) return;
  const int bar_threads = W * 32;
  auto barrier = [&]() {
    if (W > 1)
      asm volatile("bar.sync 1, %0;\n" ::"r"(bar_threads) : "memory");
    else
      __syncwarp();
  };
  const int r = tid / LPR, h = tid % LPR;
  const bool live = r < n;
  int pos = live ? r : 0x7fffffff;
  z64 v[C];
#pragma unroll
  for (int i = 0; i < C; ++i)
    v[i] = (live && h + i * LPR < nbp) ? load(r, h + i * LPR) : make_double2(0.0, 0.0);
#pragma unroll 1
  for (int kk = 0; kk < nbp; ++kk) {
    const int k = k0 + kk, hk = kk % LPR;
    z64 xk = v[0];
    if (LPR > 1) {
      const int src = (lane & ~(LPR - 1)) | hk;
      xk.x = __shfl_sync(0xffffffffu, xk.x, src);
      xk.y = __shfl_sync(0xffffffffu, xk.y, src);
    }
    const bool mine = live && pos >= k && h == hk;
    {
      const double a = gj_abs1(xk);
      // NaN compares false: such a row is never chosen
      const unsigned long long key = (mine && a >= 0.0) ? (unsigned long long)__double_as_longlong(a) + 1 : 0ull;
      const int tie = mine ? pos : 0x7fffffff;
      if (lane == gj_best_lane(key, tie)) {
        sm.key[warp] = key;
        sm.pos[warp] = tie;
        sm.val[warp] = xk;
      }
    }
    barrier();
    const unsigned long long wkey = lane < W ? sm.key[lane & 15] : 0ull;
    const int wpos = lane < W ? sm.pos[lane & 15] : 0x7fffffff;
    const int wl = gj_best_lane(wkey, wpos);
    const int p = __shfl_sync(0xffffffffu, wpos, wl);
    const z64 xp = sm.val[wl];
    const bool piv = live && pos == p;
    z64* q = sm.q[kk & 1];
    if (piv) {
#pragma unroll
      for (int i = 0; i < C; ++i) q[i * LPR + h] = v[i];
    }
    const z64 d = gj_recip(xp);
    z64 m = gj_mul(xk, d);
    if (piv) {
      if (sm.key[wl] <= 1ull && *sing == 0) *sing = k + 1;
#pragma unroll
      for (int i = 0; i < C; ++i) v[i] = make_double2(0.0, 0.0);  // q / x_pk as 0 - (-1 / x_pk) q
      m = make_double2(-d.x, -d.y);
      pos = k;
    } else if (pos == k) {
      pos = p;
    }
    barrier();
    // The columns rotate through the registers (every LPR steps): column k is
    // always in v[0]. The loop therefore stays rolled: unrolled over the columns
    // its straight-line code (5 KB a column) is fetched anew for every panel and
    // costs more than the arithmetic.
    if (LPR == 1) {
#pragma unroll
      for (int i = 1; i < C; ++i) {
        v[i - 1] = gj_eliminate(v[i], m, q[i]);
        if (i % 5 == 0) asm volatile("" ::: "memory");  // bounds the loads in flight (registers)
      }
      v[C - 1] = make_double2(-m.x, -m.y);
    } else {
#pragma unroll
      for (int i = 0; i < C; ++i) v[i] = gj_eliminate(v[i], m, q[i * LPR + h]);
      if (h == hk) v[0] = make_double2(-m.x, -m.y);
      if (hk == LPR - 1) {
        const z64 f = v[0];
#pragma unroll
        for (int i = 0; i + 1 < C; ++i) v[i] = v[i + 1];
        v[C - 1] = f;
      }
    }
  }
  barrier();  // every load of the panel (and of the last pivot row) is done
  if (live) {
    if (h == 0) moved(r, pos);
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const int g = i + nbp / LPR;
      const int col = h + LPR * (g < C ? g : g - C);  // after nbp / LPR rotations
      if (col < nbp) store(pos, col, v[i]);
    }
  }
}

}  // namespace qtx
