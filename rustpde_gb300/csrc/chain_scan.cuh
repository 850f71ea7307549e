// chain_scan.cuh -- warp-parallel linear recurrences along lane chains.
//
// The banded operators of the spectral step (Chebyshev derivative suffix sums,
// the stride-2 tridiagonal of from_ortho, the forward elimination and back
// substitution of the swept banded solve) are linear recurrences along each
// parity chain of a lane.  On this GPU an FP64 warp instruction occupies the
// FP64 pipe for the whole warp however few threads are active, so a chain run
// by one thread wastes 31/32 of the pipe.  Here each chain is run by a group
// of T threads as a scan of affine maps:
//   first order   x_t = a_t x_{t-1} + b_t
//   second order  (x_t, x_{t-1}) = [[a_t, c_t], [1, 0]] (x_{t-1}, x_{t-2}) + (b_t, 0)
// phase 1 composes each thread's block of E = ceil(len / T) maps, phase 2 scans
// the T block maps with shuffles, phase 3 replays the block from the exclusive
// prefix.  Coefficients are real; values are double or double2.  Warps with
// no chain left skip the rounds (the CTA-wide calls often have 2 chains).
#pragma once
#include <cuda_runtime.h>

namespace rbc {
namespace dev {

__device__ __forceinline__ double shfl_up_v(double v, int o, int w) { return __shfl_up_sync(0xffffffffu, v, o, w); }
__device__ __forceinline__ double2 shfl_up_v(double2 v, int o, int w) {
  return make_double2(__shfl_up_sync(0xffffffffu, v.x, o, w), __shfl_up_sync(0xffffffffu, v.y, o, w));
}
__device__ __forceinline__ double axpy_v(double a, double x, double b) { return fma(a, x, b); }
__device__ __forceinline__ double2 axpy_v(double a, double2 x, double2 b) {
  return make_double2(fma(a, x.x, b.x), fma(a, x.y, b.y));
}
template <class V> __device__ __forceinline__ V zero_val();
template <> __device__ __forceinline__ double zero_val<double>() { return 0.0; }
template <> __device__ __forceinline__ double2 zero_val<double2>() { return make_double2(0.0, 0.0); }

// The coefficients of a chain do not depend on the data, so neither do the
// composed maps of the blocks: they are computed once (scan_tables1/2, with the
// operations the scans would use, so that results do not depend on it) and only
// the values go through phases 1 and 2.  That halves the FP64 operations of a
// banded solve (15 -> 7 per element) and shortens the dependent path of an
// element from two multiply-adds to one.
constexpr int kScanT = 16;      // threads per chain

// Elements per thread of a chain.  The threads of a chain read shared memory
// 2 E elements apart, so an even E puts them on few banks: 16-way conflicts
// from E = 8 on at the lengths 2^p + 1, where E is a power of two.  FP64 cases
// take odd blocks there (two threads share a bank; box 513^2: x2 69 -> 49 us,
// y3 77 -> 49 us, the step 606 -> 506 us); shorter chains lose more by the
// longer block than by the conflicts (box 64^2: 92 -> 96 us).  The mixed form
// keeps E = ceil(len / 16): another blocking rounds the FP64 values differently
// in the last bit, which its FP32 copies of the state amplify to 2e-9 of the
// results.
__host__ __device__ __forceinline__ int scan_block(int len, int odd) {
  const int E = (len + kScanT - 1) / kScanT;
  return odd && E >= 8 ? E | 1 : E;
}

constexpr int kScanRounds = 4;  // log2(kScanT)

// First-order chains.  coef(c, t, a, b) gives the map of element t of chain c
// (t = 0 must give a = 0), store(c, t, x) receives x_t; round_a(c, gl, r) is
// the composed coefficient of thread gl before round r.  coef is called twice
// per element, first = true in the first phase.  All threads of the CTA call
// this (uniformly); it contains no barrier.
template <class V, class LenF, class CoefF, class RoundF, class StoreF>
__device__ __forceinline__ void chains1(int odd, int nch, LenF len_of, CoefF coef, RoundF round_a, StoreF store, int tid,
                                        int nth) {
  constexpr int T = kScanT;
  const int g = tid / T, gl = tid % T, ng = nth / T;
  for (int base = 0; base < nch; base += ng) {
    // a warp whose groups all lie past the last chain has no work here or in
    // later rounds (its shuffles involve only itself)
    if (base + (tid & ~31) / T >= nch) break;
    const int c = base + g;
    const bool on = c < nch;
    const int len = on ? len_of(c) : 0;
    const int E = scan_block(len, odd);
    const int t0 = gl * E, t1 = min(t0 + E, len);
    double ra[kScanRounds];
#pragma unroll
    for (int r = 0; r < kScanRounds; r++) ra[r] = on ? round_a(c, gl, r) : 0.0;
    V B = zero_val<V>();
    for (int t = t0; t < t1; t++) {
      double a;
      V b;
      coef(c, t, a, b, true);
      B = axpy_v(a, B, b);
    }
#pragma unroll
    for (int r = 0; r < kScanRounds; r++) {
      const V Bp = shfl_up_v(B, 1 << r, T);
      if (gl >= (1 << r)) B = axpy_v(ra[r], Bp, B);
    }
    V x = shfl_up_v(B, 1, T);  // value before this thread's block (map 0 has a = 0)
    if (gl == 0) x = zero_val<V>();
    for (int t = t0; t < t1; t++) {
      double a;
      V b;
      coef(c, t, a, b, false);
      x = axpy_v(a, x, b);
      store(c, t, x);
    }
  }
}

// Running sums along chains (all coefficients 1): value(c, t), store(c, t, sum).
template <class V, class LenF, class ValF, class StoreF>
__device__ __forceinline__ void chains_sum(int odd, int nch, LenF len_of, ValF value, StoreF store, int tid, int nth) {
  constexpr int T = kScanT;
  const int g = tid / T, gl = tid % T, ng = nth / T;
  for (int base = 0; base < nch; base += ng) {
    if (base + (tid & ~31) / T >= nch) break;  // as in chains1
    const int c = base + g;
    const int len = c < nch ? len_of(c) : 0;
    const int E = scan_block(len, odd);
    const int t0 = gl * E, t1 = min(t0 + E, len);
    V B = zero_val<V>();
    for (int t = t0; t < t1; t++) B = axpy_v(1.0, B, value(c, t));
#pragma unroll
    for (int o = 1; o < T; o <<= 1) {
      const V Bp = shfl_up_v(B, o, T);
      if (gl >= o) B = axpy_v(1.0, Bp, B);
    }
    V x = shfl_up_v(B, 1, T);
    if (gl == 0) x = zero_val<V>();
    for (int t = t0; t < t1; t++) {
      x = axpy_v(1.0, x, value(c, t));
      store(c, t, x);
    }
  }
}

// Second-order chains: x_t = a_t x_{t-1} + c_t x_{t-2} + b_t.  coef(c, t, a, cc,
// b, first); round_m(c, gl, r, e): entry e of the composed matrix of thread gl
// before round r.
template <class V, class LenF, class CoefF, class RoundF, class StoreF>
__device__ __forceinline__ void chains2(int odd, int nch, LenF len_of, CoefF coef, RoundF round_m, StoreF store, int tid,
                                        int nth) {
  constexpr int T = kScanT;
  const int g = tid / T, gl = tid % T, ng = nth / T;
  for (int base = 0; base < nch; base += ng) {
    if (base + (tid & ~31) / T >= nch) break;  // as in chains1
    const int c = base + g;
    const bool on = c < nch;
    const int len = on ? len_of(c) : 0;
    const int E = scan_block(len, odd);
    const int t0 = gl * E, t1 = min(t0 + E, len);
    double rm[kScanRounds][4];
#pragma unroll
    for (int r = 0; r < kScanRounds; r++)
#pragma unroll
      for (int e = 0; e < 4; e++) rm[r][e] = on ? round_m(c, gl, r, e) : 0.0;
    V B0 = zero_val<V>(), B1 = zero_val<V>();
    for (int t = t0; t < t1; t++) {
      double a, cc;
      V b;
      coef(c, t, a, cc, b, true);
      const V nb0 = axpy_v(a, B0, axpy_v(cc, B1, b));
      B1 = B0;
      B0 = nb0;
    }
#pragma unroll
    for (int r = 0; r < kScanRounds; r++) {
      const V q0 = shfl_up_v(B0, 1 << r, T), q1 = shfl_up_v(B1, 1 << r, T);
      if (gl >= (1 << r)) {
        // self o prev: B = M_self B_prev + B_self
        const V nb0 = axpy_v(rm[r][0], q0, axpy_v(rm[r][1], q1, B0));
        const V nb1 = axpy_v(rm[r][2], q0, axpy_v(rm[r][3], q1, B1));
        B0 = nb0;
        B1 = nb1;
      }
    }
    // state before the block: (x_{t0-1}, x_{t0-2}) = inclusive result of the previous thread
    V x1 = shfl_up_v(B0, 1, T), x2 = shfl_up_v(B1, 1, T);
    if (gl == 0) { x1 = zero_val<V>(); x2 = zero_val<V>(); }
    for (int t = t0; t < t1; t++) {
      double a, cc;
      V b;
      coef(c, t, a, cc, b, false);
      V x = axpy_v(a, x1, axpy_v(cc, x2, b));
      store(c, t, x);
      x2 = x1;
      x1 = x;
    }
  }
}

// The composed coefficients of one chain, by the kScanT threads of a group
// (all 32 threads of the warp call): out(r, value) before each round.
template <class CoefF, class OutF>
__device__ __forceinline__ void scan_tables1(int odd, int len, int gl, CoefF coef, OutF out) {
  constexpr int T = kScanT;
  const int E = scan_block(len, odd), t0 = gl * E, t1 = min(t0 + E, len);
  double A = 1.0;
  for (int t = t0; t < t1; t++) A = coef(t) * A;
#pragma unroll
  for (int r = 0; r < kScanRounds; r++) {
    out(r, A);
    const double Ap = __shfl_up_sync(0xffffffffu, A, 1 << r, T);
    if (gl >= (1 << r)) A = A * Ap;
  }
}
template <class CoefF, class OutF>
__device__ __forceinline__ void scan_tables2(int odd, int len, int gl, CoefF coef, OutF out) {
  constexpr int T = kScanT;
  const int E = scan_block(len, odd), t0 = gl * E, t1 = min(t0 + E, len);
  // block map: (x, x') -> (m00 x + m01 x' + B0, m10 x + m11 x' + B1)
  double m00 = 1.0, m01 = 0.0, m10 = 0.0, m11 = 1.0;
  for (int t = t0; t < t1; t++) {
    double a, cc;
    coef(t, a, cc);
    // new = [[a, cc], [1, 0]] * old
    const double n00 = fma(a, m00, cc * m10), n01 = fma(a, m01, cc * m11);
    m10 = m00; m11 = m01;
    m00 = n00; m01 = n01;
  }
#pragma unroll
  for (int r = 0; r < kScanRounds; r++) {
    out(r, 0, m00);
    out(r, 1, m01);
    out(r, 2, m10);
    out(r, 3, m11);
    const double p00 = __shfl_up_sync(0xffffffffu, m00, 1 << r, T), p01 = __shfl_up_sync(0xffffffffu, m01, 1 << r, T);
    const double p10 = __shfl_up_sync(0xffffffffu, m10, 1 << r, T), p11 = __shfl_up_sync(0xffffffffu, m11, 1 << r, T);
    if (gl >= (1 << r)) {
      const double n00 = fma(m00, p00, m01 * p10), n01 = fma(m00, p01, m01 * p11);
      const double n10 = fma(m10, p00, m11 * p10), n11 = fma(m10, p01, m11 * p11);
      m00 = n00; m01 = n01; m10 = n10; m11 = n11;
    }
  }
}

}  // namespace dev
}  // namespace rbc
