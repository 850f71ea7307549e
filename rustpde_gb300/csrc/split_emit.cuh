// split_emit.cuh -- FP64 lanes in shared memory -> the digit planes of the
// split GEMM (split_gemm.h).  Integer operations only: the FP64 pipe, the
// bottleneck of the passes that call this, is not used.
#pragma once
#include <cuda_runtime.h>

#include "split_gemm.h"

namespace rbc {
namespace dev {

// biased exponent field (1 for zeros and subnormals, whose scale it is)
__device__ __forceinline__ int split_exp(double v) {
  const int e = (__double2hiint(v) >> 20) & 0x7ff;
  return e == 0 ? 1 : e;
}

// round(v 2^(1075 - emax + shl)), |v| < 2^(emax - 1022)
__device__ __forceinline__ long long split_fix(double v, int emax, int shl) {
  const long long u = __double_as_longlong(v);
  const int f = (int)((unsigned long long)u >> 52) & 0x7ff;
  long long m = u & 0xFFFFFFFFFFFFFll;
  if (f != 0) m |= 1ll << 52;
  const int sh = emax - (f == 0 ? 1 : f);
  m <<= shl;
  m = sh == 0 ? m : sh > 60 ? 0 : (m + (1ll << (sh - 1))) >> sh;
  const long long s = u >> 63;
  return (m ^ s) - s;
}

// Digits of 8 consecutive terms of one lane, written as 16 bytes per plane.
// Adding 0x80 to each of the six low bytes turns them into unsigned bytes
// d + 128 of the balanced digits d in [-128, 127]; the rest is the top digit.
// A byte b becomes the float b - 128 through the bits of 2^23 + b; digits have
// at most 8 significant bits, so the upper half of the float is the bf16.
template <class GetX>
__device__ __forceinline__ void split_store8(unsigned char* dst, GetX get) {
  uint32_t out[kSplitDigits][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t fl[2][kSplitDigits];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const long long y = get(2 * q + h) + 0x0000808080808080ll;
      const uint32_t lo = (uint32_t)y, hi = (uint32_t)((unsigned long long)y >> 32);
      fl[h][0] = __float_as_uint((float)((int)hi >> 16));
      fl[h][1] = __float_as_uint(__uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7651)) - 8388736.0f);
      fl[h][2] = __float_as_uint(__uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7650)) - 8388736.0f);
      fl[h][3] = __float_as_uint(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7653)) - 8388736.0f);
      fl[h][4] = __float_as_uint(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7652)) - 8388736.0f);
      fl[h][5] = __float_as_uint(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7651)) - 8388736.0f);
      fl[h][6] = __float_as_uint(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7650)) - 8388736.0f);
    }
#pragma unroll
    for (int i = 0; i < kSplitDigits; i++) out[i][q] = __byte_perm(fl[0][i], fl[1][i], 0x7632);
  }
#pragma unroll
  for (int i = 0; i < kSplitDigits; i++)
    *reinterpret_cast<uint4*>(dst + i * (kSplitLanes * kSplitK * 2)) =
        make_uint4(out[i][0], out[i][1], out[i][2], out[i][3]);
}

// Lanes lane0 .. lane0 + nl - 1 of the set: lane r has n stored values val(r, k)
// (k < n; scanned for the largest exponent) and terms term(r, list, k, fix) for
// k < K[list], where fix(v) gives a value's integer.  em: nl ints of shared
// memory.  Called by all threads of the CTA; ends without a barrier.
template <class ValF, class TermF>
__device__ __forceinline__ void split_emit(const SplitLanesDev& S, int lane0, int nl, int n, int KE, int KO, int shl,
                                           ValF val, TermF term, int* em, int tid, int nth) {
  const int warp = tid >> 5, wl = tid & 31, nw = nth >> 5;
  for (int r = warp; r < nl; r += nw) {
    int e = 1;
    for (int k = wl; k < n; k += 32) e = max(e, split_exp(val(r, k)));
    e = __reduce_max_sync(0xffffffffu, e);
    if (wl == 0) {
      em[r] = e;
      S.ex[lane0 + r] = e;
    }
  }
  __syncthreads();
  const int gE = 2 * S.cE, groups = 2 * (S.cE + S.cO);
  for (int it = tid; it < nl * groups; it += nth) {
    const int g = it / nl, r = it - g * nl;  // neighbouring threads: neighbouring lanes, 16 bytes apart
    const int list = g >= gE, k0 = 8 * (list ? g - gE : g), K = list ? KO : KE;
    const int lane = lane0 + r, lb = lane & (kSplitLanes - 1), emax = em[r];
    unsigned char* dst = S.dig + (size_t)((lane / kSplitLanes) * (S.cE + S.cO) + (g >> 1)) * kSplitChunkBytes +
                         (g & 1) * (kSplitLanes * 16) + (lb >> 3) * 128 + (lb & 7) * 16;
    split_store8(dst, [&](int t) -> long long {
      const int k = k0 + t;
      return k < K ? term(r, list, k, [&](double v) { return split_fix(v, emax, shl); }) : 0ll;
    });
  }
}

// ---- nine digits (SplitMat): one list after the other, terms val(r, k) 2^colex[k]
template <class ValF>
__device__ __forceinline__ void split_emit9(const SplitLanesDev& S, int lane0, int nl, int n, int K0,
                                            const int* __restrict__ colex, ValF val, int* em, int tid, int nth) {
  const int warp = tid >> 5, wl = tid & 31, nw = nth >> 5;
  for (int r = warp; r < nl; r += nw) {
    int e = -4096;
    bool bad = false;
    for (int k = wl; k < n; k += 32) {
      const double v = val(r, k);
      const int f = split_exp(v);
      bad |= f == 0x7ff;
      if (v != 0.0) e = max(e, f + __ldg(colex + k));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    bad = __any_sync(0xffffffffu, bad);
    if (wl == 0) {
      em[r] = e;
      S.ex[lane0 + r] = bad ? kSplitBadLane9 : e == -4096 ? 1 : e;
    }
  }
  __syncthreads();
  const int g0 = 2 * S.cE, groups = 2 * (S.cE + S.cO);
  for (int it = tid; it < nl * groups; it += nth) {
    const int g = it / nl, r = it - g * nl;
    const int k0 = g < g0 ? 8 * g : K0 + 8 * (g - g0), k1 = g < g0 ? K0 : n;
    const int lane = lane0 + r, lb = lane & (kSplitLanes - 1), emax = em[r];
    unsigned char* dst = S.dig + (size_t)((lane / kSplitLanes) * (S.cE + S.cO) + (g >> 1)) * (9 * kSplitLanes * kSplitK * 2) +
                         (g & 1) * (kSplitLanes * 16) + (lb >> 3) * 128 + (lb & 7) * 16;
    uint32_t out[9][4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t fl[2][9];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int k = k0 + 2 * q + h;
        const double v = k < k1 ? val(r, k) : 0.0;
        const long long u = __double_as_longlong(v);
        const int f = (int)((unsigned long long)u >> 52) & 0x7ff;
        unsigned long long m = (unsigned long long)u & 0xFFFFFFFFFFFFFull, lo = 0, hi = 0;
        if (f != 0) m |= 1ull << 52;
        // m 2^(kSplitShl9 - (emax - exponent)), rounded to nearest
        const int p = kSplitShl9 - (emax - ((f == 0 ? 1 : f) + (k < k1 ? __ldg(colex + k) : 0)));
        if (m != 0) {
          if (p >= 0) {
            lo = m << p;
            hi = p > 0 ? m >> (64 - p) : 0;
          } else if (p > -60) {
            lo = (m + (1ull << (-p - 1))) >> -p;
          }
        }
        if (u < 0) {
          lo = 0ull - lo;
          hi = ~hi + (lo == 0 ? 1 : 0);
        }
        const unsigned long long b = lo + 0x8080808080808080ull;
        const int top = (int)(long long)hi + (b < lo ? 1 : 0);
        fl[h][0] = __float_as_uint((float)top);
        const uint32_t w[2] = {(uint32_t)(b >> 32), (uint32_t)b};
#pragma unroll
        for (int i = 1; i < 9; i++)
          fl[h][i] = __float_as_uint(
              __uint_as_float(__byte_perm(w[(i - 1) >> 2], 0x4B000000u, 0x7650 + 3 - ((i - 1) & 3))) - 8388736.0f);
      }
#pragma unroll
      for (int i = 0; i < 9; i++) out[i][q] = __byte_perm(fl[0][i], fl[1][i], 0x7632);
    }
#pragma unroll
    for (int i = 0; i < 9; i++)
      *reinterpret_cast<uint4*>(dst + i * (kSplitLanes * kSplitK * 2)) =
          make_uint4(out[i][0], out[i][1], out[i][2], out[i][3]);
  }
}

}  // namespace dev
}  // namespace rbc
