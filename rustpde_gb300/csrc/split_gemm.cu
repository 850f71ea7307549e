// split_gemm.cu -- FP64 lanes times dense operators as exact digit products on
// tcgen05 (see split_gemm.h).
//
// One CTA computes a tile of 128 lanes x NT (32 or 16) outputs.  Per 16-term
// chunk it multiplies the seven digit planes A_i of the lanes with the digit
// planes W_j of the operator, i + j <= 7, into eight FP32 accumulators, one
// per weight d = i + j.  The planes W_0 .. W_m lie side by side as one operand
// and the accumulators side by side in tensor memory, so one MMA of N = NT
// (m + 1) columns, started at column i NT, does all products of A_i: 7 MMAs a
// chunk (8 in a list's first chunk, where they also initialise the
// accumulators).
//
// Exactness: |A_i digit| <= 128, |W_j digit| <= 128 (64 for j = 0); an
// accumulator sums at most (d + 1) K products, six of them for d = 7.  The
// operators' digits average half of their bound, so that for K <= 320 terms a
// list the sums of the weights d <= 5 stay below 2^24 whatever the lane's digits.
// A lane made for it could take d = 6 past that (random-signed sums have a
// standard deviation below 2^18) and lose its last unit with each product, less
// than 2^-55 of the largest product in all.
//
// Work split: warp 8 copies the chunks (28 KB of lane digits, 7 KB of operator
// digits at NT = 32; cp.async.bulk into a ring of three), one thread of warp 9
// issues the MMAs, warps 0-7 read the accumulators (warp w: lanes 32 (w % 4),
// half of the tile's outputs, w / 4).  The two lists of a wide tile use the same
// 256 tensor-memory columns one after the other, which leaves room for a second
// CTA on the SM: one CTA's epilogue runs under the other's MMAs.  A narrow
// tile's lists have columns of their own.
//
// Bound: one tile's serial chain (first copy, the chunks one after the other,
// and the epilogue's about 100 instructions per pair of outputs), not a pipe: ncu
// shows the tensor pipe 16 % busy and the L2 at 7 % of its rate with 153 CTAs (box
// 264^2, x backward), 54 % and 30 % with 297 (513^2), where two CTAs share most SMs.
// Hence narrow tiles in small launches.  Box 264^2, a GEMM alone with a cold L2,
// with 32-wide against 16-wide tiles: y backward 26.4 -> 17.5 us, x backward 26.8
// -> 18.5, x forward 18.1 -> 11.8, y forward 20.7 -> 12.4 (the same transforms
// inside the FP64 passes: about 100, 150, 60 and 70 us).  Wider tiles than 32 would
// need the tensor memory of the second CTA.
//
// Every wait is bounded: on time-out the tile sets kStatusGemmTimeout, makes its
// outputs NaN, waits (bounded) for its copies and MMAs in flight, frees its
// tensor memory and returns.
#include "split_gemm.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "lane_gemm.h"
#include "pdl.cuh"
#include "per_device.h"
#include "tc_ptx.cuh"

namespace rbc {
namespace dev {

__device__ long long g_split_wait_limit = kWaitLimit;

constexpr int kSplitThreads = 320;
// The two precisions: 7 digits (transforms), 9 digits (eigenbasis products,
// whose terms span more exponents than a transform's).
template <int D>
struct SplitForm {
  static constexpr int kAcc = D + 1;                         // accumulators (weights i + j)
  static constexpr int kTile = D == 7 ? kSplitTile : 16;     // widest tile
  static constexpr int kStages = D == 7 ? 3 : 2;             // copy ring (two CTAs an SM)
  static constexpr int kChunk = D * kSplitLanes * kSplitK * 2;
  static constexpr int kStageBytes = kChunk + D * kTile * 32;
  static constexpr size_t kSmem = (size_t)kStages * kStageBytes + 128;
};
constexpr int kSplitCols = 256;  // tensor-memory columns of a CTA

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void mma_commit(uint64_t* m) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(m))
               : "memory");
}
// 8 columns of a warp's 32 tensor-memory lanes; the caller waits (tcgen05.wait::ld)
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
}

// instruction descriptor: D f32, A and B bf16, both K-major, M = 128
__device__ __forceinline__ uint32_t split_idesc(int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
}

// bounded wait of one thread
__device__ __forceinline__ bool thread_mbar_wait(uint64_t* m, uint32_t parity, long long limit,
                                                 volatile int* abort_flag) {
  for (long long i = 0; i < limit; i++) {
    if (mbar_try(m, parity)) return true;
    if ((i & 1023) == 1023 && *abort_flag) break;
  }
  *abort_flag = 1;
  return false;
}

// 8 sums of this thread's lane from the eight accumulators, in units of the
// d = 5 accumulator (the two lowest rounded off): 64-bit multiply-adds of
// 32-bit integers, the two highest weights on the high word alone.
__device__ __forceinline__ void split_sums(uint32_t addr, int NT, long long (&v)[8]) {
  uint32_t r[8], q[8];
#pragma unroll
  for (int d = 6; d >= 0; d -= 2) {
    tmem_ld8(addr + d * NT, r);
    tmem_ld8(addr + (d + 1) * NT, q);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int a = __float2int_rn(__uint_as_float(r[j])), b = __float2int_rn(__uint_as_float(q[j]));
      if (d == 6) v[j] = (a + ((b + 128) >> 8) + 128) >> 8;
      else if (d == 4) v[j] = (long long)a * 256 + (v[j] + b);
      else if (d == 2) v[j] = (long long)a * (1 << 24) + ((long long)b * (1 << 16) + v[j]);
      else v[j] += (long long)((unsigned long long)(unsigned)(a * 256 + b) << 32);
    }
  }
}

// v 2^e as a double, rounded to nearest (halves away from zero; integer
// operations; results outside the normal range through ldexp)
__device__ __forceinline__ double split_double(long long v, int e) {
  const long long s = v >> 63;
  const unsigned long long m = (unsigned long long)((v ^ s) - s);  // < 2^63
  if (m == 0) return 0.0;
  const int lz = __clzll((long long)m) - 1;  // the leading bit goes to bit 62
  const unsigned long long t = ((m << lz) + 512) >> 10;
  const int ef = 62 - lz + e + 1023;
  if (ef < 1 || ef > 2045) return ldexp((double)v, e);
  return __longlong_as_double((long long)((((unsigned long long)(ef - 1)) << 52) + t) |
                              (s & (long long)0x8000000000000000ull));
}

template <int D>
__device__ __forceinline__ void split_tile(const SplitJobDev& J, const int lane0, const int n0, const int NT) {
  using F = SplitForm<D>;
  const int tid = threadIdx.x, warp = tid >> 5, wl = tid & 31;
  extern __shared__ __align__(128) unsigned char sm[];
  unsigned char* tail = sm + (size_t)F::kStages * F::kStageBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(tail);  // [F::kStages]
  uint64_t* empty = full + F::kStages;               // [F::kStages]
  uint64_t* accfull = empty + F::kStages;            // [2], see split_acc_wait
  uint64_t* accempty = accfull + 2;
  uint64_t* drain = accempty + 1;                    // MMAs in flight when the tile gave up
  uint32_t* slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(slot + 1);
  volatile int* issued = abort_flag + 1;   // chunks whose MMAs were issued
  volatile int* copied = abort_flag + 2;   // chunks whose copies were issued
  volatile int* lists = abort_flag + 3;    // lists committed to accfull
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"((uint32_t)kSplitCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < F::kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int l = 0; l < 2; l++) mbar_init(&accfull[l], 1);
    mbar_init(accempty, 256);
    mbar_init(drain, 1);
    *abort_flag = 0;
    *issued = 0;
    *copied = 0;
    *lists = 0;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *slot;
  const long long limit = g_split_wait_limit;
  const int nlist = J.nc[1] > 0 ? 2 : 1;
  const int total = J.nc[0] + J.nc[1];
  // the lists of a wide tile share the columns, those of a narrow one have their own
  const bool shared_cols = NT == F::kTile;
  const uint32_t list_cols = shared_cols ? 0u : (uint32_t)(8 * NT);

  if (warp == 8) {
    if (wl == 0) {
      const unsigned char* a0 = J.dig + (size_t)(lane0 / kSplitLanes) * J.ctot * F::kChunk;
      const uint32_t wbytes = (uint32_t)(D * NT * 32);
      const unsigned char* w0 = (NT == kSplitTile ? J.w : J.w16) + (size_t)n0 * total * (D * 32);
      for (int c = 0; c < total; c++) {
        const int s = c % F::kStages, ch = c < J.nc[0] ? J.c0[0] + c : J.c0[1] + c - J.nc[0];
        if (c >= F::kStages &&
            !thread_mbar_wait(&empty[s], (uint32_t)((c / F::kStages - 1) & 1), limit, abort_flag))
          break;
        unsigned char* st = sm + (size_t)s * F::kStageBytes;
        mbar_arrive_expect_tx(&full[s], F::kChunk + wbytes);
        bulk_g2s(st, a0 + (size_t)ch * F::kChunk, F::kChunk, &full[s]);
        bulk_g2s(st + F::kChunk, w0 + (size_t)c * wbytes, wbytes, &full[s]);
        *copied = c + 1;
      }
    }
  } else if (warp == 9) {
    if (wl == 0) {
      const uint32_t w_lbo = (uint32_t)(D * NT / 8) * 128, plane = kSplitLanes * kSplitK * 2;
      for (int c = 0; c < total; c++) {
        const int s = c % F::kStages;
        if (!thread_mbar_wait(&full[s], (uint32_t)((c / F::kStages) & 1), limit, abort_flag)) break;
        const bool first = c == 0 || c == J.nc[0];
        if (c == J.nc[0] && shared_cols && !thread_mbar_wait(accempty, 0, limit, abort_flag)) break;
        const uint32_t acc = tmem + (c >= J.nc[0] ? list_cols : 0u);
        tc_fence_after();
        const uint32_t sa = smem_u32(sm + (size_t)s * F::kStageBytes), sw = sa + F::kChunk;
        const uint64_t w = umma_desc(sw, w_lbo, 128);
        if (first) {
          // digit plane 1 initialises accumulators 1 .. D, plane 0 accumulator 0
          const uint64_t a1 = umma_desc(sa + plane, kSplitLanes * 16, 128), a0 = umma_desc(sa, kSplitLanes * 16, 128);
          mma_bf16(acc + NT, a1, w, split_idesc(D * NT), 0u);
          mma_bf16(acc, a0, w, split_idesc(NT), 0u);
          mma_bf16(acc + NT, a0, umma_desc(sw + (NT / 8) * 128, w_lbo, 128), split_idesc((D - 1) * NT), 1u);
        }
#pragma unroll
        for (int i = 0; i < D; i++) {
          if (first && i < 2) continue;
          const int nj = i == 0 ? D : F::kAcc - i;
          mma_bf16(acc + i * NT, umma_desc(sa + i * plane, kSplitLanes * 16, 128), w, split_idesc(nj * NT), 1u);
        }
        // the last chunks' buffers are not reused: nobody waits for them
        if (c + F::kStages < total) mma_commit(&empty[s]);
        *issued = c + 1;
        if (c + 1 == J.nc[0] || c + 1 == total) {
          mma_commit(&accfull[split_acc_wait(c < J.nc[0] ? 0 : 1).barrier]);
          *lists = *lists + 1;
        }
      }
      if (split_drain_commit(*issued, total)) mma_commit(drain);
    }
  } else {
    // warp w: lanes 32 (w % 4) .., outputs (NT / 2) (w / 4) .. of the tile, 8 at a time
    const int h = warp >> 2, lane = lane0 + 32 * (warp & 3) + wl, nb = NT / 16;
    const uint32_t addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (NT / 2) * h;
    const bool valid = lane < J.lanes;
    const int r = lane / J.nf, f = lane - r * J.nf, p = r % J.parts;
    const int n1 = n0 + (NT / 2) * h, N = J.N, m_lo = J.m_lo, m_hi = nlist == 2 ? J.m_hi : 0;
    const long long es = J.es;
    double* out = J.out + f * J.fs + (r / J.parts) * J.qs + p * J.ps;
    double* mir = out + (J.mirror - n1) * es;
    out += n1 * es;
    const int ex = valid ? J.ex[lane] : 1, e = ex + J.ex_bias;
    auto list_wait = [&](int list) {  // that list's accumulators are complete
      const SplitAccWait w = split_acc_wait(list);
      return warp_mbar_wait(&accfull[w.barrier], w.parity, limit, abort_flag);
    };
    const bool nan = ex == (D == 9 ? kSplitBadLane9 : 0x7ff);
    if constexpr (D == 9) {
      // 8 outputs: the five high and the five low weights in 64-bit integers
      // each, both lists added, then one FP64 multiply-add
      long long hi[8], lo[8];
#pragma unroll
      for (int j = 0; j < 8; j++) hi[j] = lo[j] = 0;
      bool ok = true;
      for (int list = 0; list < nlist && ok; list++) {
        ok = list_wait(list);
        if (!ok) break;
        tc_fence_after();
        uint32_t r8[8];
#pragma unroll
        for (int d = 0; d < F::kAcc; d++) {
          tmem_ld8(addr + d * NT, r8);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          const int w = 8 * (4 - d % 5);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const long long x = (long long)__float2int_rn(__uint_as_float(r8[j])) << w;
            if (d < 5) hi[j] += x;
            else lo[j] += x;
          }
        }
        tc_fence_before();
        if (list == 0) mbar_arrive(accempty);
      }
      if (ok && valid) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int n = n1 + j;
          if (n < N) {
            const double x = fma((double)hi[j], 1099511627776.0, (double)lo[j]);  // hi 2^40 + lo
            const int ee = e + J.rowex[n];
            // scaled in two exact steps (each factor a normal power of two)
            const int e1 = ee / 2, e2 = ee - e1;
            const double y = x * __longlong_as_double((long long)(1023 + e1) << 52) *
                             __longlong_as_double((long long)(1023 + e2) << 52);
            *out = nan ? __longlong_as_double(0x7FF8000000000000ll) : y;
          }
          out += es;
        }
      }
    } else {
      long long v[2][8], o[8];
      bool ok = list_wait(0);
      if (ok && (shared_cols || nlist == 1)) {
        tc_fence_after();
        split_sums(addr, NT, v[0]);
        if (nb == 2) split_sums(addr + 8, NT, v[1]);
        tc_fence_before();
        mbar_arrive(accempty);
      }
      if (ok && nlist == 2) {
        ok = list_wait(1);
        tc_fence_after();
        if (ok && !shared_cols) split_sums(addr, NT, v[0]);
      }
      if (ok) {
#pragma unroll
        for (int b = 0; b < 2; b++) {
          if (b == nb) break;
          if (nlist == 2) split_sums(addr + list_cols + 8 * b, NT, o);
          if (!valid) continue;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int n = n1 + 8 * b + j;
            if (n < N) {
              double x = split_double(nlist == 2 ? v[b][j] + o[j] : v[b][j], e);
              if (nan) x = __longlong_as_double(0x7FF8000000000000ll);
              *out = x;
            }
            if (n >= m_lo && n < m_hi) {
              double x = split_double(v[b][j] - o[j], e);
              if (nan) x = __longlong_as_double(0x7FF8000000000000ll);
              *mir = x;
            }
            out += es;
            mir -= es;
          }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_flag != 0 && tid < kSplitLanes && lane0 + tid < J.lanes) {
    // FP64 callers need not ask for a status: the outputs say that they are lost
    const int lane = lane0 + tid, r = lane / J.nf, f = lane - r * J.nf;
    double* out = J.out + f * J.fs + (r / J.parts) * J.qs + (r % J.parts) * J.ps;
    for (int n = n0; n < min(n0 + NT, J.N); n++) {
      out[n * J.es] = __longlong_as_double(0x7FF8000000000000ll);
      if (nlist == 2 && n >= J.m_lo && n < J.m_hi)
        out[(J.mirror - n) * J.es] = __longlong_as_double(0x7FF8000000000000ll);
    }
  }
  if (*abort_flag != 0 && tid == 0) {
    if (J.status != nullptr) atomicOr(J.status, kStatusGemmTimeout);
    // copies that no MMA waited for, then every commit, the last of which covers
    // all MMAs issued, before the memory is given back
    const int n = *issued, nw = *copied, nl = *lists;
    for (int c = n; c < nw; c++)
      for (long long i = 0; i < kWaitLimit; i++)
        if (mbar_try(&full[c % F::kStages], (uint32_t)((c / F::kStages) & 1))) break;
    for (int c = max(0, n - F::kStages); c < n; c++)
      if (c + F::kStages < total)
        for (long long i = 0; i < kWaitLimit; i++)
          if (mbar_try(&empty[c % F::kStages], (uint32_t)((c / F::kStages) & 1))) break;
    for (int l = 0; l < nl; l++) {
      const SplitAccWait w = split_acc_wait(l);
      for (long long i = 0; i < kWaitLimit; i++)
        if (mbar_try(&accfull[w.barrier], w.parity)) break;
    }
    if (split_drain_commit(n, total))
      for (long long i = 0; i < kWaitLimit; i++)
        if (mbar_try(drain, 0)) break;
  }
  __syncthreads();
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kSplitCols));
}

// tile table entries (job, first lane, first output, tile width)
template <int D>
__global__ void __launch_bounds__(kSplitThreads, 2) k_split_gemm(const SplitJobDev* __restrict__ jobs,
                                                                 const int4* __restrict__ tiles) {
  pdl_enter();
  const int4 tl = tiles[blockIdx.x];
  const SplitJobDev& J = jobs[tl.x];
  if (J.active != nullptr && *J.active == 0) return;
  split_tile<D>(J, tl.y, tl.z, tl.w);
}

// one or two jobs passed by value: the tiles of a lane block side by side
struct SplitJobs2 {
  SplitJobDev j[2];
  int first;  // tiles of job 0
  int most;   // tile width
};
template <int D>
__global__ void __launch_bounds__(kSplitThreads, 2) k_split_gemm_one(const __grid_constant__ SplitJobs2 P) {
  const int second = (int)blockIdx.x >= P.first, b = blockIdx.x - (second ? P.first : 0);
  const SplitJobDev& J = P.j[second];
  const int per = (J.N + P.most - 1) / P.most, n0 = (b % per) * P.most;
  split_tile<D>(J, (b / per) * kSplitLanes, n0, J.N - n0 > 16 ? P.most : 16);
}

}  // namespace dev

size_t split_dig_bytes(int lanes, int cE, int cO, int digits) {
  return (size_t)((lanes + kSplitLanes - 1) / kSplitLanes) * (cE + cO) * digits * (kSplitLanes * kSplitK * 2);
}

SplitMat pack_split_mat(const std::vector<double>& M, int n) {
  SplitMat m;
  m.N = n;
  m.K[0] = std::min(n, split_chunks((n + 1) / 2) * kSplitK);
  m.K[1] = n - m.K[0];
  m.colex.assign(n, 0);
  m.rowex.assign(n, 0);
  // columns scaled by powers of two to a largest entry in [1/2, 1), then rows
  for (int k = 0; k < n; k++) {
    double mx = 0.0;
    for (int r = 0; r < n; r++) mx = std::max(mx, std::fabs(M[(size_t)r * n + k]));
    if (mx > 0.0) std::frexp(mx, &m.colex[k]);
  }
  for (int r = 0; r < n; r++) {
    double mx = 0.0;
    for (int k = 0; k < n; k++) mx = std::max(mx, std::fabs(std::ldexp(M[(size_t)r * n + k], -m.colex[k])));
    if (mx > 0.0) std::frexp(mx, &m.rowex[r]);
  }
  const int nc[2] = {split_chunks(m.K[0]), split_chunks(m.K[1])}, total = nc[0] + nc[1];
  const size_t chunk = (size_t)9 * 16 * 32;
  m.bytes16.assign((size_t)((n + 15) / 16) * total * chunk, 0);
  for (int r = 0; r < n; r++)
    for (int k = 0; k < n; k++) {
      const double w = std::ldexp(M[(size_t)r * n + k], -m.colex[k] - m.rowex[r]);  // |w| < 1
      if (w == 0.0) continue;
      int e;
      const double f = std::frexp(w, &e);  // w = f 2^e, 1/2 <= |f| < 1
      // |w| 2^70 = |f| 2^53 2^(17 + e): 53 bits shifted, as (high word, low word)
      uint64_t a = (uint64_t)std::ldexp(std::fabs(f), 53), lo, hi;
      const int sh = 17 + e;
      if (sh >= 0) {
        lo = a << sh;
        hi = sh > 0 ? a >> (64 - sh) : 0;
      } else {
        hi = 0;
        lo = -sh > 60 ? 0 : (a + (1ull << (-sh - 1))) >> -sh;
      }
      if (w < 0) {
        lo = 0 - lo;
        hi = ~hi + (lo == 0 ? 1 : 0);
      }
      const uint64_t b = lo + 0x8080808080808080ull;
      const int64_t top = (int64_t)hi + (b < lo ? 1 : 0);
      const int list = k >= m.K[0], kl = list ? k - m.K[0] : k, kk = kl % kSplitK;
      unsigned char* c = m.bytes16.data() + ((size_t)(r / 16) * total + (list ? nc[0] : 0) + kl / kSplitK) * chunk;
      for (int i = 0; i < 9; i++) {
        const int d = i == 0 ? (int)top : (int)((b >> (8 * (8 - i))) & 255) - 128;
        const float fl = (float)d;
        uint32_t u;
        memcpy(&u, &fl, 4);
        const uint16_t v = (uint16_t)(u >> 16);
        const int row = i * 16 + r % 16;
        memcpy(c + (size_t)(kk >> 3) * (9 * 16 / 8) * 128 + (row >> 3) * 128 + (row & 7) * 16 + (kk & 7) * 2, &v, 2);
      }
    }
  return m;
}

static int tile_width(int left, int most) { return left > 16 ? most : 16; }

SplitOp pack_split_op(const std::vector<int64_t>& E, int KE, const std::vector<int64_t>& O, int KO, int N) {
  SplitOp op;
  op.N = N;
  op.K[0] = KE;
  op.K[1] = KO;
  const int nc[2] = {split_chunks(KE), split_chunks(KO)};
  const int total = nc[0] + nc[1];
  for (int v = 0; v < 2; v++) {
    std::vector<unsigned char>& bytes = v ? op.bytes16 : op.bytes;
    const int most = v ? 16 : kSplitTile;
    for (int n0 = 0; n0 < N; n0 += most) {
      const int NT = tile_width(N - n0, most);
      const size_t base = bytes.size();
      const size_t chunk = (size_t)kSplitDigits * NT * 32;
      bytes.resize(base + total * chunk, 0);
      for (int list = 0; list < 2; list++) {
        const std::vector<int64_t>& M = list ? O : E;
        const int K = list ? KO : KE;
        for (int n = n0; n < std::min(n0 + NT, N); n++)
          for (int k = 0; k < K; k++) {
            const int64_t y = M[(size_t)n * K + k] + 0x0000808080808080ll;
            unsigned char* c = bytes.data() + base + (size_t)((list ? nc[0] : 0) + k / kSplitK) * chunk;
            for (int i = 0; i < kSplitDigits; i++) {
              const int d = i == 0 ? (int)(y >> 48) : (int)((y >> (8 * (6 - i))) & 255) - 128;
              const float f = (float)d;
              uint32_t u;
              memcpy(&u, &f, 4);
              const uint16_t b = (uint16_t)(u >> 16);  // exact: at most 8 significant bits
              const int row = i * NT + (n - n0), kk = k % kSplitK;
              memcpy(c + (size_t)(kk >> 3) * (kSplitDigits * NT / 8) * 128 + (row >> 3) * 128 + (row & 7) * 16 +
                         (kk & 7) * 2,
                     &b, 2);
            }
          }
      }
    }
  }
  return op;
}

// A launch whose 32-wide tiles would leave SMs idle takes 16-wide ones: twice
// the CTAs, each with half the epilogue (the results are the same: the sums
// are exact).
void split_tiles(const std::vector<SplitJobDev>& jobs, std::vector<int4>& tiles) {
  auto blocks = [](const SplitJobDev& j) { return (j.lanes + kSplitLanes - 1) / kSplitLanes; };
  long wide = 0;
  for (const SplitJobDev& j : jobs) wide += (long)blocks(j) * ((j.N + kSplitTile - 1) / kSplitTile);
  const int most = wide <= kSplitNarrowTiles || (!jobs.empty() && jobs[0].digits == 9) ? 16 : kSplitTile;
  for (size_t j = 0; j < jobs.size(); j++)
    for (int b = 0; b < blocks(jobs[j]); b++)
      for (int n = 0; n < jobs[j].N; n += most)
        tiles.push_back(make_int4((int)j, b * kSplitLanes, n, tile_width(jobs[j].N - n, most)));
  // longest first, so that the last tiles to start are the shortest
  std::stable_sort(tiles.begin(), tiles.end(), [&](const int4& a, const int4& b) {
    return jobs[a.x].nc[0] + jobs[a.x].nc[1] > jobs[b.x].nc[0] + jobs[b.x].nc[1];
  });
}

cudaError_t configure_split_kernels() {
  static PerDeviceFlag done;
  if (done.test()) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(dev::k_split_gemm<7>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)dev::SplitForm<7>::kSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dev::k_split_gemm<9>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dev::SplitForm<9>::kSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dev::k_split_gemm_one<7>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dev::SplitForm<7>::kSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dev::k_split_gemm_one<9>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dev::SplitForm<9>::kSmem);
  if (e == cudaSuccess) done.set();
  return e;
}

cudaError_t launch_split_gemm(const SplitJobDev* jobs, const int4* tiles, int ntiles, int digits, cudaStream_t st) {
  if (ntiles == 0) return cudaSuccess;
  if (digits == 9) return launch_pdl(dev::k_split_gemm<9>, ntiles, dev::kSplitThreads, dev::SplitForm<9>::kSmem, st, jobs, tiles);
  return launch_pdl(dev::k_split_gemm<7>, ntiles, dev::kSplitThreads, dev::SplitForm<7>::kSmem, st, jobs, tiles);
}

cudaError_t launch_split_gemm_one(const SplitJobDev* jobs, int njobs, cudaStream_t st) {
  dev::SplitJobs2 p{};
  auto blocks = [](const SplitJobDev& j) { return (j.lanes + kSplitLanes - 1) / kSplitLanes; };
  auto tiles = [&](const SplitJobDev& j, int most) { return blocks(j) * ((j.N + most - 1) / most); };
  long wide = 0;
  for (int k = 0; k < njobs; k++) {
    p.j[k] = jobs[k];
    wide += tiles(jobs[k], kSplitTile);
  }
  const bool nine = jobs[0].digits == 9;
  p.most = nine || wide <= kSplitNarrowTiles ? 16 : kSplitTile;
  p.first = tiles(p.j[0], p.most);
  const int total = p.first + (njobs > 1 ? tiles(p.j[1], p.most) : 0);
  if (total == 0) return cudaSuccess;
  if (nine) dev::k_split_gemm_one<9><<<total, dev::kSplitThreads, dev::SplitForm<9>::kSmem, st>>>(p);
  else dev::k_split_gemm_one<7><<<total, dev::kSplitThreads, dev::SplitForm<7>::kSmem, st>>>(p);
  return cudaGetLastError();
}

cudaError_t set_split_wait_limit(long long polls) {
  const long long v = polls < 0 ? dev::kWaitLimit : polls;
  return cudaMemcpyToSymbol(dev::g_split_wait_limit, &v, sizeof v);
}

}  // namespace rbc
