// step_split.cu -- the transforms of the plain FP64 step as split GEMMs
// (split_gemm.h): the part of Integrate::update up to the transformed
// convection term (src/navier/navier.rs:540-633, conv_term.rs:22-42).
//
//   S1  rows:     y stencil and derivative of ux, uy, temp          -> digits
//   G1            backward Chebyshev along y                         -> spl_yw
//   S2  columns:  x stencils and derivatives (box) or i k / s (Fourier) -> digits;
//                 box: also d/dx p0
//   G2            backward transform along x                         -> spl_ph
//   S3  columns:  convection products                                -> digits
//   G3            forward transform along x, rows < kx               -> spl_q
//   S4  rows < kx of the result                                      -> digits
//   G4            forward Chebyshev along y, columns < ky            -> m_cv
//
// The passes that follow take m_cv like the mixed form's.  Every GEMM stores
// its outputs with the lanes adjacent in memory, so that its stores are
// coalesced and the next pass, whose lanes run across them, reads a contiguous
// block.
//
// What this replaces: the same transforms inside the CTA passes (step_fp64.cu),
// as FP64 FFTs (n = 2^p + 1) or dense FP64 products.  At two FP64 operations
// per clock and SM those were most of a step.
#include "step_split.h"

#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <tuple>

#include "lane_ops.cuh"
#include "pdl.cuh"
#include "per_device.h"
#include "prims.h"
#include "shared_dev.h"
#include "split_emit.cuh"
#include "step_fp64.h"

namespace rbc {
namespace dev {

// S1: row i of ux, uy, temp.  Lanes i L + (2 f + which) P + part: L = 6 P, P parts.
template <class T>
__global__ void __launch_bounds__(256) k_spl_y1(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  const int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  constexpr int P = sizeof(T) / 8;
  const int i = w.y, ny = c.ny, myc = c.myc, ld = c.ny + 1, N = c.ny - 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  T* O = reinterpret_cast<T*>(smem);  // 3 ortho lanes
  T* D = O + 3 * ld;                  // 3 derivative lanes
  T* IN = D + 3 * ld;
  int* em = reinterpret_cast<int*>(IN + 3 * ld);
  const T* f3[3] = {static_cast<const T*>(c.ux), static_cast<const T*>(c.uy), static_cast<const T*>(c.temp)};
#pragma unroll
  for (int f = 0; f < 3; f++)
    for (int k = tid; k < myc; k += nth) IN[f * ld + k] = f3[f][(size_t)i * myc + k];
  __syncthreads();
  to_ortho<T>(c.ycd, IN, ld, O, ld, 3, tid, nth);
  cheb_diff<T>(c.odd, O, ld, D, ld, ny, 3, 1, nullptr, 0, tid, nth);
  const double* base = reinterpret_cast<const double*>(O);
  auto lane = [&](int r) {  // r = (2 f + which) P + part
    const int part = P == 2 ? r & 1 : 0, l = P == 2 ? r >> 1 : r;
    return base + (size_t)((l & 1) * 3 + (l >> 1)) * ld * P + part;
  };
  split_emit(
      c.spl_y1, i * 6 * P, 6 * P, ny, (N >> 1) + 1, (N + 1) >> 1, kSplitShlValue,
      [&](int r, int k) { return lane(r)[k * P]; },
      [&](int r, int list, int k, auto fix) { return fix(lane(r)[(2 * k + list) * P]); }, em, tid, nth);
}
static size_t smem_spl_y1(const CaseDev& c) {
  return (size_t)9 * (c.ny + 1) * (c.kind == KIND_PERIODIC ? 16 : 8) + 64;
}

// S2, box: column j.  Lanes 8 j + (u, v, then for ux, uy, temp: d/dx, d/dy).
__global__ void __launch_bounds__(256) k_spl_x1_box(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  const int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y, nx = c.nx, ny = c.ny, mxc = c.mxc, ld = c.nx + 1, N = c.nx - 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  extern __shared__ double2 smem[];
  double* OR = reinterpret_cast<double*>(smem);  // ortho lanes Y0u Y0v Y0t p0 Y1u Y1v Y1t
  double* D = OR + 7 * ld;                       // d/dx of the first four
  double* IN = D + 4 * ld;
  int* em = reinterpret_cast<int*>(IN + 7 * ld);
  // columns of the block: Y0u Y1u Y0v Y1v Y0t Y1t
  const double* yw = c.spl_yw + (size_t)j * 6 * mxc;
  for (int idx = tid; idx < 6 * mxc; idx += nth) {
    const int k = idx / 6, s = idx - 6 * k;
    IN[((s & 1) * 4 + (s >> 1)) * ld + k] = yw[idx];
  }
  const double* p0 = static_cast<const double*>(c.p0);
  for (int k = tid; k < nx; k += nth) OR[3 * ld + k] = p0[(size_t)k * ny + j];
  __syncthreads();
  for (int l = 0; l < 7; l++) {
    if (l == 3) continue;
    const BasisDev& b = (l & 3) == 2 ? c.xt : c.xu;
    for (int k = tid; k < nx; k += nth) OR[l * ld + k] = stencil_at(b, IN + l * ld, k);
  }
  __syncthreads();
  cheb_diff<double>(c.odd, OR, ld, D, ld, nx, 4, 1, nullptr, 0, tid, nth);
  double* gp = static_cast<double*>(c.s[0]);  // d/dx p0 / aspect
  for (int l = 0; l < 3; l++)
    for (int k = tid; k < nx; k += nth) D[l * ld + k] *= inv_asp;
  for (int k = tid; k < nx; k += nth) gp[(size_t)k * ny + j] = D[3 * ld + k] * inv_asp;
  __syncthreads();
  auto lane = [&](int r) {
    const int f = (r - 2) >> 1;
    return r < 2 ? OR + r * ld : r & 1 ? OR + (4 + f) * ld : D + f * ld;
  };
  split_emit(
      c.spl_x1, 8 * j, 8, nx, (N >> 1) + 1, (N + 1) >> 1, kSplitShlValue, [&](int r, int k) { return lane(r)[k]; },
      [&](int r, int list, int k, auto fix) { return fix(lane(r)[2 * k + list]); }, em, tid, nth);
}
static size_t smem_spl_x1_box(const CaseDev& c) { return (size_t)18 * (c.nx + 1) * 8 + 64; }

// S2, periodic: the same lanes from i k / aspect and the y derivatives.
__global__ void __launch_bounds__(256) k_spl_x1_per(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  const int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y, mx = c.mx, ld = c.mx, kim = (c.nx - 1) / 2;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  extern __shared__ double2 smem[];
  double2* L = smem;  // 8 lanes
  int* em = reinterpret_cast<int*>(L + 8 * ld);
  const double2* yw = reinterpret_cast<const double2*>(c.spl_yw + (size_t)j * 12 * mx);
  for (int idx = tid; idx < 6 * mx; idx += nth) {
    const int k = idx / 6, s = idx - 6 * k, f = s >> 1;  // Y0u Y1u Y0v Y1v Y0t Y1t
    const double2 v = yw[idx];
    if (s & 1) {
      L[(3 + 2 * f) * ld + k] = v;
    } else {
      L[(2 + 2 * f) * ld + k] = mul_ik(v, (double)k) * inv_asp;
      if (f < 2) L[f * ld + k] = v;
    }
  }
  __syncthreads();
  // c2r ignores the imaginary parts of the mean and (n even) of the Nyquist mode
  const double* b = reinterpret_cast<const double*>(L);
  split_emit(
      c.spl_x1, 8 * j, 8, mx + kim, mx, kim, kSplitShlValue,
      [&](int r, int k) { return b[2 * (r * ld + (k < mx ? k : k - mx + 1)) + (k < mx ? 0 : 1)]; },
      [&](int r, int list, int k, auto fix) { return fix(b[2 * (r * ld + k + list) + list]); }, em, tid, nth);
}
static size_t smem_spl_x1_per(const CaseDev& c) { return (size_t)8 * c.mx * 16 + 64; }

// S3: products of column j -> digits of their forward x transform, lanes 3 j + f
__global__ void __launch_bounds__(256) k_spl_prod(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  const int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y, nx = c.nx, ny = c.ny, ld = c.nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* PR = reinterpret_cast<double*>(smem);
  int* em = reinterpret_cast<int*>(PR + 3 * ld);
  for (int x = tid; x < nx; x += nth) {
    const double2* ph = reinterpret_cast<const double2*>(c.spl_ph + ((size_t)x * ny + j) * 8);
    const double2 uv = ph[0], gu = ph[1], gv = ph[2], gt = ph[3];
    const size_t g = (size_t)x * ny + j;
    PR[x] = uv.x * gu.x + uv.y * gu.y;
    PR[ld + x] = uv.x * gv.x + uv.y * gv.y;
    double p = uv.x * gt.x + uv.y * gt.y;
    p = p + uv.x * c.bc_dx[g];
    p = p + uv.y * c.bc_dy[g];
    PR[2 * ld + x] = p;
  }
  __syncthreads();
  const bool per = c.kind == KIND_PERIODIC;
  // fold: Chebyshev pairs (k, n-1-k), Fourier pairs (k, n-k)
  const int KE = per ? nx / 2 + 1 : (nx + 1) / 2, KO = per ? (nx - 1) / 2 : nx / 2;
  split_emit(
      c.spl_p, 3 * j, 3, nx, KE, KO, kSplitShlSum, [&](int r, int k) { return PR[r * ld + k]; },
      [&](int r, int list, int k, auto fix) {
        const int a = per ? k + list : k, b = per ? nx - a : nx - 1 - a;
        const long long u = fix(PR[r * ld + a]);
        if (a == b || b == nx) return u;  // the centre; the first Fourier point
        const long long v = fix(PR[r * ld + b]);
        return list ? u - v : u + v;
      },
      em, tid, nth);
}
static size_t smem_spl_prod(const CaseDev& c) { return (size_t)3 * (c.nx + 1) * 8 + 64; }

// S4: row e of the x-transformed products -> digits of the forward y transform, lanes 3 e + f
__global__ void __launch_bounds__(256) k_spl_q(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  const int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int e = w.y, ny = c.ny, N = c.ny - 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* Q = reinterpret_cast<double*>(smem);  // [k][3]
  int* em = reinterpret_cast<int*>(Q + 3 * ny);
  const double* q = c.spl_q + (size_t)e * 3 * ny;
  for (int k = tid; k < 3 * ny; k += nth) Q[k] = q[k];
  __syncthreads();
  split_emit(
      c.spl_cq, 3 * e, 3, ny, (ny + 1) / 2, ny / 2, kSplitShlSum, [&](int r, int k) { return Q[3 * k + r]; },
      [&](int r, int list, int k, auto fix) {
        const long long u = fix(Q[3 * k + r]);
        if (2 * k == N) return u;
        const long long v = fix(Q[3 * (N - k) + r]);
        return list ? u - v : u + v;
      },
      em, tid, nth);
}
static size_t smem_spl_q(const CaseDev& c) { return (size_t)3 * c.ny * 8 + 64; }

}  // namespace dev

// ---------------------------------------------------------------------------
// operators
// ---------------------------------------------------------------------------
void split_terms(bool fourier, int n, int K[2]) {
  K[0] = fourier ? n / 2 + 1 : (n + 1) / 2;
  K[1] = fourier ? (n - 1) / 2 : n / 2;
}

SplitOp make_split_op(int kind, int n, int rows, int* wshift) {
  const bool four = kind >= SOP_C2R;
  const int N = four ? n : n - 1;  // angles: 2 pi j k / n (Fourier), pi j k / (n - 1) (Chebyshev)
  const int period = four ? n : 2 * N;
  // entries scale * cos or sin: forward Chebyshev 2/N, c2r 2/n, the others 1
  const bool small = kind == SOP_CHEB_FWD_E || kind == SOP_CHEB_FWD_O || kind == SOP_C2R;
  int ws = 0;
  if (small)
    while ((2 << (ws + 1)) <= N) ws++;  // (2 / N) 2^ws <= 1
  *wshift = ws;
  const long double scale = ldexpl(small ? 2.0L / (long double)N : 1.0L, kSplitOpBits + ws);
  const long double pi2 = 6.283185307179586476925286766559005768L;
  std::vector<int64_t> cs(period), ch(period), sn(period);
  for (int t = 0; t < period; t++) {
    const long double a = pi2 * (long double)t / (long double)period;
    cs[t] = llroundl(scale * cosl(a));
    ch[t] = llroundl(0.5L * scale * cosl(a));
    sn[t] = llroundl(scale * sinl(a));
  }
  auto at = [&](const std::vector<int64_t>& tab, long jk) { return tab[(size_t)(jk % period)]; };
  int K[2];
  split_terms(four, n, K);
  std::vector<int64_t> E, O;
  auto two_lists = [&](int H) { E.resize((size_t)H * K[0]); O.resize((size_t)H * K[1]); };
  switch (kind) {
    case SOP_CHEB_BWD: {
      // T_k(x_j) = (-1)^k cos(pi j k / N)
      const int H = (n + 1) / 2;
      two_lists(H);
      for (int j = 0; j < H; j++) {
        for (int m = 0; m < K[0]; m++) E[(size_t)j * K[0] + m] = at(cs, (long)j * (2 * m));
        for (int m = 0; m < K[1]; m++) O[(size_t)j * K[1] + m] = 2 * j == N ? 0 : -at(cs, (long)j * (2 * m + 1));
      }
      return pack_split_op(E, K[0], O, K[1], H);
    }
    case SOP_CHEB_FWD_E:
    case SOP_CHEB_FWD_O: {
      // coefficient k: (-1)^k (2 / N) c_k sum_j c_j cos(pi j k / N) v_j, c = 1/2 at the ends
      const int par = kind == SOP_CHEB_FWD_O, KL = K[par], M = (rows - par + 1) / 2;
      E.resize((size_t)M * KL);
      for (int m = 0; m < M; m++)
        for (int j = 0; j < KL; j++) {
          const int k = 2 * m + par;
          const int halves = (k == 0 || k == N) + (j == 0);
          int64_t v = halves == 0 ? at(cs, (long)j * k) : halves == 1 ? at(ch, (long)j * k) : llroundl(0.25L * scale);
          E[(size_t)m * KL + j] = par ? -v : v;
        }
      return pack_split_op(E, KL, O, 0, M);
    }
    case SOP_C2R: {
      // v_j = (1/n) (re_0 + 2 sum re_k cos - 2 sum im_k sin), the Nyquist mode once
      const int H = n / 2 + 1;
      two_lists(H);
      for (int j = 0; j < H; j++) {
        for (int k = 0; k < K[0]; k++)
          E[(size_t)j * K[0] + k] = (k == 0 || 2 * k == n) ? at(ch, (long)j * k) : at(cs, (long)j * k);
        for (int k = 0; k < K[1]; k++) O[(size_t)j * K[1] + k] = -at(sn, (long)j * (k + 1));
      }
      return pack_split_op(E, K[0], O, K[1], H);
    }
    case SOP_R2C_RE:
    case SOP_R2C_IM: {
      const int im = kind == SOP_R2C_IM, KL = K[im];
      E.resize((size_t)rows * KL);
      for (int k = 0; k < rows; k++)
        for (int j = 0; j < KL; j++) E[(size_t)k * KL + j] = im ? -at(sn, (long)(j + 1) * k) : at(cs, (long)j * k);
      return pack_split_op(E, KL, O, 0, rows);
    }
  }
  throw std::runtime_error("make_split_op: unknown kind");
}

SplitOpDev shared_split_op(Arena& owner, int kind, int n, int rows) {
  static SharedDev<std::tuple<int, int, int, int>, SplitOpDev> cache;
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  return cache.get(std::make_tuple(dev, kind, n, rows), owner, [&](SplitOpDev& d) {
    const SplitOp op = make_split_op(kind, n, rows, &d.wshift);
    d.N = op.N;
    const size_t n32 = (op.bytes.size() + 127) & ~size_t(127);
    auto mem = make_dev_block(n32 + op.bytes16.size());
    unsigned char* p = static_cast<unsigned char*>(mem->p);
    cuda_check(cudaMemcpy(p, op.bytes.data(), op.bytes.size(), cudaMemcpyHostToDevice), "upload shared operator");
    cuda_check(cudaMemcpy(p + n32, op.bytes16.data(), op.bytes16.size(), cudaMemcpyHostToDevice),
               "upload shared operator");
    d.w = p;
    d.w16 = p + n32;
    return mem;
  });
}

// The eigenbasis matrices of a tensor solver's axis 0 in nine digits.
SplitMatDev shared_split_mat(Arena& owner, int kind, int n, bool poisson, bool fwd) {
  static SharedDev<std::tuple<int, int, int, bool, bool>, SplitMatDev> cache;
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  return cache.get(std::make_tuple(dev, kind, n, poisson, fwd), owner, [&](SplitMatDev& d) {
    std::vector<double> F, B;
    tensor_eigenbasis(make_basis(kind, n), poisson, F, B);
    const SplitMat m = pack_split_mat(fwd ? F : B, n - 2);
    const size_t nb = (m.bytes16.size() + 127) & ~size_t(127), ne = (size_t)m.N * 4;
    auto mem = make_dev_block(nb + 2 * ne);
    unsigned char* p = static_cast<unsigned char*>(mem->p);
    cuda_check(cudaMemcpy(p, m.bytes16.data(), m.bytes16.size(), cudaMemcpyHostToDevice), "upload shared operator");
    cuda_check(cudaMemcpy(p + nb, m.colex.data(), ne, cudaMemcpyHostToDevice), "upload shared operator");
    cuda_check(cudaMemcpy(p + nb + ne, m.rowex.data(), ne, cudaMemcpyHostToDevice), "upload shared operator");
    d.w16 = p;
    d.colex = reinterpret_cast<const int*>(p + nb);
    d.rowex = reinterpret_cast<const int*>(p + nb + ne);
    d.N = m.N;
    d.K0 = m.K[0];
    d.K1 = m.K[1];
    return mem;
  });
}

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
// The split form has six more launches than the transforms inside the passes
// and does their work on the tensor cores.  Measured, us per step, inside the
// passes | split:
//   dense axes      box 64^2 113 | 127, 80^2 133 | 139, 96^2 143 | 143, 112^2 182 | 172,
//                   128^2 187 | 172; periodic 96x80 92 | 92, 128^2 117 | 111, 64x256 261 | 139
//   FFT (2^p + 1)   box 129^2 171 | 174, 257^2 371 | 301; periodic 128x65 82 | 92,
//                   256x129 115 | 120, 512x257 250 | 195
//   Fourier length with a prime factor above 8 (a direct sum in the passes):
//                   22x17 144 | 72, 26x33 178 | 74, 66x48 154 | 82, 110x33 162 | 80,
//                   47x33 1648 | 76, 106x33 2088 | 80
// so the lines lie at 9000 grid points where an axis has no fast butterfly in
// the passes, at 48000 where every axis has one, and nowhere for a Fourier
// length with a prime factor above 8.  A list holds at most 320 terms
// (split_gemm.cu), hence lengths up to 640.
bool split_step_size(const CaseDev& c) {
  if (c.nx < 16 || c.ny < 16 || c.nx > 640 || c.ny > 640) return false;
  bool fast = c.cy.use_fft != 0;
  int radix = 2;
  if (c.kind != KIND_PERIODIC) fast = fast && c.cx.use_fft != 0;
  else if (c.fx.log2M < 0)
    for (int k = 0; k < c.fx.nrad; k++) radix = std::max(radix, c.fx.rad[k]);
  if (radix > 8) return true;
  return c.nx * c.ny >= (fast ? 48000 : 9000);
}

SplitJobDev split_op_job(const SplitLanesDev& s, const SplitOpDev& op, int lanes, int shl, double* out, long long ls,
                         long long es, unsigned int* status) {
  SplitJobDev j{};
  j.dig = s.dig;
  j.ex = s.ex;
  j.w = op.w;
  j.w16 = op.w16;
  j.out = out;
  j.status = status;
  j.es = es;
  j.lanes = lanes;
  j.nf = 1;
  j.parts = 1;
  j.qs = ls;
  j.ctot = s.cE + s.cO;
  j.c0[0] = 0;
  j.nc[0] = s.cE;
  j.c0[1] = s.cE;
  j.nc[1] = s.cO;
  j.N = op.N;
  j.ex_bias = split_ex_bias(shl, op.wshift);
  j.digits = kSplitDigits;
  return j;
}

SplitJobDev split_mat_job(const SplitLanesDev& s, const SplitMatDev& m, int lanes, double* out, long long es,
                          unsigned int* status) {
  SplitJobDev j{};
  j.dig = s.dig;
  j.ex = s.ex;
  j.w = j.w16 = m.w16;
  j.out = out;
  j.status = status;
  j.es = es;
  j.lanes = lanes;
  j.nf = 1;
  j.parts = 1;
  j.qs = 1;
  j.ctot = s.cE + s.cO;
  j.nc[0] = s.cE;
  j.c0[1] = s.cE;
  j.nc[1] = s.cO;
  j.N = m.N;
  j.ex_bias = split_ex_bias9();
  j.digits = 9;
  j.rowex = m.rowex;
  return j;
}

// Dense FP64 products inside X3 and X4 | split GEMMs, us per step: box 144^2
// 144 | 158, 160^2 156 | 160, 192^2 178 | 174, 224^2 199 | 184, 264^2 280 | 227.
// (An accumulator's exact range ends at 256 terms a list.)
bool split_eig_size(const CaseDev& c) { return c.kind != KIND_PERIODIC && c.nx >= 176 && c.nx <= 514; }

void add_split_launches(const CaseDev& c, bool on, StepPlan& p) {
  const bool per = c.kind == KIND_PERIODIC;
  const int P = per ? 2 : 1;
  auto cta = [&](int kernel, int lanes, size_t smem) {
    StepLaunch L;
    L.kernel = kernel;
    L.smem = on ? (smem + 127) & ~size_t(127) : 0;
    if (on)
      for (int i = 0; i < lanes; i++) L.items.push_back(make_int4(0, i, 1, 0));
    p.launches.push_back(L);
  };
  auto gemm = [&](const std::vector<SplitJobDev>& jobs) {
    StepLaunch L;
    L.kernel = K_SPLIT_GEMM;
    L.smem = 0;
    if (on) L.sjobs = jobs;
    p.launches.push_back(L);
  };
  auto job = [&](const SplitLanesDev& s, const SplitOpDev& op, int lanes, int shl, double* out, long long es) {
    return split_op_job(s, op, lanes, shl, out, 1, es, c.status);  // lanes adjacent
  };
  // one list of a forward transform: terms E (par 0) or O (par 1)
  auto one = [&](SplitJobDev j, const SplitLanesDev& s, int par) {
    j.c0[0] = par ? s.cE : 0;
    j.nc[0] = par ? s.cO : s.cE;
    j.nc[1] = 0;
    return j;
  };
  // S1, G1
  cta(per ? K_SPL_Y1_C : K_SPL_Y1_R, c.mxc, dev::smem_spl_y1(c));
  const int l1 = 6 * P * c.mxc;
  SplitJobDev g1 = job(c.spl_y1, c.sop_yb, l1, kSplitShlValue, c.spl_yw, l1);
  g1.mirror = c.ny - 1;
  g1.m_lo = 0;
  g1.m_hi = c.ny / 2;
  gemm({g1});
  // S2, G2
  cta(per ? K_SPL_X1_PER : K_SPL_X1_BOX, c.ny, per ? dev::smem_spl_x1_per(c) : dev::smem_spl_x1_box(c));
  const int l2 = 8 * c.ny;
  SplitJobDev g2 = job(c.spl_x1, c.sop_xb, l2, kSplitShlValue, c.spl_ph, l2);
  g2.mirror = per ? c.nx : c.nx - 1;
  g2.m_lo = per ? 1 : 0;
  g2.m_hi = per ? (c.nx + 1) / 2 : c.nx / 2;
  gemm({g2});
  // S3, G3: spl_q row e (periodic: 2 k + part) holds 3 ny values
  cta(K_SPL_PROD, c.ny, dev::smem_spl_prod(c));
  const int l3 = 3 * c.ny;
  gemm({one(job(c.spl_p, c.sop_xf[0], l3, kSplitShlSum, c.spl_q, 2 * l3), c.spl_p, 0),
        one(job(c.spl_p, c.sop_xf[1], l3, kSplitShlSum, c.spl_q + l3, 2 * l3), c.spl_p, 1)});
  // S4, G4: m_cv[f][row][m]
  cta(K_SPL_Q, P * c.kx, dev::smem_spl_q(c));
  std::vector<SplitJobDev> g4;
  for (int par = 0; par < 2; par++) {
    SplitJobDev j = one(job(c.spl_cq, c.sop_yf[par], 3 * P * c.kx, kSplitShlSum,
                            static_cast<double*>(c.m_cv) + par * P, 2 * P),
                        c.spl_cq, par);
    j.nf = 3;
    j.parts = P;
    j.fs = (long long)c.kx * c.ky * P;
    j.qs = (long long)c.ky * P;
    j.ps = 1;
    g4.push_back(j);
  }
  gemm(g4);
}

cudaError_t configure_step_split_kernels() {
  static PerDeviceFlag done;
  if (done.test()) return cudaSuccess;
  const int big = (int)smem_limit();
  cudaError_t e = configure_split_kernels();
#define SET_ATTR(k) \
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  SET_ATTR(dev::k_spl_y1<double>);
  SET_ATTR(dev::k_spl_y1<double2>);
  SET_ATTR(dev::k_spl_x1_box);
  SET_ATTR(dev::k_spl_x1_per);
  SET_ATTR(dev::k_spl_prod);
  SET_ATTR(dev::k_spl_q);
#undef SET_ATTR
  if (e == cudaSuccess) done.set();
  return e;
}

cudaError_t launch_step_split_kernel(int kernel, int nblocks, size_t smem, cudaStream_t s, const CaseDev* cases,
                                     const int4* work) {
  const dim3 g(nblocks), b(256);
  switch (kernel) {
    case K_SPL_Y1_R: return launch_pdl(dev::k_spl_y1<double>, g, b, smem, s, cases, work);
    case K_SPL_Y1_C: return launch_pdl(dev::k_spl_y1<double2>, g, b, smem, s, cases, work);
    case K_SPL_X1_BOX: return launch_pdl(dev::k_spl_x1_box, g, b, smem, s, cases, work);
    case K_SPL_X1_PER: return launch_pdl(dev::k_spl_x1_per, g, b, smem, s, cases, work);
    case K_SPL_PROD: return launch_pdl(dev::k_spl_prod, g, b, smem, s, cases, work);
    case K_SPL_Q: return launch_pdl(dev::k_spl_q, g, b, smem, s, cases, work);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace rbc
